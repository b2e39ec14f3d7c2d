"""The Python extension is an option: the library is built without it, and one made for another torch or Python is not used."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(code, **env):
    return subprocess.run([sys.executable, "-W", "ignore", "-c", code], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True)


def test_built_for_this_torch():
    r = run("from oxillama_b200 import build; build.build()\n"
            "import sys, torch; from oxillama_b200 import device as d\n"
            "assert d._native.torch_version == str(torch.__version__) and d._native.python_version == sys.hexversion >> 16\n"
            "assert d._native.__file__ == build.EXT")
    assert r.returncode == 0, r.stderr


# An extension of another torch, of another Python, and one that does not say (as it was made before).
@pytest.mark.parametrize("made_for", ["dict(torch_version='2.0.0', python_version=sys.hexversion >> 16)",
                                      "dict(torch_version=str(torch.__version__), python_version=0x030b)", "dict()"])
def test_another_torch_is_not_used(made_for):
    r = run("import sys, types, torch, oxillama_b200\n"
            "m = types.ModuleType('oxillama_b200._qk_torch'); m.gemv = m.gemm = m.bind = None\n"
            f"m.__dict__.update({made_for})\n"
            "sys.modules[m.__name__] = oxillama_b200._qk_torch = m\n"
            "from oxillama_b200 import device\n"
            "assert device._native is None and device._bound_lib() is None")
    assert r.returncode == 0, r.stderr


# No C++ compiler: the library is there all the same, and what an earlier build left is gone.
@pytest.mark.parametrize("cxx", ["false", "no-such-compiler"])
def test_library_is_built_without_it(cxx, tmp_path):
    ext = tmp_path / "_qk_torch.cpython-399-x.so"
    for old in (ext, tmp_path / "_qk_torch.so"):
        old.write_bytes(b"old")
        os.utime(old, (0, 0))
    r = run("from oxillama_b200 import build; import os\n"
            f"build.EXT = {str(ext)!r}\n"
            "assert build.build() == build.LIB and os.path.exists(build.LIB)\n"
            f"assert not os.listdir({str(tmp_path)!r})", CXX=cxx)
    assert r.returncode == 0, r.stderr


# Made by another command (another torch): made again, although its source is no newer.
def test_made_again_for_another_torch(tmp_path):
    ext = tmp_path / "_qk_torch.cpython-399-x.so"
    r = run("from oxillama_b200 import build; import os, torch\n"
            f"build.EXT = {str(ext)!r}; build.OBJ = {str(tmp_path)!r}\n"
            "made = []\n"
            "build.subprocess.check_call = lambda cmd: (made.append(cmd), open(build.EXT, 'w').close())\n"
            "build._build_extension(); build._build_extension(); assert len(made) == 1\n"
            "torch.__version__ = '0.0.0'\n"
            "build._build_extension(); assert len(made) == 2 and any('0.0.0' in c for c in made[1])")
    assert r.returncode == 0, r.stderr
