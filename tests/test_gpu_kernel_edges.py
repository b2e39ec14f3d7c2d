"""GPU kernels at the sizes where their tiling can go wrong: remainders of every tile, the smallest
call, both sides of each dispatch rule.  The reference is the f64 product of the oracle's dequantised
weights.

Bounds, per output (a: largest |w| of the 32-column block, x: the activation, sums over a row):
  * fp16 operands: a term carries at most four independent roundings to 11 bits (the scale, the
    minimum, the weight, the activation), each uniform within 2^-11 of its value, so the error of a sum
    has sigma <= 2^-11 sqrt(4 / 3) sqrt(sum a^2 x^2); 7 sigma.
  * f32-grade sums: block sums are exact, the activation lies on a 254^3 grid of its block's largest
    value, and the f32 additions over two terms per block each round within 2^-24:
    sigma <= 2^-23 (1 + sqrt(2 K / 32)) sqrt(sum a^2 xmax^2); 7 sigma.
"""
import numpy as np
import pytest

import oracle_lib as O
from oxillama_b200 import synth as S

pytestmark = pytest.mark.gpu

TC_TYPES = [S.Q4_K, S.Q8_0, S.Q4_0, S.Q6_K, S.IQ4_XS]


def block_max(a):
    """|a| replaced by the largest of its 32-column block."""
    pad = -a.shape[1] % 32
    b = np.pad(np.abs(a), ((0, 0), (0, pad))).reshape(a.shape[0], -1, 32).max(axis=2)
    return np.repeat(b, 32, axis=1)[:, : a.shape[1]].astype(np.float64)


def assert_product(y, x, wd, half):
    import torch
    xd, w = torch.from_numpy(x).cuda().double(), torch.from_numpy(wd).cuda().double()
    ref = (xd @ w.T).cpu().numpy()
    a = torch.from_numpy(block_max(wd) ** 2).cuda()
    xx = x.astype(np.float64) if half else block_max(x)
    s = np.sqrt((torch.from_numpy(xx ** 2).cuda() @ a.T).cpu().numpy())
    sigma = 2.0 ** -11 * np.sqrt(4 / 3) if half else 2.0 ** -23 * (1 + np.sqrt(2 * x.shape[1] / 32))
    assert np.all(np.isfinite(y))
    assert np.all(np.abs(y - ref) <= 7 * sigma * s + 1e-30), float((np.abs(y - ref) / (sigma * s + 1e-30)).max())


def device_product(t, w, x, rows, cols, m, launches=None):
    """The product, and in `launches` what such a call launches."""
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status
    dw = DeviceWeights(t, w, rows, cols)
    y = torch.full((m, rows), float("nan"), device="cuda")
    xd = torch.from_numpy(x).cuda()

    def call():
        if m == 1:
            dw.gemv(xd, y)
        else:
            dw.gemm(xd, y, m)

    if launches is not None:
        from launches import launched
        launches += launched(call)
        y.fill_(float("nan"))
    call()
    check_device_status()
    dw.free()
    return y.cpu().numpy()


# Rows around the 128- and 256-row tiles, columns around super-blocks, tokens around the tile widths
# (16 .. 64 in one CTA, up to 256 in a pair, several token blocks); K split over many CTAs (128 x 8192),
# over few (2048 rows), a tile with both accumulator halves of unequal width (129, 300 tokens).
@pytest.mark.parametrize("rows,cols,m", [(1, 256, 5), (127, 512, 16), (129, 768, 17), (257, 2048, 64), (128, 8192, 65), (300, 1280, 128),
                                         (2048, 1024, 129), (513, 2304, 257), (640, 512, 300), (384, 256, 700)])
@pytest.mark.parametrize("t", TC_TYPES)
def test_tensor_core_matmul_edges(t, rows, cols, m):
    if t in (S.Q8_0, S.Q4_0):
        cols += 32 * (m % 7)  # a last super-block that is not whole
    w, x = S.gen_weight(t, rows, cols, seed=m), S.gen_acts(m, cols, seed=m)
    assert_product(device_product(t, w, x, rows, cols, m), x, O.dequant_matrix(t, w, rows, cols), True)


# One to five rows (five: the tensor cores, or chunks of rows for the formats without them); fewer rows
# than a chunk, a ragged last chunk, several 2048-column tiles with a short last one, fewer chunks than SMs and more.
@pytest.mark.parametrize("rows,cols", [(1, 256), (9, 2048), (1190, 2304), (37, 14336), (5003, 512)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("t", TC_TYPES + [S.Q5_K, S.Q3_K, S.Q2_K])
def test_decode_kernel_edges(t, m, rows, cols):
    w, x = S.gen_weight(t, rows, cols, seed=rows + m), S.gen_acts(m, cols, seed=rows + m)
    # (more than one row of 14336 columns may not fit the shared memory beside the tiles: tensor cores)
    # the tensor cores (fp16 operands) take what the decode kernels do not: at 14336 columns those have room beside
    # the tiles for one split row of Q8_0 and Q6_K, for two of the others
    most = {S.Q8_0: 1, S.Q6_K: 1}.get(t, 2) if cols == 14336 else 2 if t == S.Q6_K else 4
    half = t in TC_TYPES and m > most
    assert_product(device_product(t, w, x, rows, cols, m), x, O.dequant_matrix(t, w, rows, cols), half)


# Gate and up in one launch (up to four rows), as two groups of one matmul with silu(g) * u in the
# conversion (more), and one after the other (different formats).
@pytest.mark.parametrize("tgu,td,hidden,inter", [(S.Q4_0, S.Q8_0, 544, 1056), (S.Q8_0, S.Q4_0, 2080, 320), (S.IQ4_XS, S.Q4_K, 256, 2560),
                                                 (S.Q5_K, S.Q6_K, 2304, 512), (S.Q3_K, S.Q4_K, 512, 768), (S.Q2_K, S.Q2_K, 768, 256)])
@pytest.mark.parametrize("m", [1, 2, 4, 5, 70])
def test_ffn_edges(tgu, td, hidden, inter, m):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status, ffn
    ws = [S.gen_weight(q, r, c, seed=71, stream=i, d_range=(1e-3, 3e-3)) for i, (q, r, c) in
          enumerate([(tgu, inter, hidden), (tgu, inter, hidden), (td, hidden, inter)])]
    x = S.gen_acts(m, hidden, seed=71) * np.float32(0.25)
    st, ref = O.ffn(tgu, ws[0], ws[1], td, ws[2], x, m, hidden, inter, hidden)
    assert st == 0
    dw = [DeviceWeights(tgu, ws[0], inter, hidden), DeviceWeights(tgu, ws[1], inter, hidden), DeviceWeights(td, ws[2], hidden, inter)]
    y = torch.full((m, hidden), float("nan"), device="cuda")
    ffn(*dw, torch.from_numpy(x).cuda(), y, m)
    check_device_status()
    half = any(q in TC_TYPES and m > (2 if q == S.Q6_K else 4) for q in (tgu, td))
    # three chained products: each within 1e-3 of its largest value on fp16 operands, within 2e-5 in f32
    assert np.abs(y.cpu().numpy() - ref).max() <= (3e-3 if half else 6e-5) * np.abs(ref).max()
    for d in dw:
        d.free()


# Gate and up as a prompt has them: pairs of CTAs, tiles of one and of two accumulator halves, equal and not (160 to 240
# tokens), several tiles a pair, a ragged last token block, segments of one to a few super-blocks.
@pytest.mark.parametrize("t,hidden,inter", [(S.Q6_K, 512, 14336), (S.Q4_K, 256, 14336), (S.Q6_K, 1024, 4736), (S.IQ4_XS, 768, 9472)])
@pytest.mark.parametrize("m", [129, 150, 200, 300, 512, 700, 801])
def test_ffn_of_a_prompt(t, hidden, inter, m):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status, ffn
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    ws = [S.gen_weight(t, r, c, seed=72, stream=i, d_range=(1e-3, 3e-3)) for i, (r, c) in enumerate(shapes)]
    x = torch.from_numpy(S.gen_acts(m, hidden, seed=72) * np.float32(0.25)).cuda()
    g, u, d = (torch.from_numpy(O.dequant_matrix(t, w, r, c)).cuda().double() for w, (r, c) in zip(ws, shapes))
    ref = (torch.nn.functional.silu(x.double() @ g.T) * (x.double() @ u.T)) @ d.T
    dw = [DeviceWeights(t, w, r, c) for w, (r, c) in zip(ws, shapes)]
    y = torch.full((m, hidden), float("nan"), device="cuda")
    ffn(*dw, x, y, m)
    check_device_status()
    # three chained products, each within 1e-3 of its largest value (fp16 operands)
    assert float((y.double() - ref).abs().max()) <= 3e-3 * float(ref.abs().max())
    for w in dw:
        w.free()


# Up to 16 tokens: every expert that is hit, on the decode kernels up to four rows and on the tensor cores
# beside them above; one expert takes all tokens, another none; also shards that start inside, with that
# expert and without.  A token whose experts here have up to four rows each keeps the f32-grade bound.
@pytest.mark.parametrize("t", [S.Q4_K, S.Q8_0, S.Q6_K, S.IQ4_XS])
@pytest.mark.parametrize("tokens,top_k", [(1, 1), (1, 3), (2, 2), (4, 2), (5, 1), (9, 3), (16, 2)])
def test_moe_few_tokens(t, tokens, top_k):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    hidden, inter, n = 512, 2304, 6
    w = [[S.gen_weight(t, r, c, seed=81, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(n)]
         for k, (r, c) in enumerate([(inter, hidden), (inter, hidden), (hidden, inter)])]
    dq = [np.stack([O.dequant_matrix(t, a, r, c) for a in ws]) for ws, (r, c) in zip(w, [(inter, hidden), (inter, hidden), (hidden, inter)])]
    x = S.gen_acts(tokens, hidden, seed=82) * np.float32(0.25)
    logits = S.gen_acts(tokens, n, seed=83)
    logits[:, 5], logits[:, 1] = -30.0, logits[:, 1] + 6.0
    for b, e in ((0, n), (1, 4), (2, 6)):
        ids, wts = O.moe_route(logits, top_k)
        ref = np.zeros((tokens, hidden))
        for i in range(tokens):
            for s in range(top_k):
                if b <= ids[i, s] < e:
                    g, u, d = (q[ids[i, s]].astype(np.float64) for q in dq)
                    hg = g @ x[i]
                    ref[i] += wts[i, s] * (d @ (hg / (1 + np.exp(-hg)) * (u @ x[i])))
        ex = moe.MoeExperts(t, w[0][b:e], w[1][b:e], w[2][b:e], hidden, inter, n, expert_begin=b)
        y = torch.full((tokens, hidden), float("nan"), device="cuda")
        ex.forward(torch.from_numpy(logits).cuda(), torch.from_numpy(x).cuda(), y, top_k)
        check_device_status()
        ex.free()
        check_moe(y.cpu().numpy(), ref, ids, b, e)


def check_moe(y, ref, ids, b, e):
    # three chained products, each within 1e-3 of its largest value on fp16 operands, within 2e-5 in f32
    local = (ids >= b) & (ids < e)
    many = local & (np.bincount(ids[ids >= 0], minlength=e)[ids] > 4)
    bound = np.where(many.any(axis=1), 3e-3, 6e-5)[:, None] * np.abs(ref).max()
    assert np.all(np.abs(y - ref) <= bound)


# The same with a down projection of another format and hidden rows of several k-tiles.
@pytest.mark.parametrize("t,td,hidden,inter", [(S.Q4_K, S.Q6_K, 512, 4608), (S.IQ4_XS, S.Q8_0, 256, 6400), (S.Q4_0, S.Q4_K, 4352, 512)])
@pytest.mark.parametrize("tokens", [1, 3, 9])
def test_moe_few_tokens_mixed(t, td, hidden, inter, tokens):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import DeviceWeights, check_device_status
    n, top_k = 4, 2
    shapes = [(t, inter, hidden), (t, inter, hidden), (td, hidden, inter)]
    w = [[S.gen_weight(q, r, c, seed=83, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(n)] for k, (q, r, c) in enumerate(shapes)]
    x, logits = S.gen_acts(tokens, hidden, seed=84) * np.float32(0.25), S.gen_acts(tokens, n, seed=84)
    ids, wts = O.moe_route(logits, top_k)
    ref = np.zeros((tokens, hidden))
    for e in range(n):
        g, u, d = (O.dequant_matrix(q, ws[e], r, c).astype(np.float64) for ws, (q, r, c) in zip(w, shapes))
        at, slot = np.nonzero(ids == e)
        hg = x[at] @ g.T
        ref[at] += wts[at, slot][:, None] * ((hg / (1 + np.exp(-hg)) * (x[at] @ u.T)) @ d.T)
    dn = [DeviceWeights(td, ws, hidden, inter) for ws in w[2]]
    ex = moe.MoeExperts(t, w[0], w[1], [S.gen_weight(t, hidden, inter)] * n, hidden, inter, n)
    ex._d = type(ex._d)(*[d.handle for d in dn])  # (the class uploads one format)
    y = torch.full((tokens, hidden), float("nan"), device="cuda")
    ex.forward(torch.from_numpy(logits).cuda(), torch.from_numpy(x).cuda(), y, top_k)
    check_device_status()
    check_moe(y.cpu().numpy(), ref, ids, 0, n)
    ex.free()
    for d in dn:
        d.free()


# Long rows: a job of the decode kernels holds one row where two split activation rows do not fit beside
# the tiles, so 16 experts of four rows each make 64 of them; also nine experts at the edge of the job list.
@pytest.mark.parametrize("n,tokens,top_k", [(16, 16, 4), (9, 11, 3), (16, 16, 2), (8, 8, 4)])
def test_moe_few_tokens_long_rows(n, tokens, top_k):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    t, hidden, inter = S.Q8_0, 256, 12288
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    w = [[S.gen_weight(t, r, c, seed=85, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(2)] for k, (r, c) in enumerate(shapes)]
    dq = [[torch.from_numpy(O.dequant_matrix(t, a, r, c)).cuda().double() for a in ws] for ws, (r, c) in zip(w, shapes)]
    x = S.gen_acts(tokens, hidden, seed=86) * np.float32(0.25)
    logits = S.gen_acts(tokens, n, seed=87) * np.float32(0.1)
    for i in range(tokens):  # every expert gets its share of the rows
        for k in range(top_k):
            logits[i, (i + k * (n // top_k)) % n] += 5.0
    ids, wts = O.moe_route(logits, top_k)
    xd = torch.from_numpy(x).cuda()
    ref = torch.zeros(tokens, hidden, dtype=torch.float64, device="cuda")
    for i in range(tokens):
        for s in range(top_k):
            g, u, d = (q[ids[i, s] % 2] for q in dq)
            hg = g @ xd[i].double()
            ref[i] += float(wts[i, s]) * (d @ (hg / (1 + torch.exp(-hg)) * (u @ xd[i].double())))
    ex = moe.MoeExperts(t, *[[ws[e % 2] for e in range(n)] for ws in w], hidden, inter, n)
    lg = torch.from_numpy(logits).cuda()
    ys = []
    for xi in (torch.zeros_like(xd), xd):  # rows that were left out would show what the first call left
        ys.append(torch.full((tokens, hidden), float("nan"), device="cuda"))
        ex.forward(lg, xi, ys[-1], top_k)
        check_device_status()
    ex.free()
    assert torch.all(ys[0] == 0)
    # up to four rows of an expert: gate and up f32-grade; the down projection of several such rows may
    # take fp16 operands (its K is long)
    assert float((ys[1] - ref).abs().max()) <= 1e-3 * float(ref.abs().max())


# Host buffers: x and y each go through a staging buffer of 256 KB or are copied, on both sides of it.
@pytest.mark.parametrize("rows,cols,m", [(1, 256, 1), (14336, 512, 4), (16384, 512, 4), (16385, 512, 4), (64, 8192, 8), (64, 8448, 8),
                                         (4096, 4096, 16), (4104, 4096, 17)])
def test_host_call_around_the_staging_size(rows, cols, m):
    from oxillama_b200.kernels import KernelDispatcher, QuantTensor
    w, x = S.gen_weight(S.Q4_K, rows, cols, seed=91), S.gen_acts(m, cols, seed=91)
    y = np.full((m, rows), np.nan, np.float32)
    KernelDispatcher().get_kernel(S.Q4_K).gemm(QuantTensor(w, (rows, cols), S.Q4_K), x, y, m, rows, cols)
    assert_product(y, x, O.dequant_matrix(S.Q4_K, w, rows, cols), m > 4)


# Host calls run on a stream of the context that nothing orders behind the caller's: they share no scratch
# with device calls still in flight there (a matmul's converted activations and counters, split activations).
@pytest.mark.parametrize("rows,cols,m", [(4096, 4096, 96), (512, 12288, 3)])
def test_host_call_beside_device_calls(rows, cols, m):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status
    from oxillama_b200.kernels import KernelDispatcher, QuantTensor
    w, wh = S.gen_weight(S.Q4_K, rows, cols, seed=95), S.gen_weight(S.Q4_K, 256, 4096, seed=96)
    dw, x, xh = DeviceWeights(S.Q4_K, w, rows, cols), torch.from_numpy(S.gen_acts(m, cols, seed=95)).cuda(), S.gen_acts(1, 4096, seed=96)
    kern, qt = KernelDispatcher().get_kernel(S.Q4_K), QuantTensor(wh, (256, 4096), S.Q4_K)
    want, yh0, yh = torch.empty(m, rows, device="cuda"), np.empty((1, 256), np.float32), np.empty((1, 256), np.float32)
    dw.gemm(x, want, m)
    check_device_status()
    kern.gemv(qt, xh, yh0)
    side, ys = torch.cuda.Stream(), [torch.empty(m, rows, device="cuda") for _ in range(24)]
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(4):
        for y in ys:
            dw.gemm(x, y, m, stream=side)
        kern.gemv(qt, xh, yh)
        side.synchronize()
        assert np.array_equal(yh, yh0)
        assert all(torch.equal(y, want) for y in ys)
    dw.free()


# Calls of the formats without a tensor-core matmul may overlap on different streams of one context: each
# stream has its own place for split activations, and the calls of streams that found none left (20 streams),
# like those of a captured graph, use none.
@pytest.mark.parametrize("t", [S.Q5_K, S.Q3_K, S.Q2_K])
def test_calls_on_many_streams(t):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status
    from oxillama_b200.kernels import Context
    rows, cols, ctx = 1024, 12288, Context()
    dw = DeviceWeights(t, S.gen_weight(t, rows, cols, seed=97), rows, cols, ctx=ctx)
    xs = [torch.from_numpy(S.gen_acts(m, cols, seed=m)).cuda() for m in (1, 2)]
    want = [torch.empty(len(x), rows, device="cuda") for x in xs]
    for x, y in zip(xs, want):
        dw.gemm(x, y, len(x))
    streams = [torch.cuda.Stream() for _ in range(20)]
    ys = [[torch.empty_like(w) for w in want] for _ in range(40)]
    graph, yg = torch.cuda.CUDAGraph(), torch.empty_like(want[1])
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        dw.gemm(xs[1], yg, 2)
    for i, pair in enumerate(ys):
        for x, y in zip(xs, pair):
            dw.gemm(x, y, len(x), stream=streams[i % 20])
        graph.replay()
    torch.cuda.synchronize()
    check_device_status(ctx)
    assert torch.equal(yg, want[1])
    assert all(torch.equal(y, w) for pair in ys for y, w in zip(pair, want))
    dw.free()


# Activations at the ends of the f32 range, on the kernels that split them into digits (in the CTAs and by
# the kernel before: 512 and 9216 columns) and through a host call.  Tiny rows keep the f32-grade bound down
# to 1e-36, below it on that value's grid; a row with an infinity or a NaN gives no finite number, and its
# neighbour does not notice.
@pytest.mark.parametrize("cols", [512, 9216])
@pytest.mark.parametrize("t", TC_TYPES + [S.Q5_K, S.Q3_K, S.Q2_K])
def test_decode_activation_range(t, cols):
    import torch
    from oxillama_b200.kernels import KernelDispatcher, QuantTensor
    rows = 40
    kern = KernelDispatcher().get_kernel(t)
    big, small = (5e-3, 1e-2) if t == S.Q6_K else (2.0, 4.0), (1e-6, 1e-5)
    for scale, d_range in ((1e-30, big), (1e-36, big), (3e-38, big), (1e36, small), (6e37, small)):
        w = S.gen_weight(t, rows, cols, seed=98, d_range=d_range)  # (scales large: products of tiny rows stay normal numbers)
        wd = O.dequant_matrix(t, w, rows, cols).astype(np.float64)
        x = S.gen_acts(2, cols, seed=98).clip(-4, 4)
        if scale > 1:  # one large value: the sums must not overflow
            x[:, 1:] = 0
            x[:, 0] = (4, -4)
        x = (x * np.float64(scale)).astype(np.float32)
        ref = x.astype(np.float64) @ wd.T
        s = np.sqrt(np.maximum(block_max(x), 1e-36 if scale < 1 else 0) ** 2 @ (block_max(wd) ** 2).T)
        bound = 7 * 2.0 ** -23 * (1 + np.sqrt(2 * cols / 32)) * s
        ys = [device_product(t, w, x, rows, cols, 2), device_product(t, w, x[:1], rows, cols, 1), np.empty((2, rows), np.float32)]
        kern.gemm(QuantTensor(w, (rows, cols), t), x, ys[2], 2, rows, cols)
        for y in ys:
            assert np.all(np.abs(y - ref[: len(y)]) <= bound[: len(y)]), (scale, float((np.abs(y - ref[: len(y)]) / bound[: len(y)]).max()))
    w = S.gen_weight(t, rows, cols, seed=98)
    x = S.gen_acts(2, cols, seed=99)
    want = device_product(t, w, x, rows, cols, 2)
    for bad in (np.nan, np.inf, -np.inf):
        xb = x.copy()
        xb[1, cols - 7] = bad
        y = device_product(t, w, xb, rows, cols, 2)
        assert not np.isfinite(y[1]).any() and np.array_equal(y[0], want[0])



# The conversion of activations to fp16 at the lower end of the f32 range, where the row's scale is a power
# of two without a finite reciprocal (below 2^-118) or the row is subnormal, and at rows longer than it
# keeps in registers (16384 columns).
@pytest.mark.parametrize("rows,cols,m", [(96, 512, 5), (96, 512, 70), (40, 16640, 6)])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e-37, 1e-41])
def test_conversion_of_small_rows(rows, cols, m, scale):
    w = S.gen_weight(S.Q4_K, rows, cols, seed=101, d_range=(2.0, 4.0))
    wd = O.dequant_matrix(S.Q4_K, w, rows, cols).astype(np.float64)
    x = S.gen_acts(m, cols, seed=101)
    x[1::2] = (x[1::2] * np.float64(scale)).astype(np.float32)  # every second row: a scale of its own
    x[2] = 0
    y = device_product(S.Q4_K, w, x, rows, cols, m)
    ref = x.astype(np.float64) @ wd.T
    s = np.sqrt(x.astype(np.float64) ** 2 @ (block_max(wd) ** 2).T)
    assert np.all(np.abs(y - ref) <= 7 * 2.0 ** -11 * np.sqrt(4 / 3) * s + 2.0 ** -149)


# silu(g) * u of tiny activations (products of about 1e-40), and of rows longer than the conversion keeps in
# shared memory (28160 columns).
@pytest.mark.parametrize("hidden,inter,m,scale", [(512, 768, 5, 1e-20), (512, 768, 70, 1e-20), (256, 28416, 5, 1.0), (256, 28416, 5, 1e-20)])
def test_ffn_conversion(hidden, inter, m, scale):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status, ffn
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    ws = [S.gen_weight(S.Q4_K, r, c, seed=102, stream=i, d_range=(1e-3, 3e-3)) for i, (r, c) in enumerate(shapes)]
    g, u, d = (O.dequant_matrix(S.Q4_K, w, r, c).astype(np.float64) for w, (r, c) in zip(ws, shapes))
    x = (S.gen_acts(m, hidden, seed=102) * np.float64(scale)).astype(np.float32)
    hg = x.astype(np.float64) @ g.T
    ref = (hg / (1 + np.exp(-hg)) * (x.astype(np.float64) @ u.T)) @ d.T
    dw = [DeviceWeights(S.Q4_K, w, r, c) for w, (r, c) in zip(ws, shapes)]
    y = torch.full((m, hidden), float("nan"), device="cuda")
    ffn(*dw, torch.from_numpy(x).cuda(), y, m)
    check_device_status()
    # three chained products, each within 1e-3 of its largest value (fp16 operands)
    assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()
    for w in dw:
        w.free()


# The first matmul of a context, captured: up to 128 rows of 4096 columns need no more scratch than the
# context starts with, whichever tiles and K split the shape gets (the last two: tiles that cover more rows
# than the scratch would hold, of which only the sixteens with activations count).
@pytest.mark.parametrize("t,rows,cols,m", [(S.Q4_K, 4096, 4096, 8), (S.Q6_K, 300, 8192, 60), (S.Q8_0, 1024, 3840, 128),
                                           (S.Q5_K, 512, 9216, 4), (S.IQ4_XS, 14336, 4096, 120), (S.Q4_K, 4096, 8192, 107),
                                           (S.Q4_0, 2396, 12288, 74)])
def test_first_call_in_a_capture(t, rows, cols, m):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status
    from oxillama_b200.kernels import Context
    w, x = S.gen_weight(t, rows, cols, seed=103), S.gen_acts(m, cols, seed=103)
    want = device_product(t, w, x, rows, cols, m)
    ctx = Context()
    dw, xd, y = DeviceWeights(t, w, rows, cols, ctx=ctx), torch.from_numpy(x).cuda(), torch.zeros(m, rows, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dw.gemm(xd, y, m)
    graph.replay()
    torch.cuda.synchronize()
    check_device_status(ctx)
    assert np.array_equal(y.cpu().numpy(), want)
    dw.free()


# Batches of the formats without a tensor-core matmul: on the decode kernels in pieces of up to four rows, or,
# where the matrix is too small for that many launches, in one launch of the generic kernel.
@pytest.mark.parametrize("rows,cols,m,launches", [(8, 256, 300, 1), (64, 512, 70, 1), (256, 1024, 256, 1), (2048, 2048, 24, 24), (37, 14336, 6, 12)])
@pytest.mark.parametrize("t", [S.Q5_K, S.Q3_K, S.Q2_K])
def test_batches_without_tensor_cores(t, rows, cols, m, launches):
    import torch
    from cuda.bindings import runtime
    from oxillama_b200.device import DeviceWeights
    w, x = S.gen_weight(t, rows, cols, seed=104), S.gen_acts(m, cols, seed=104)
    assert_product(device_product(t, w, x, rows, cols, m), x, O.dequant_matrix(t, w, rows, cols), False)
    dw, xd, y = DeviceWeights(t, w, rows, cols), torch.from_numpy(x).cuda(), torch.empty(m, rows, device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        dw.gemm(xd, y, m)
    err, _, n = runtime.cudaGraphGetNodes(graph.raw_cuda_graph())
    assert int(err) == 0 and n <= launches
    dw.free()


# Few rows: the last box of 128 rows ends in zeroed chunks behind the matrix (or, where those would be many
# bytes, outside of it); a shard's end is not the matrix's.
@pytest.mark.parametrize("t,rows,cols,m", [(S.Q8_0, 8, 1280, 600), (S.Q4_K, 1, 256, 300), (S.IQ4_XS, 120, 768, 70), (S.Q6_K, 129, 512, 40), (S.Q4_K, 8, 262144, 5)])
def test_matmul_of_few_rows(t, rows, cols, m):
    import torch
    from oxillama_b200.device import DeviceWeights, check_device_status
    w, x = S.gen_weight(t, rows, cols, seed=105), S.gen_acts(m, cols, seed=105)
    wd = O.dequant_matrix(t, w, rows, cols)
    assert_product(device_product(t, w, x, rows, cols, m), x, wd, True)
    b, e = rows // 3, rows - rows // 4
    dw = DeviceWeights(t, w, rows, cols, row_begin=b, row_end=e)
    y = torch.full((m, e - b), float("nan"), device="cuda")
    dw.gemm(torch.from_numpy(x).cuda(), y, m)
    check_device_status()
    dw.free()
    assert_product(y.cpu().numpy(), x, wd[b:e], True)


# Either form of the activations' conversion (up to 63 rows, from 64 rows of up to 4096 columns, longer ones).
@pytest.mark.parametrize("cols,m", [(256, 63), (256, 64), (4096, 64), (4352, 64)])
@pytest.mark.parametrize("t", TC_TYPES)
def test_conversion_forms(t, cols, m):
    rows = 100
    w, x = S.gen_weight(t, rows, cols, seed=106), S.gen_acts(m, cols, seed=106)
    assert_product(device_product(t, w, x, rows, cols, m), x, O.dequant_matrix(t, w, rows, cols), True)


# Expert layers with one to three super-blocks a row (a tile each to a CTA pair, however few) and rows that the
# conversion takes in either form, up to 4096 columns and above.
@pytest.mark.parametrize("t,hidden,inter", [(S.Q4_K, 256, 256), (S.Q8_0, 768, 288), (S.Q6_K, 512, 4352)])
@pytest.mark.parametrize("tokens", [17, 300])
def test_moe_short_rows(t, hidden, inter, tokens):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    n, top_k, shapes = 4, 2, [(inter, hidden), (inter, hidden), (hidden, inter)]
    w = [[S.gen_weight(t, r, c, seed=107, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(n)] for k, (r, c) in enumerate(shapes)]
    x, logits = S.gen_acts(tokens, hidden, seed=108) * np.float32(0.25), S.gen_acts(tokens, n, seed=109)
    ids, wts = O.moe_route(logits, top_k)
    ref = np.zeros((tokens, hidden))
    for e in range(n):
        g, u, d = (O.dequant_matrix(t, ws[e], r, c).astype(np.float64) for ws, (r, c) in zip(w, shapes))
        at, slot = np.nonzero(ids == e)
        hg = x[at] @ g.T
        ref[at] += wts[at, slot][:, None] * ((hg / (1 + np.exp(-hg)) * (x[at] @ u.T)) @ d.T)
    ex = moe.MoeExperts(t, *w, hidden, inter, n)
    y = torch.full((tokens, hidden), float("nan"), device="cuda")
    ex.forward(torch.from_numpy(logits).cuda(), torch.from_numpy(x).cuda(), y, top_k)
    check_device_status()
    ex.free()
    # three chained products, each within 1e-3 of its largest value (fp16 operands)
    assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()


# Groups of every size around the activation boxes (one to four of whole 8-row atoms): tiles of 64 tokens in one CTA
# and of 96 and 256 in a pair.  The bound: three chained products, each within 1e-3 of its largest value.
@pytest.mark.parametrize("counts", [[1, 15, 16, 17, 47, 48, 49, 64, 65, 0], [96, 97, 64, 65, 81, 80, 1, 33, 95, 20],
                                    [160, 161, 128, 127, 40, 41, 79, 300, 2, 0]])
@pytest.mark.parametrize("t", [S.Q4_K, S.IQ4_XS])
def test_moe_group_sizes(t, counts):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    n, hidden, inter = len(counts), 512, 768
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    w = [[S.gen_weight(t, r, c, seed=111, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(n)] for k, (r, c) in enumerate(shapes)]
    which = np.random.default_rng(112).permutation(np.repeat(np.arange(n), counts))
    tokens = len(which)
    x = S.gen_acts(tokens, hidden, seed=113) * np.float32(0.25)
    logits = np.zeros((tokens, n), np.float32)
    logits[np.arange(tokens), which] = 9.0
    ref = np.zeros((tokens, hidden))
    for e in range(n):
        g, u, d = (O.dequant_matrix(t, ws[e], r, c).astype(np.float64) for ws, (r, c) in zip(w, shapes))
        at = which == e
        hg = x[at] @ g.T
        ref[at] = (hg / (1 + np.exp(-hg)) * (x[at] @ u.T)) @ d.T
    ex = moe.MoeExperts(t, *w, hidden, inter, n)
    y = torch.full((tokens, hidden), float("nan"), device="cuda")
    ex.forward(torch.from_numpy(logits).cuda(), torch.from_numpy(x).cuda(), y, 1)
    check_device_status()
    ex.free()
    assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()


# Chunks through the ring of weight tiles: fewer than groups of warps, one more or fewer than the stages, several rounds
# of the ring, one to three k-tiles a chunk with the last one whole, half and one span.  (Q6_K takes further stages where
# a CTA has more tiles than a multiple of the groups holds: at 4096 columns up to 4736 rows four, above them seven.)
RING_SHAPES = [(5, 8448), (1190, 12288), (9480, 4096), (5003, 8448), (5003, 6144), (5003, 8192)]


@pytest.mark.parametrize("t,rows,cols", [(t, *s) for t in (S.Q6_K, S.Q4_K, S.Q8_0) for s in RING_SHAPES] +
                         [(S.Q6_K, 4736, 4096), (S.Q6_K, 4737, 4096), (S.Q6_K, 24100, 4096)])
@pytest.mark.parametrize("m", [1, 2, 3])
def test_decode_ring(t, m, rows, cols):
    w = S.gen_weight(t, rows, cols, seed=121)
    x = S.gen_acts(m, cols, seed=122)
    y = device_product(t, w, x, rows, cols, m)
    # (three rows of Q6_K, and of Q8_0 two of 12288 columns or three of 8448, go to the tensor cores: fp16 operands)
    most = 2 if t == S.Q6_K else {12288: 1, 8448: 2}.get(cols, 3) if t == S.Q8_0 else 3
    assert_product(y, x, O.dequant_matrix(t, w, rows, cols), half=m > most)


# Routing and lists of a grouped call: one round of 1024 (token, slot) pairs and several, up to eight experts and up to 32, a
# shard of them, the last size that one block plans and the first that it does not.  Equal logits go to the lower experts, and
# so do those of a token with a NaN among them.  Routing as the stand-alone entry point gives it (tested against the
# oracle); the bound is test_moe_short_rows'.
@pytest.mark.parametrize("n,top_k,tokens,begin,local", [(8, 2, 512, 0, 8), (8, 3, 683, 0, 8), (9, 2, 40, 3, 5), (32, 3, 400, 8, 16),
                                                        (4, 4, 4096, 0, 4), (4, 4, 4097, 0, 4), (3, 1, 18, 0, 1)])
def test_moe_group_plan(n, top_k, tokens, begin, local):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    hidden, inter = 256, 256
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    w = [[S.gen_weight(S.Q8_0, r, c, seed=131, stream=3 * e + k, d_range=(1e-3, 3e-3)) for e in range(local)] for k, (r, c) in enumerate(shapes)]
    x, logits = S.gen_acts(tokens, hidden, seed=132) * np.float32(0.25), S.gen_acts(tokens, n, seed=133)
    logits[7] = 0.5
    logits[11] = np.nan
    logits[tokens - 1, n - 1] = np.nan
    ids, wts = (v.cpu().numpy() for v in moe.route(torch.from_numpy(logits).cuda(), top_k))
    assert all(np.array_equal(ids[t], np.arange(top_k)) for t in (7, 11, tokens - 1))
    ref = np.zeros((tokens, hidden))
    for e in range(local):
        g, u, d = (O.dequant_matrix(S.Q8_0, ws[e], r, c).astype(np.float64) for ws, (r, c) in zip(w, shapes))
        at, slot = np.nonzero(ids == begin + e)
        hg = x[at] @ g.T
        np.add.at(ref, at, wts[at, slot][:, None] * ((hg / (1 + np.exp(-hg)) * (x[at] @ u.T)) @ d.T))
    ex = moe.MoeExperts(S.Q8_0, *w, hidden, inter, n, expert_begin=begin)
    y = torch.full((tokens, hidden), float("nan"), device="cuda")
    ex.forward(torch.from_numpy(logits).cuda(), torch.from_numpy(x).cuda(), y, top_k)
    check_device_status()
    ex.free()
    assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()


# One row by pairs of CTAs, half of K each (148 SMs: where 2 ceil(chunks / 148) > ceil(chunks / 74)): a single chunk, one and two
# for some pairs, the most that a pair can be given; halves of equal and of unequal length, the last block ragged; and neighbours
# that stay with whole chunks: even shares, a chunk or a column less than it takes, halves of 33 and 32 spans, and IQ4_XS with a
# chunk for nearly every pair.
PAIRS = [(3, 14336), (592, 13568), (592, 13500), (1190, 14592), (1185, 14400), (1776, 16128), (18352, 13312)]
WHOLE = [(593, 13500), (1777, 16128), (18353, 13312), (1184, 14336), (592, 16640)]


@pytest.mark.parametrize("t,rows,cols,pair", [(t, *s, True) for t in (S.Q6_K, S.Q5_K) for s in PAIRS] +
                         [(t, *s, False) for t in (S.Q6_K, S.Q5_K) for s in WHOLE] +
                         [(S.IQ4_XS, 4096, 13824, True), (S.IQ4_XS, 1190, 14000, True), (S.IQ4_XS, 440, 14000, True), (S.IQ4_XS, 441, 14000, False),
                          (S.IQ4_XS, 592, 14336, False), (S.IQ4_XS, 4096, 13568, False), (S.Q3_K, 592, 11264, True),
                          (S.Q3_K, 4096, 11008, True), (S.Q3_K, 1190, 11200, True), (S.Q3_K, 592, 10752, False), (S.Q6_K, 592, 13056, False),
                          (S.Q5_K, 592, 12288, True), (S.Q5_K, 592, 12032, False), (S.Q4_K, 592, 14336, False)])
def test_decode_pairs(t, rows, cols, pair):
    from launches import sm_count
    assert sm_count() == 148
    w = S.gen_weight(t, rows, cols, seed=141)
    x = S.gen_acts(1, cols, seed=142)
    ks = []
    y = device_product(t, w, x, rows, cols, 1, ks)
    assert ((ks[-1].name, ks[-1].ints[4]) == ("qk_gemv_imma_kernel", 3)) == pair, ks
    assert_product(y, x, O.dequant_matrix(t, w, rows, cols), half=False)
    assert np.array_equal(y, device_product(t, w, x, rows, cols, 1))  # the same bits on every run


# Decode launches may start before the one ahead has ended, and with QK_PDL=0, by which a developer's build rules that out, none
# may, those of pairs of CTAs included.  (Read once per process; other builds do not know the knob.)
@pytest.mark.parametrize("pdl", [0, 1])
def test_pdl_knob(pdl):
    import os
    import subprocess
    import sys
    from oxillama_b200 import _lib
    if pdl == 0 and b"QK_PDL" not in open(_lib.LIB_PATH, "rb").read():
        pytest.skip("built without QK_DEV_KNOBS")
    code = f"""
import sys; sys.path[:0] = [{os.path.dirname(__file__)!r}, {os.path.dirname(os.path.dirname(__file__))!r}]
import torch
from launches import launched, programmatic_edges
from oxillama_b200 import synth as S
from oxillama_b200.device import DeviceWeights
for t, rows, cols, mode in ((S.Q6_K, 592, 14336, 3), (S.Q6_K, 592, 4096, 0), (S.Q4_K, 592, 4096, 0)):
    w = DeviceWeights(t, S.gen_weight(t, rows, cols, seed=1), rows, cols)
    x, y = torch.zeros(cols, device="cuda"), torch.zeros(rows, device="cuda")
    call = lambda: (w.gemv(x, y), w.gemv(x, y))
    assert [k.ints[4] for k in launched(call)] == [mode, mode], launched(call)
    assert programmatic_edges(call) == ({pdl}, 1), programmatic_edges(call)
"""
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "QK_PDL": str(pdl)}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


# Rows whose scales lie anywhere in fp16's range (each row is expanded over a power of two of its own): rows of subnormal
# scales, of the largest, and of both kinds of blocks in one row; a row of zeros; all ways of writing out (whole tiles in one
# CTA and in pairs, clusters, partials through the workspace).  Weights of up to 65504 * 63 * 15 stay within f32 sums.
# The bound is assert_product's.
@pytest.mark.parametrize("t", [S.Q4_K, S.Q6_K])
@pytest.mark.parametrize("rows,cols,m", [(200, 512, 9), (4096, 2048, 33), (600, 1024, 130), (130, 8192, 300), (40, 256, 5)])
def test_matmul_row_scales(t, rows, cols, m):
    bb, nb = S.BLOCK_BYTES[t], cols // 256
    w = S.gen_weight(t, rows, cols, seed=151).reshape(rows, nb, bb).copy()
    at = [0, 2] if t == S.Q4_K else [208]
    top = 900.0 if t == S.Q4_K else 440.0  # 63 d, 128 d: weights up to fp16's largest, as before
    r, k = np.arange(rows)[:, None], np.arange(nb)[None, :]
    d = 2.0 ** np.array([-24, -20, -14, -10, -4, 0, 6, 9])[r % 8] * np.where(r % 3 == 0, 2.0 ** -(k % 5), 1.0)
    for o in at:
        w[:, :, o:o + 2] = np.minimum(d, top).astype(np.float16)[:, :, None].view(np.uint8)
    w[17:18] = 0
    w = w.reshape(-1)
    x = S.gen_acts(m, cols, seed=152)
    wd = O.dequant_matrix(t, w, rows, cols)
    y = device_product(t, w, x, rows, cols, m)
    assert_product(y, x, wd, half=True)
    assert np.all(y[:, 17] == 0)


# The arithmetic of rows of ordinary blocks, restated: weights rounded once to fp16's grid (subnormals included) over the power of two
# of the largest scale that the blocks' d allows, whatever sub-scales are in use (here a quarter to an eighth of the int8 range), and
# activations over a power of two of their row.  What is left is the f32 sums'.
@pytest.mark.parametrize("rows,cols,m", [(200, 1024, 24), (1024, 4096, 8), (300, 2048, 130)])
def test_matmul_q6k_row_factor(rows, cols, m):
    t, bb, nb = S.Q6_K, S.BLOCK_BYTES[S.Q6_K], cols // 256
    w = S.gen_weight(t, rows, cols, seed=171, d_range=(1e-4, 2e-3)).reshape(rows, nb, bb).copy()
    w[:, :, 192:208] = np.random.default_rng(172).integers(-32, 32, (rows, nb, 16)).astype(np.int8).view(np.uint8)
    w[:, 1, 208:210] = np.array([1e-4], np.float16).view(np.uint8)
    w[:, 2, 208:210] = np.array([2e-3], np.float16).view(np.uint8)
    x = S.gen_acts(m, cols, seed=173)
    x[:, :256] = x[:, 512:] = 0  # the block with the smallest scale alone, whose weights lie near the subnormals
    y = device_product(t, w.reshape(-1), x, rows, cols, m)
    d = w[:, :, 208:210].copy().view(np.float16).astype(np.float64)[:, :, 0]
    top = 128 * np.abs(d).max(1)
    f, e = np.frexp(top)
    factor = 2.0 ** (e + 8 + (f > 0.998))
    half = lambda v: v.astype(np.float16).astype(np.float64)
    s = half(w[:, :, 192:208].view(np.int8) * (d * 2.0 ** 24 / factor[:, None])[:, :, None])
    off = half(s * -(2.0 ** -19))
    blk = w[:, :, :192].astype(np.int64)
    q = np.empty((rows, nb, 256), np.int64)
    for g in range(2):
        for k in range(4):
            lo = blk[:, :, 64 * g + 32 * (k & 1):64 * g + 32 * (k & 1) + 32] >> (4 * (k >> 1)) & 15
            q[:, :, 128 * g + 32 * k:128 * g + 32 * k + 32] = lo | (blk[:, :, 128 + 32 * g:160 + 32 * g] >> (2 * k) & 3) << 4
    wt = half(q * 2.0 ** -24 * np.repeat(s, 16, 2) + np.repeat(off, 16, 2)).reshape(rows, cols) * factor[:, None]
    scale = 2.0 ** (np.frexp(np.abs(x).max(1).astype(np.float64))[1] - 10)[:, None]
    ref = half(x / scale) * scale @ wt.T
    assert np.linalg.norm(y - ref) <= 3e-6 * np.linalg.norm(ref)


# Rows whose blocks differ widely, and calls in which only the small blocks count: the activations are 0 where a row's large block
# lies, or smaller there by as much as its scale is larger.  A row's weights are expanded over one factor, so the small blocks would
# keep few of their bits: from a spread on (2^5 and 2^8 lie on either side) the matrix is expanded another way.  Scales near
# fp16's largest, negative ones, blocks whose minima or a single sub-scale make them large; all ways of writing out.  The bound is
# assert_product's, whatever the spread.
def unequal_blocks(t, rows, cols, ratio, seed, kind="d", d=1e-3):
    bb, nb = S.BLOCK_BYTES[t], cols // 256
    w = S.gen_weight(t, rows, cols, seed=seed, d_range=(1e-3, 2e-3)).reshape(rows, nb, bb).copy()
    at = 208 if t == S.Q6_K else 0
    for o in ([208] if t == S.Q6_K else [0, 2]):
        f = w[:, :, o:o + 2].copy().view(np.float16).astype(np.float64) * (d / 1e-3)
        w[:, :, o:o + 2] = f.astype(np.float16).view(np.uint8)
    big = np.float16(1.5 * d * 2.0 ** ratio)
    if kind == "d" or t == S.Q6_K:
        w[:, 1, at:at + 2] = np.array([big]).view(np.uint8)
        w[1::3, 1, at + 1] |= 0x80  # negative
    else:  # "dmin": its minima alone make the block large; "unused": not even they, being 0 times that
        w[:, 1, 2:4] = np.array([big]).view(np.uint8)
        if kind == "unused":
            w[:, 1, 4:16] = np.array([1, 2, 3, 4, 0, 0, 0, 0, 7, 8, 9, 10], np.uint8)
    return w.reshape(-1)


@pytest.mark.parametrize("t", [S.Q4_K, S.Q6_K])
@pytest.mark.parametrize("rows,cols,m", [(200, 1024, 9), (4096, 2048, 33), (600, 1024, 130), (130, 8192, 300)])
@pytest.mark.parametrize("ratio,d", [(0, 1e-3), (5, 1e-3), (8, 1e-3), (12, 1e-3), (16, 1e-3), (15, 1.2), (12, 2e-5)])
def test_matmul_unequal_blocks(t, rows, cols, m, ratio, d):
    w = unequal_blocks(t, rows, cols, ratio, seed=155, d=d)
    wd = O.dequant_matrix(t, w, rows, cols)
    for small in (0.0, 2.0 ** -ratio):
        x = S.gen_acts(m, cols, seed=156)
        x[:, 256:512] *= np.float32(small)
        assert_product(device_product(t, w, x, rows, cols, m), x, wd, half=True)


@pytest.mark.parametrize("kind", ["dmin", "unused"])
def test_matmul_large_minima(kind):
    t, rows, cols, m = S.Q4_K, 264, 1024, 24
    for ratio in (4, 9, 14, 18):
        w = unequal_blocks(t, rows, cols, ratio, seed=157, kind=kind)
        x = S.gen_acts(m, cols, seed=158)
        x[:, 256:512] = 0
        assert_product(device_product(t, w, x, rows, cols, m), x, O.dequant_matrix(t, w, rows, cols), half=True)


# One marked matrix among those of a call: gate or up of a feed-forward block, an expert's; and that it is the marked calls, and they
# alone, that go the other way.
@pytest.mark.parametrize("t", [S.Q4_K, S.Q6_K])
def test_unequal_blocks_among_others(t):
    import torch
    from launches import launched
    from oxillama_b200 import moe
    from oxillama_b200.device import DeviceWeights, check_device_status, ffn
    hidden, inter, m, n = 512, 768, 40, 4
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    WIDE = 0x100

    def formats(call):
        return [k.ints[0] for k in launched(call) if k.name == "qk_gemm_tc_kernel"]

    def block(x, g, u, d):
        hg = x @ g.T
        return (hg / (1 + np.exp(-hg)) * (x @ u.T)) @ d.T

    x = S.gen_acts(m, hidden, seed=162) * np.float32(0.25)
    x[:, 256:512] *= np.float32(2.0 ** -12)
    xd, y = torch.from_numpy(x).cuda(), torch.empty((m, hidden), device="cuda")
    for marked in (None, 0, 1, 2):
        ws = [unequal_blocks(t, r, c, 12 if k == marked else 0, seed=163 + k) for k, (r, c) in enumerate(shapes)]
        if marked == 2:  # its large block would drown the others
            ws[2] = unequal_blocks(t, hidden, inter, -12, seed=165)
        dw = [DeviceWeights(t, w, r, c) for w, (r, c) in zip(ws, shapes)]
        g, u, d = (O.dequant_matrix(t, w, r, c).astype(np.float64) for w, (r, c) in zip(ws, shapes))
        assert formats(lambda: ffn(*dw, xd, y, m)) == [t | (WIDE if marked in (0, 1) else 0), t | (WIDE if marked == 2 else 0)]
        ref = block(x.astype(np.float64), g, u, d)
        y.fill_(float("nan"))
        ffn(*dw, xd, y, m)
        check_device_status()
        assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()
        for w in dw:
            w.free()
    for marked in (None, 1, 2):
        w = [[unequal_blocks(t, r, c, (12 if k == 1 else -12) if k == marked and e == 2 else 0, seed=170 + 3 * e + k) for e in range(n)]
             for k, (r, c) in enumerate(shapes)]
        logits = S.gen_acts(m, n, seed=168)
        ids, wts = (v.cpu().numpy() for v in moe.route(torch.from_numpy(logits).cuda(), 2))
        ref = np.zeros((m, hidden))
        for e in range(n):
            g, u, d = (O.dequant_matrix(t, ws[e], r, c).astype(np.float64) for ws, (r, c) in zip(w, shapes))
            at, slot = np.nonzero(ids == e)
            np.add.at(ref, at, wts[at, slot][:, None] * block(x[at].astype(np.float64), g, u, d))
        ex = moe.MoeExperts(t, *w, hidden, inter, n)
        ld = torch.from_numpy(logits).cuda()
        assert formats(lambda: ex.forward(ld, xd, y, 2)) == [t | (WIDE if marked == 1 else 0), t | (WIDE if marked == 2 else 0)]
        y.fill_(float("nan"))
        ex.forward(ld, xd, y, 2)
        check_device_status()
        ex.free()
        assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()


# Chunks of several k-tiles through a ring that hands its stages back one by one, where a CTA has more tiles than the ring stages
# (twelve at most): every depth of the ring is reached, passed by one chunk and gone round, with one, two and four groups of warps;
# matrices with a chunk that some CTAs do not have; and rows of a single k-tile, which go to a kernel without the hand-over where the
# format has one.  (Kernels: without it 0, with it 1.)
@pytest.mark.parametrize("t,m,cols", [(S.Q4_K, 1, 16384), (S.Q4_K, 2, 14336), (S.Q4_K, 4, 8448), (S.Q8_0, 1, 12288), (S.Q6_K, 1, 8192),
                                      (S.Q6_K, 2, 12032), (S.Q4_0, 3, 8192), (S.IQ4_XS, 1, 8448), (S.Q5_K, 4, 12288), (S.Q3_K, 2, 8448),
                                      (S.Q2_K, 2, 12288)])
def test_decode_ring_by_tile(t, m, cols):
    from launches import sm_count
    sms, ktiles = sm_count(), -(-cols // 4096)
    most = -(-13 // ktiles)  # chunks whose tiles are more than any ring holds
    for chunks in (1, 2, 3, most, most + 1):
        rows = 8 * sms * chunks - (1000 if chunks == most else 3)
        w = S.gen_weight(t, rows, cols, seed=161)
        x = S.gen_acts(m, cols, seed=162)
        ks = []
        y = device_product(t, w, x, rows, cols, m, ks)
        assert ks[-1].name == "qk_gemv_imma_kernel" and ks[-1].ints[-1] == 1, ks
        assert_product(y, x, O.dequant_matrix(t, w, rows, cols), half=False)
        assert np.array_equal(y, device_product(t, w, x, rows, cols, m))


@pytest.mark.parametrize("t,m,by_tile", [(S.Q4_K, 3, 0), (S.Q4_K, 4, 1), (S.Q4_0, 3, 0), (S.Q4_0, 2, 1), (S.Q3_K, 2, 0), (S.Q2_K, 2, 0), (S.Q2_K, 1, 1),
                                         (S.Q8_0, 3, 1), (S.IQ4_XS, 2, 0), (S.Q5_K, 3, 0), (S.Q5_K, 4, 1), (S.Q6_K, 2, 1)])
def test_decode_ring_of_single_tiles(t, m, by_tile):
    for rows, cols in ((320, 1280), (9481, 3584), (2400, 4096)):
        w = S.gen_weight(t, rows, cols, seed=163)
        x = S.gen_acts(m, cols, seed=164)
        ks = []
        y = device_product(t, w, x, rows, cols, m, ks)
        assert [(k.name, k.ints[0], k.ints[-1]) for k in ks if k.name != "qk_xsplit_kernel"] == [("qk_gemv_imma_kernel", m, by_tile)], ks
        assert_product(y, x, O.dequant_matrix(t, w, rows, cols), half=False)


# What DeviceWeights.gemv / .gemm take and refuse is the same with the extension and without it.
@pytest.mark.parametrize("native", [True, False])
def test_device_call_arguments(native, monkeypatch):
    import torch
    from oxillama_b200 import device
    from oxillama_b200.kernels import QuantError
    assert device._native is not None, "the extension is not built"
    rows, cols = 64, 512
    w = S.gen_weight(S.Q4_K, rows, cols, seed=171)
    dw = device.DeviceWeights(S.Q4_K, w, rows, cols)
    if not native:
        dw._call = None
    xn = S.gen_acts(3, cols, seed=172)
    wd = O.dequant_matrix(S.Q4_K, w, rows, cols)
    x = torch.from_numpy(xn).cuda()

    class Sub(torch.Tensor):
        pass

    side = torch.cuda.Stream()
    for xs, stream in ((x, None), (x.clone().requires_grad_(), None), (torch.nn.Parameter(x.clone()), None), (x.clone().as_subclass(Sub), None),
                       (x, side)):
        y = torch.full((3, rows), float("nan"), device="cuda")
        torch.cuda.synchronize()
        dw.gemv(xs[0].detach() if xs.requires_grad else xs[0], y[0], stream=stream)
        torch.cuda.synchronize()
        assert_product(y[:1].cpu().numpy(), xn[:1], wd, half=False)
        dw.gemm(xs, y, 3, stream=stream)
        torch.cuda.synchronize()
        assert_product(y.cpu().numpy(), xn, wd, half=False)
    wide = torch.full((3, 200), 7.0, device="cuda")  # a block of columns of a wider result; sizes as numpy gives them
    dw.gemm(x, wide, np.int64(3), ldy=np.int32(200), col_offset=100)
    got = wide.cpu().numpy()
    assert_product(got[:, 100:164], xn, wd, half=False)
    assert np.all(got[:, :100] == 7) and np.all(got[:, 164:] == 7)
    y = torch.empty(3, rows, device="cuda")
    for bad in (x.double(), x.cpu(), x.t(), x[:, ::2], x.half()):
        with pytest.raises(TypeError):
            dw.gemv(bad, y)
        with pytest.raises(TypeError):
            dw.gemm(bad, y, 3)
    with pytest.raises(TypeError):
        dw.gemv(x, y.t())
    with pytest.raises(QuantError):
        dw.gemv(x[0, :500].contiguous(), y)
    with pytest.raises(QuantError):
        dw.gemm(x, y, 4)
    with pytest.raises(QuantError):
        dw.gemm(x, y, 3, ldy=rows - 1)
    with pytest.raises(AttributeError):
        dw.gemv(xn, y)
    dw.gemm(x, y, 0)
    dw.free()
    with pytest.raises(QuantError):
        dw.gemv(x, y)


# silu(g) * u by clusters of eight and four CTAs a row of more than 8192 columns, as long as they are no more than twice the SMs
# (148: up to 37 and 74 rows), by one from there on and for shorter rows.  8448 and 8500 columns are 33 and 34 spans: of eight parts
# of five spans the last is empty, its CTA comes to the meeting at once; 9248 leaves the last part short and its last span ragged.  Every format,
# Q4_K with its order of 64 columns.  Many calls in turn give the same bits.
# The bound: three chained products, each within 1e-3 of its largest value.
@pytest.mark.parametrize("t,hidden,inter,ms", [(S.Q4_K, 256, 512, (5, 18, 38)), (S.Q8_0, 256, 2336, (18, 37)), (S.IQ4_XS, 256, 4864, (18, 19)),
                                               (S.Q4_0, 512, 1312, (9, 30)), (S.Q6_K, 256, 8448, (5, 37, 38, 74, 75)), (S.Q8_0, 256, 9248, (37, 38)),
                                               (S.Q4_K, 256, 8500, (5, 37, 38, 74, 75, 149)), (S.Q4_K, 256, 14336, (8, 38)), (S.IQ4_XS, 256, 8448, (5, 37, 38, 75)),
                                               (S.Q4_0, 256, 9248, (5, 74))])
def test_ffn_conversion_by_clusters(t, hidden, inter, ms):
    import torch
    from launches import launched, sm_count
    from oxillama_b200.device import DeviceWeights, check_device_status, ffn
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    ws = [S.gen_weight(t, r, c, seed=181, stream=i, d_range=(1e-3, 3e-3)) for i, (r, c) in enumerate(shapes)]
    g, u, d = (O.dequant_matrix(t, w, r, c).astype(np.float64) for w, (r, c) in zip(ws, shapes))
    dw = [DeviceWeights(t, w, r, c) for w, (r, c) in zip(ws, shapes)]
    for m in ms:
        x = S.gen_acts(m, hidden, seed=182) * np.float32(0.25)
        hg = x.astype(np.float64) @ g.T
        ref = (hg / (1 + np.exp(-hg)) * (x.astype(np.float64) @ u.T)) @ d.T
        xd, y = torch.from_numpy(x).cuda(), torch.full((m, hidden), float("nan"), device="cuda")
        cl = next((c for c in (8, 4) if inter > 8192 and m * c <= 2 * sm_count()), 1)
        glu, = [k for k in launched(lambda: ffn(*dw, xd, y, m)) if k.name == "qk_glu16_kernel"]
        assert glu.ints[-1] == cl and glu.grid[0] == m * cl, glu
        y.fill_(float("nan"))
        ffn(*dw, xd, y, m)
        check_device_status()
        assert np.abs(y.cpu().numpy() - ref).max() <= 3e-3 * np.abs(ref).max()
        again = torch.empty((20, m, hidden), device="cuda")
        for z in again:
            ffn(*dw, xd, z, m)
        check_device_status()
        assert all(torch.equal(z, y) for z in again)
    for w in dw:
        w.free()


# Experts' jobs of one row (a single token) and of two, whose scales go to the lanes by different ways: one span of columns for
# eight warps, one that leaves some of them out, a second tile with a ragged last block; rows that are no multiple of a chunk's.
# Against each expert's own product in f64.  The bound is that of f32-grade sums for each of the three products (top of this file;
# a block's largest value is up to 2 times the root mean square of these weights, 2.5 times that of these activations and 4 times that
# of silu(g) u), which are independent, and half as much again for what silu makes of an error.  (7e-6 to 3e-5; with two digits of the
# activations for three the result is off by 2e-5 to 8e-5 at the same sizes.)
@pytest.mark.parametrize("t", [S.Q4_K, S.Q6_K])
@pytest.mark.parametrize("hidden,inter", [(256, 40), (1284, 264), (4352, 2304)])
def test_moe_decode_one_row(t, hidden, inter):
    import torch
    from oxillama_b200 import moe
    from oxillama_b200.device import check_device_status
    n, top_k = 4, 2
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    w = [[S.gen_weight(t, r, c, seed=151, stream=3 * e + k, d_range=(1e-4, 3e-4)) for e in range(n)] for k, (r, c) in enumerate(shapes)]
    logits = torch.tensor([[3., 1., 2., 0.], [3., 0., 1., 2.]])  # a job of two rows and two of one
    ex = moe.MoeExperts(t, *w, hidden, inter, n)
    for tokens in (1, 2):
        x = S.gen_acts(tokens, hidden, seed=152) * np.float32(0.25)
        ids, wts = (v.cpu().numpy() for v in moe.route(logits[:tokens].cuda(), top_k))
        ref = np.zeros((tokens, hidden))
        for tok in range(tokens):
            for e, wt in zip(ids[tok], wts[tok]):
                g, u, d = (O.dequant_matrix(t, ws[e], r, c).astype(np.float64) for ws, (r, c) in zip(w, shapes))
                hg = g @ x[tok]
                ref[tok] += wt * (d @ (hg / (1 + np.exp(-hg)) * (u @ x[tok])))
        y = torch.full((tokens, hidden), float("nan"), device="cuda")
        ex.forward(logits[:tokens].cuda(), torch.from_numpy(x).cuda(), y, top_k)
        check_device_status()
        sigma = [2.0 ** -23 * (1 + np.sqrt(2 * k / 32)) * 2 * a for k, a in ((hidden, 2.5), (hidden, 2.5), (inter, 4))]
        assert np.linalg.norm(y.cpu().numpy() - ref) <= 1.5 * np.linalg.norm(sigma) * np.linalg.norm(ref)
    ex.free()
