"""The tensor-core GEMM with split operands: edges of its tiles and chunks, packed alignments, ranges, streams, capture.

Tolerances (relative 2-norm): an accumulator takes 24 truncating steps of 2^-24 with f32 activations (three products of eight K = 16
steps), 16 with bf16, 32 with bf16 from K = 2048 on (two chunks), and grows with the root of the steps, so its sum is at most
steps * 2/3 * 2^-24 off: 9.5e-7, 6.4e-7, 1.27e-6 (_bound); accumulators add up in quadrature, and so do their f32 sums.  Where 1e-6 is
written out it lies above what the f32 bound gives and below that of bf16 pairs, which stay at half of theirs.
"""
import numpy as np
import pytest

from oracle import oracle as O
from gpu_util import run_matmul, to_dev

pytestmark = pytest.mark.gpu

FMTS = [O.FMT_Q4, O.FMT_Q8]


def _inputs(fmt, m, k, n, seed=0):
    rng = np.random.Generator(np.random.PCG64(seed + m + k + n))
    return O.synth_weights(fmt, k, n, seed=seed + 1), rng.standard_normal((m, k)).astype(np.float32)


def _dense(fmt, w, k, n):
    from meganeura_b200 import ops
    return ops.dequantize(fmt, w, k, n).astype(np.float64)


@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("fmt", FMTS)
# tokens: one group of 16, one tile, two tiles, three; k: odd block counts, a chunk and one block, several chunks;
# n: less than a tile, ragged, block counts of every remainder by 4
@pytest.mark.parametrize("m,k,n", [(1, 160, 1), (16, 256, 128), (17, 288, 33), (128, 416, 127), (129, 608, 129), (257, 1056, 259), (300, 4128, 70), (40, 8192, 2048)])
def test_edges(fmt, act, m, k, n):
    import torch
    from meganeura_b200 import ops
    w, x = _inputs(fmt, m, k, n)
    d = np.random.Generator(np.random.PCG64(3)).standard_normal((m, n)).astype(np.float32) if m % 2 else None
    xd = torch.from_numpy(x).cuda()
    if act == "bf16":
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    got = run_matmul(fmt, xd, w, k, n, addend=d, route="gemm")
    ops.device_status()
    want = x.astype(np.float64) @ _dense(fmt, w, k, n) + (0.0 if d is None else d)
    assert O.rel_l2(got, want) <= 1e-6


def test_unaligned_activations():
    import torch
    from meganeura_b200 import ops
    m, k, n = 33, 320, 65
    w, x = _inputs(O.FMT_Q4, m, k, n)
    for dtype in (torch.float32, torch.bfloat16):
        buf = torch.zeros(m * k + 1, device="cuda", dtype=dtype)
        a = buf[1:].reshape(m, k)
        a.copy_(torch.from_numpy(x))
        got = ops.matmul(O.FMT_Q4, a, to_dev(w), k, n, route="gemm").cpu().numpy()
        assert O.rel_l2(got, a.float().cpu().numpy().astype(np.float64) @ _dense(O.FMT_Q4, w, k, n)) <= 1e-6


@pytest.mark.parametrize("fmt", FMTS)
def test_ranges_of_rows(fmt):
    # rows of very different magnitude, and one whose chunks differ by 10^20: each keeps its own relative accuracy
    m, k, n = 20, 512, 130
    w, x = _inputs(fmt, m, k, n)
    x *= (10.0 ** np.linspace(-30, 30, m)).astype(np.float32)[:, None]
    x[7, :] = x[8, :]
    x[7, 128:] *= np.float32(1e-20)
    x[3] = 0
    got = run_matmul(fmt, x, w, k, n, route="gemm")
    want = x.astype(np.float64) @ _dense(fmt, w, k, n)
    for r in range(m):
        assert np.linalg.norm(got[r] - want[r]) <= 1e-6 * np.linalg.norm(want[r])


@pytest.mark.parametrize("fmt", FMTS)
def test_not_finite_and_large_scales_as_in_plain_f32(fmt):
    import torch
    from meganeura_b200 import ops
    m, k, n = 40, 384, 140
    w, x = _inputs(fmt, m, k, n)
    w = w.copy()
    x[3, 17], x[5, 200], x[9, 300] = np.inf, -np.inf, np.nan
    x[11, 5], x[11, 6] = np.inf, -np.inf
    x[13] = 3e38
    scales = w[:4 * (k // 32) * n].view(np.float16)[0::2] if fmt == O.FMT_Q4 else w.reshape(-1, 36)[:, :2].copy().view(np.float16)[:, 0]
    big = {4: 60000.0, 70: np.inf, 139: 700.0}                # columns
    for col, value in big.items():
        scales[col * (k // 32) + 2] = value
    if fmt == O.FMT_Q8:
        w.reshape(-1, 36)[:, :2] = scales[:, None].view(np.uint8).reshape(-1, 2)
    xd, wd = to_dev(x), to_dev(w)
    got = ops.matmul(fmt, xd, wd, k, n, route="gemm")
    ops.set_option("gemm.force_tiled", 1)
    try:
        plain = ops.matmul(fmt, xd, wd, k, n, route="gemm")
    finally:
        ops.set_option("gemm.force_tiled", 0)
    got, plain = got.cpu().numpy(), plain.cpu().numpy()
    finite = np.isfinite(plain)
    assert np.array_equal(np.isnan(got), np.isnan(plain)) and np.array_equal(np.isposinf(got), np.isposinf(plain)) and np.array_equal(np.isneginf(got), np.isneginf(plain))
    assert (np.abs(got[finite] - plain[finite]) <= 1e-4 * np.abs(plain[finite]).max(initial=0.0)).all()
    ordinary = [r for r in range(m) if r not in (3, 5, 9, 11, 13)]
    cols = [c for c in range(n) if c not in big]
    assert O.rel_l2(got[np.ix_(ordinary, cols)], plain[np.ix_(ordinary, cols)]) <= 2e-6


def test_two_streams_at_once():
    import torch
    from meganeura_b200 import ops
    shapes = [(O.FMT_Q4, 300, 1536, 2048), (O.FMT_Q8, 60, 4096, 512)]
    work = []
    for i, (fmt, m, k, n) in enumerate(shapes):
        w, x = _inputs(fmt, m, k, n, seed=i)
        xd, wd = to_dev(x), to_dev(w)
        work.append((fmt, xd, wd, k, n, ops.matmul(fmt, xd, wd, k, n, route="gemm"), torch.cuda.Stream()))
    torch.cuda.synchronize()
    outs = []
    for _ in range(10):
        for fmt, xd, wd, k, n, want, stream in work:
            with torch.cuda.stream(stream):
                outs.append((ops.matmul(fmt, xd, wd, k, n, route="gemm", stream=stream), want))
    torch.cuda.synchronize()
    assert all(torch.equal(got, want) for got, want in outs)          # sums do not depend on timing


def test_captured_in_a_graph():
    import torch
    from meganeura_b200 import ops
    fmt, m, k, n = O.FMT_Q4, 50, 1024, 300
    w, x = _inputs(fmt, m, k, n)
    xd, wd, out = to_dev(x), to_dev(w), torch.zeros((m, n), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.matmul(fmt, xd, wd, k, n, out=out, route="gemm")
    for seed in range(3):
        xd.copy_(torch.from_numpy(_inputs(fmt, m, k, n, seed=seed)[1]))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ops.matmul(fmt, xd, wd, k, n, route="gemm"))


def _bound(act, k):
    """Truncating steps per accumulator (two or three products of eight, two chunks of bf16 from K = 2048 on), see above."""
    return (24 if act == "f32" else 32 if k >= 2048 else 16) * 2 / 3 * 2.0 ** -24 + 1e-8


def _q4_weights(kind, k, n, seed, zero_at=()):
    """Minima that have nothing to do with -8 d; rows of W in `zero_at` dequantize to exactly 0 (not for kind "quantized")."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "quantized":
        from meganeura_b200 import ops
        return ops.quantize(O.FMT_Q4, rng.standard_normal((k, n)).astype(np.float32) * 0.02)
    # d of 7 bits, so that its multiples up to 15 are exact in f16
    d = np.exp(rng.uniform(np.log(1e-3), np.log(1e-1), size=(n, k // 32))).astype(np.float32)
    d = (d.view(np.uint32) >> 17 << 17).view(np.float32)
    zero = {"seven": 7, "plus": 0, "above": 15}[kind]
    codes = rng.integers(0, 16, size=(k, n), dtype=np.uint8)
    m = -zero * d if zero else d * rng.integers(-20, 21, size=d.shape).astype(np.float32)
    codes[list(zero_at)] = zero
    return O.pack_q4_np(codes, d.astype(np.float16).view(np.uint16), m.astype(np.float16).view(np.uint16))


@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("kind", ["seven", "plus", "above", "quantized"])
@pytest.mark.parametrize("m,k,n", [(20, 160, 70), (33, 288, 129), (40, 2176, 70), (17, 4128, 200), (130, 2048, 33)])
def test_q4_minima(kind, act, m, k, n):
    import torch
    w, x = _q4_weights(kind, k, n, m + k), _inputs(O.FMT_Q4, m, k, n)[1]
    xd = to_dev(x)
    if act == "bf16":
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    got = run_matmul(O.FMT_Q4, xd, w, k, n, route="gemm")
    assert O.rel_l2(got, x.astype(np.float64) @ _dense(O.FMT_Q4, w, k, n)) <= _bound(act, k)


@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("kind", ["seven", "above", "q8"])
@pytest.mark.parametrize("size", [1e3, 1e5])
def test_large_activation_at_a_weight_of_zero(kind, act, size):
    """It adds nothing to a sum, so it may not add an error either: in every row, relative to the row's own result."""
    import torch
    m, k, n = 24, 2176, 150
    at = range(5, k, 128)
    fmt = O.FMT_Q8 if kind == "q8" else O.FMT_Q4
    w, x = _inputs(fmt, m, k, n)
    if kind == "q8":
        w = w.copy()
        blocks = w.reshape(n, k // 32, 36)
        for kk in at:
            blocks[:, kk // 32, 4 + kk % 32] = 0
    else:
        w = _q4_weights(kind, k, n, 9, at)
    assert (_dense(fmt, w, k, n)[list(at)] == 0).all()
    x[:, list(at)] = size * np.where(np.arange(m) % 2, 1, -1)[:, None]
    xd = to_dev(x)
    if act == "bf16":
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    got = run_matmul(fmt, xd, w, k, n, route="gemm")
    want = x.astype(np.float64) @ _dense(fmt, w, k, n)
    for r in range(m):
        assert O.rel_l2(got[r], want[r]) <= _bound(act, k)


@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("fmt", FMTS)
def test_nothing_but_nan_and_infinities(fmt, act):
    """Every sum of a long K takes the way of those that are not finite; no bounded wait may run out meanwhile."""
    import torch
    from meganeura_b200 import ops
    m, k, n = 48, 4096, 300
    w, x = _inputs(fmt, m, k, n)
    x[:] = np.nan
    x[40:44] = np.inf                                         # signs of the weights decide: NaN wherever both come up
    x[44] = 1.0
    x[44, k - 1] = np.nan                                     # the last element
    x[45:] = 0.5                                              # ordinary rows beside them
    d = np.ones((m, n), dtype=np.float32)
    xd = to_dev(x).to(torch.bfloat16) if act == "bf16" else to_dev(x)
    got = run_matmul(fmt, xd, w, k, n, addend=d, route="gemm")
    ops.device_status()
    assert np.isnan(got[:45]).all()
    assert O.rel_l2(got[45:], x[45:].astype(np.float64) @ _dense(fmt, w, k, n) + 1.0) <= _bound(act, k)


@pytest.mark.parametrize("fmt", FMTS)
def test_infinities_in_place(fmt):
    """The addend is the output: sums that are computed again read it before it is overwritten."""
    import torch
    from meganeura_b200 import ops
    m, k, n = 150, 288, 260
    w, x = _inputs(fmt, m, k, n)
    x[7, 3] = x[140, 200] = np.inf
    xd, wd = to_dev(x), to_dev(w)
    out = torch.full((m, n), 2.0, device="cuda")
    want = ops.matmul(fmt, xd, wd, k, n, addend=out.clone(), route="gemm")
    ops.matmul(fmt, xd, wd, k, n, addend=out, out=out, route="gemm")
    torch.cuda.synchronize()
    assert torch.equal(torch.nan_to_num(out, nan=7.0), torch.nan_to_num(want, nan=7.0)) and bool(torch.isinf(out[[7, 140]]).any())


@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("fmt", FMTS)
# one value per 128 k so much larger than the others; 2^29 (bf16: 2^27) is where plain f32 sums take over
@pytest.mark.parametrize("size", [2.0 ** 20, 2.0 ** 26, 2.0 ** 28, 2.0 ** 33, 2.0 ** 60, 2.0 ** 100])
def test_span_of_magnitudes(fmt, act, size):
    """A large activation at weights of zero leaves the small ones their bits.

    Down to 2^-29 of the largest value an f32 keeps 22 bits, 2^-23 of its value at most; that adds in quadrature to the sums.
    Plain f32 sums in order of k are sqrt(k / 3) * 2^-24 off."""
    import torch
    m, k, n = 24, 2176, 150
    at = list(range(70, k, 128))
    if fmt == O.FMT_Q4:
        w = _q4_weights("seven", k, n, 4, at)
    else:
        w = _inputs(fmt, m, k, n)[0].copy()
        for kk in at:
            w.reshape(n, k // 32, 36)[:, kk // 32, 4 + kk % 32] = 0
    x = _inputs(fmt, m, k, n)[1]
    x = np.sign(x) * np.maximum(np.abs(x), 0.5).astype(np.float32)
    x[:, at] = size
    x[1::2, at] = -size
    x[5] = 0                                                  # nothing but the large ones
    x[5, at] = size
    xd = to_dev(x)
    if act == "bf16":
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    got = run_matmul(fmt, xd, w, k, n, route="gemm")
    want = x.astype(np.float64) @ _dense(fmt, w, k, n)
    assert (got[5] == 0).all()
    bound = max(_bound(act, k), 2 * (k / 3) ** 0.5 * 2.0 ** -24)
    for r in range(m):
        assert r == 5 or O.rel_l2(got[r], want[r]) <= bound


@pytest.mark.parametrize("fmt", FMTS)
# shapes that do not stream and ones that do, each with the rows from which on the GEMM takes them
@pytest.mark.parametrize("m,k,n", [(16, 288, 193), (16, 576, 1001), (1, 6176, 193), (1, 2912, 2099), (2, 8800, 3841), (3, 12320, 1001), (5, 1056, 4096), (16, 4128, 64), (16, 4096, 4896)])
def test_few_rows_lose_nothing(fmt, m, k, n):
    """Up to 16 f32 rows that leave the GEMV for the GEMM come no farther from the exact product."""
    import torch
    from meganeura_b200 import ops
    w, x = _q4_weights("quantized", k, n, 1) if fmt == O.FMT_Q4 else _inputs(fmt, m, k, n)[0], _inputs(fmt, m, k, n)[1]
    want = x.astype(np.float64) @ _dense(fmt, w, k, n)
    got = {r: run_matmul(fmt, x, w, k, n, route=r) for r in ("auto", "gemv", "gemm")}
    again = run_matmul(fmt, x, w, k, n, route="gemm")
    assert np.array_equal(got["gemm"], again)                 # sums do not depend on which CTA comes last
    assert O.rel_l2(got["gemm"], want) <= O.rel_l2(got["gemv"], want)
    assert O.rel_l2(got["auto"], want) <= O.rel_l2(got["gemv"], want)


@pytest.mark.parametrize("fmt", FMTS)
# below, at and above the line where bf16 rows of K = 128 leave the tiled kernel; fewer than 64 rows stay
@pytest.mark.parametrize("m,n,split", [(64, 16384, False), (64, 16388, True), (200, 5251, True), (1030, 1030, True), (63, 17000, False)])
def test_one_chunk_of_bf16(fmt, m, n, split):
    import torch
    from meganeura_b200 import ops
    k = 128
    w = _q4_weights("quantized", k, n, m) if fmt == O.FMT_Q4 else _inputs(fmt, m, k, n)[0]
    xd, wd = to_dev(_inputs(fmt, m, k, n)[1]).to(torch.bfloat16), to_dev(w)
    got = ops.matmul(fmt, xd, wd, k, n)
    ops.set_option("gemm.force_tiled", 1)
    try:
        tiled = ops.matmul(fmt, xd, wd, k, n)
    finally:
        ops.set_option("gemm.force_tiled", 0)
    assert torch.equal(got, tiled) != split
    want = xd.double().cpu().numpy() @ _dense(fmt, w, k, n)
    assert O.rel_l2(got.cpu().numpy(), want) <= _bound("bf16", k)


def test_captured_graph_serves_as_a_child_graph():
    """Kernels only: a graph that holds allocation nodes is refused as a child graph."""
    import torch
    from cuda.bindings import runtime as cudart
    from meganeura_b200 import ops

    def call(fn, *args):
        out = fn(*args)
        assert out[0] == cudart.cudaError_t.cudaSuccess, (fn.__name__, out[0])
        return out[1] if len(out) == 2 else out[1:]
    shapes = [(O.FMT_Q4, 40, 1024, 300), (O.FMT_Q8, 200, 2048, 700), (O.FMT_Q4, 130, 512, 1000)]
    work = []
    for i, (fmt, m, k, n) in enumerate(shapes):
        w, x = _inputs(fmt, m, k, n, seed=i)
        xd, wd = to_dev(x), to_dev(w)
        work.append((fmt, xd, wd, k, n, torch.zeros((m, n), device="cuda"), ops.matmul(fmt, xd, wd, k, n, route="gemm")))
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    side = torch.cuda.Stream()
    with torch.cuda.graph(graph):                             # two streams of one capture, two calls on one of them
        side.wait_stream(torch.cuda.current_stream())
        for i, (fmt, xd, wd, k, n, out, _) in enumerate(work):
            with torch.cuda.stream(side if i == 1 else torch.cuda.current_stream()):
                ops.matmul(fmt, xd, wd, k, n, out=out, route="gemm")
        torch.cuda.current_stream().wait_stream(side)
    raw = cudart.cudaGraph_t(graph.raw_cuda_graph())
    parent = call(cudart.cudaGraphCreate, 0)
    call(cudart.cudaGraphAddChildGraphNode, parent, None, 0, raw)
    exe = call(cudart.cudaGraphInstantiate, parent, 0)
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(3):
        for item in work:
            item[5].zero_()
        call(cudart.cudaGraphLaunch, exe, stream)
        torch.cuda.synchronize()
        assert all(torch.equal(out, want) for *_, out, want in work)
    call(cudart.cudaGraphExecDestroy, exe)
    call(cudart.cudaGraphDestroy, parent)
    ops.device_status()


def test_workspace_of_a_captured_graph_goes_back_with_it():
    import torch
    from meganeura_b200 import ops
    fmt, m, k, n = O.FMT_Q4, 1024, 4096, 512
    w, x = _inputs(fmt, m, k, n)
    xd, wd, out = to_dev(x), to_dev(w), torch.zeros((m, n), device="cuda")

    def capture():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.matmul(fmt, xd, wd, k, n, out=out, route="gemm")
        graph.replay()
        torch.cuda.synchronize()
        del graph
        torch.cuda.synchronize()
        ops.matmul(fmt, xd, wd, k, n, out=out, route="gemm")  # the call that follows returns it
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    capture()
    free = [capture() for _ in range(6)]
    assert min(free) >= free[0] - (8 << 20)                   # a workspace of this size is 40 MB


@pytest.mark.parametrize("fmt", FMTS)
def test_session_with_a_prompt_captured(fmt):
    """A session of matmuls of many rows steps, captures and replays on new inputs."""
    import meganeura_b200 as mg
    m, k, n = 37, 512, 384
    w1, w2 = _inputs(fmt, m, k, n)[0], _inputs(fmt, m, n, k, seed=3)[0]
    g = mg.Graph()
    x = g.input("x", [m, k])
    param = g.parameter_q4 if fmt == O.FMT_Q4 else g.parameter_q8
    y = g.matmul(g.matmul(x, param("w1", [k, n])), param("w2", [n, k]))
    g.set_outputs([y])
    s = mg.build_inference_session(g)
    s.upload_param("w1", w1)
    s.upload_param("w2", w2)
    d1, d2 = _dense(fmt, w1, k, n), _dense(fmt, w2, n, k)
    for seed in range(4):
        a = _inputs(fmt, m, k, n, seed=seed)[1]
        s.set_input("x", a)
        if seed == 1:
            s.capture()
        s.step()
        s.wait()
        got = s.read_output(m * k).reshape(m, k)
        assert O.rel_l2(got, a.astype(np.float64) @ d1 @ d2) <= 2 * _bound("f32", k)
