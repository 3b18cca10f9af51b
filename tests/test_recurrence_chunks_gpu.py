"""Time mixing and mLSTM in chunks on the tensor cores: portions of 64 and more tokens whose gated output is rounded to bf16.

The output is read through a linear layer with an identity matrix, so it is bf16: half an ulp is 2^-9 of the value; the rest of
the tolerance of 2^-8 of the largest value is far above what three-part products leave.
"""
import numpy as np
import pytest

from oracle import petotar_oracle as P
from graph_util import close, rng_of, run, session
from petotar_util import bf16_round

pytestmark = pytest.mark.gpu

# chunks of 16: a multiple, one more, one less; several segments; short portions in between take the token-by-token kernels
PORTIONS = (64, 1, 65, 30, 700, 79, 2)


def _identity(g, x, n, params):
    params["eye"] = np.eye(n, dtype=np.float32)
    return g.matmul_bt(x, g.parameter_bf16("eye", [n, n]))


@pytest.mark.parametrize("heads,dim,vdim,cap", [(2, 32, 48, 12.0), (3, 24, 8, 2.0), (1, 128, 256, 15.0), (2, 64, 100, 4.0), (1, 256, 16, 8.0), (2, 10, 128, 6.0)])
def test_mlstm(heads, dim, vdim, cap):
    import meganeura_b200 as mg
    from meganeura_b200._lib import FMT_BF16, GATE_SIGMOID, ROWS_TOKENS, lib
    r = rng_of(heads, dim, vdim)
    n, nv, rows = heads * dim, heads * vdim, max(PORTIONS)
    tabs = {"q": r.standard_normal((90, n)), "k": r.standard_normal((90, n)), "v": r.standard_normal((90, nv)), "g": r.standard_normal((90, nv)),
              "i": r.standard_normal((90, heads)) * 6 - 2, "f": r.standard_normal((90, heads)) * 6 + 3}
    tabs = {c: a.astype(np.float32) for c, a in tabs.items()}
    hw = r.standard_normal(nv).astype(np.float32)
    g = mg.Graph()
    ids = g.input_u32_rows("ids", rows, ROWS_TOKENS)
    e = {c: g.embedding_scaled(ids, g.parameter(c, list(a.shape)), 1.0) for c, a in tabs.items()}
    state = g.parameter("state", [lib.mgq_mlstm_state_elements(heads, dim, vdim)])
    o = g.mlstm(e["q"], e["k"], e["v"], e["i"], e["f"], state, heads, cap)
    params = {**tabs, "hw": hw}
    y = _identity(g, g.head_gate(o, e["g"], heads, g.parameter("hw", [nv]), 1e-5, GATE_SIGMOID, FMT_BF16), nv, params)
    s = session(g, [y], params)
    S, nn, m, at = np.zeros((heads, dim, vdim)), np.zeros((heads, dim)), np.zeros(heads), 0
    for cnt in PORTIONS:
        toks = (np.arange(at, at + cnt) * 11) % 90
        at += cnt
        s.set_rows(ROWS_TOKENS, cnt)
        s.set_input_u32("ids", toks)
        got = run(s, (cnt, nv))
        li, lf = P.mlstm_gates(tabs["i"][toks].astype(np.float64), tabs["f"][toks].astype(np.float64), cap)
        oo = P.mlstm_scan(tabs["q"][toks].reshape(cnt, heads, dim) * dim ** -0.5, tabs["k"][toks].reshape(cnt, heads, dim).astype(np.float64),
                          tabs["v"][toks].reshape(cnt, heads, vdim).astype(np.float64), li, lf, S, nn, m)
        close(got, P.unit_rms(oo, 1e-5).reshape(cnt, nv) * hw * P.sigmoid(tabs["g"][toks]), 2 ** -8)


@pytest.mark.parametrize("heads,dim,rank", [(2, 32, 8), (3, 24, 5), (1, 64, 200), (2, 128, 4), (4, 8, 16), (1, 256, 3)])
def test_wkv(heads, dim, rank):
    import meganeura_b200 as mg
    from meganeura_b200._lib import FMT_BF16, GATE_SILU, ROWS_TOKENS, lib
    r = rng_of(heads, dim, rank)
    n, rows, width = heads * dim, max(PORTIONS), 64
    tabs = {c: r.standard_normal((90, n)).astype(np.float32) for c in "rkvg"}
    tabs["low"] = r.standard_normal((90, width)).astype(np.float32)
    mus = r.uniform(0, 1, (1, width)).astype(np.float32)
    w1 = bf16_round(r.standard_normal((rank, width)).astype(np.float32) * width ** -0.5 * 2)
    w2 = bf16_round(r.standard_normal((n, rank)).astype(np.float32) * min(1.0, (5 / rank) ** 0.5))
    w0, u, hw = r.uniform(-5, 0, n).astype(np.float32), r.standard_normal(n).astype(np.float32), r.standard_normal(n).astype(np.float32)
    g = mg.Graph()
    ids = g.input_u32_rows("ids", rows, ROWS_TOKENS)
    e = {c: g.embedding_scaled(ids, g.parameter(c, list(a.shape)), 1.0) for c, a in tabs.items()}
    shift = g.parameter("shift", [2, width])
    mix = g.token_shift(e["low"], [g.parameter("mu", [width])], shift)
    decay = g.lora_decay(g.matmul_bt(g.slot(mix, 0), g.parameter_bf16("w1", [rank, width])), g.parameter_bf16("w2", [n, rank]), g.parameter("w0", [n]))
    o = g.wkv(e["r"], e["k"], e["v"], decay, g.parameter("u", [n]), g.parameter("state", [lib.mgq_wkv_state_elements(heads, dim)]), heads, shift)
    params = {**tabs, "mu": mus[0], "w1": w1, "w2": w2, "w0": w0, "u": u, "hw": hw}
    y = _identity(g, g.head_gate(o, e["g"], heads, g.parameter("hw", [n]), 1e-4, GATE_SILU, FMT_BF16), n, params)
    s = session(g, [y], params)
    prev, S, at = np.zeros(width), np.zeros((heads, dim, dim)), 0
    for cnt in PORTIONS:
        toks = (np.arange(at, at + cnt) * 7) % 90
        at += cnt
        s.set_rows(ROWS_TOKENS, cnt)
        s.set_input_u32("ids", toks)
        got = run(s, (cnt, n))
        h = tabs["low"][toks].astype(np.float64)
        low = P.token_shift(h, prev, mus[0])
        prev = h[-1]
        ro, ko, vo, go = (tabs[c][toks].astype(np.float64) for c in "rkvg")
        oo = P.wkv_scan(*(a.reshape(cnt, heads, dim) for a in (ro, ko, vo)), P.wkv_decay(low, w1, w2, w0).reshape(cnt, heads, dim), u.reshape(heads, dim), S)
        close(got, P.unit_rms(oo, 1e-4).reshape(cnt, n) * hw * go * P.sigmoid(go), 2 ** -8)



@pytest.mark.parametrize("kind,heads,dim,vdim", [("wkv", 2, 64, 64), ("wkv", 1, 128, 128), ("wkv", 1, 256, 256), ("mlstm", 2, 64, 100), ("mlstm", 1, 128, 256), ("mlstm", 1, 256, 64)])
def test_no_farther_from_64_bits_than_token_by_token(kind, heads, dim, vdim):
    """The second half of every head's keys repeats the first, and the queries of both cancel to 2^-12: what is left of an output
    shows the last bits of f32 sums through the bf16 rounding.  A long portion may be as far off as the same tokens in short
    ones, which take the token-by-token kernels; a third part left out, or sums that truncate, are three times as far and more."""
    import meganeura_b200 as mg
    from meganeura_b200._lib import FMT_BF16, GATE_SIGMOID, ROWS_TOKENS, lib
    r = rng_of(heads, dim, vdim, 5)
    rows, short, half, rank, delta = 512, 32, dim // 2, 4, 2.0 ** -12
    n, nv = heads * dim, heads * vdim

    def doubled(a):                                           # [.., heads, half] -> [.., heads * dim]
        return np.concatenate([a, a], -1).reshape(*a.shape[:-2], n).astype(np.float32)
    q1 = r.standard_normal((rows, heads, half))
    q = np.concatenate([q1, -q1 * (1 + delta * r.standard_normal(q1.shape))], -1).reshape(rows, n).astype(np.float32)
    tabs = {"q": q, "k": doubled(r.standard_normal((rows, heads, half))), "v": r.standard_normal((rows, nv)).astype(np.float32), "g": np.zeros((rows, nv), np.float32)}
    g = mg.Graph()
    ids = g.input_u32_rows("ids", rows, ROWS_TOKENS)
    params = {"hw": np.ones(nv, np.float32)}
    if kind == "mlstm":
        tabs |= {c: (r.standard_normal((rows, heads)) + b).astype(np.float32) for c, b in (("i", 0), ("f", 3))}
    else:
        tabs["low"] = (r.standard_normal((rows, rank)) * 0.3).astype(np.float32)
        params |= {"w2": bf16_round(doubled(r.standard_normal((rank, heads, half))).T.copy() * np.float32(0.2)), "w0": doubled(r.uniform(-6, -2, (heads, half))),
                   "u": doubled(r.standard_normal((heads, half)))}
    e = {c: g.embedding_scaled(ids, g.parameter(c, list(a.shape)), 1.0) for c, a in tabs.items()}
    if kind == "mlstm":
        o = g.mlstm(e["q"], e["k"], e["v"], e["i"], e["f"], g.parameter("state", [lib.mgq_mlstm_state_elements(heads, dim, vdim)]), heads, 15.0)
    else:
        decay = g.lora_decay(e["low"], g.parameter_bf16("w2", [n, rank]), g.parameter("w0", [n]))
        o = g.wkv(e["q"], e["k"], e["v"], decay, g.parameter("u", [n]), g.parameter("state", [lib.mgq_wkv_state_elements(heads, dim)]), heads)
    params |= tabs
    y = _identity(g, g.head_gate(o, e["g"], heads, g.parameter("hw", [nv]), 1e-20, GATE_SIGMOID, FMT_BF16), nv, params)
    d = {c: a.astype(np.float64) for c, a in tabs.items()}
    qq, kk, vv = d["q"].reshape(rows, heads, dim), d["k"].reshape(rows, heads, dim), d["v"].reshape(rows, heads, vdim)
    if kind == "mlstm":
        oo = P.mlstm_scan(qq * dim ** -0.5, kk, vv, *P.mlstm_gates(d["i"], d["f"], 15.0), np.zeros((heads, dim, vdim)), np.zeros((heads, dim)), np.zeros(heads))
    else:
        w = np.exp(-np.exp(np.tanh(d["low"]) @ params["w2"].astype(np.float64).T + params["w0"])).reshape(rows, heads, dim)
        oo = P.wkv_scan(qq, kk, vv, w, params["u"].astype(np.float64).reshape(heads, dim), np.zeros((heads, dim, dim)))
    want = P.unit_rms(oo, 1e-20).reshape(rows, nv) * 0.5
    off = {}
    for portion in (rows, short):
        s = session(g, [y], params)
        got = []
        for at in range(0, rows, portion):
            s.set_rows(ROWS_TOKENS, portion)
            s.set_input_u32("ids", np.arange(at, at + portion))
            got.append(run(s, (portion, nv)))
        off[portion] = np.linalg.norm(np.concatenate(got) - want) / np.linalg.norm(want)
    assert off[rows] <= 1.5 * off[short] + 2.0 ** -10         # bf16 rounding is in both


@pytest.mark.parametrize("kind", ["wkv", "mlstm"])
def test_long_portions_in_pieces(kind):
    """Portions longer than a piece of 2048 tokens give the bits that separate portions give, and the workspace does not grow with
    the capacity beyond a piece."""
    import torch
    import meganeura_b200 as mg
    from meganeura_b200._lib import FMT_BF16, FMT_F32, GATE_SIGMOID, ROWS_TOKENS, lib
    heads, dim, rank = 8, 32, 4
    r = rng_of(heads, dim)
    n = heads * dim
    tabs = {c: r.standard_normal((90, n)).astype(np.float32) for c in "qkvg"} | {c: r.standard_normal((90, heads)).astype(np.float32) + b for c, b in (("i", 0), ("f", 3))}
    tabs["low"] = (r.standard_normal((90, rank)) * 0.3).astype(np.float32)

    def build(rows, out_dtype):
        g = mg.Graph()
        ids = g.input_u32_rows("ids", rows, ROWS_TOKENS)
        e = {c: g.embedding_scaled(ids, g.parameter(c, list(a.shape)), 1.0) for c, a in tabs.items()}
        params = {**tabs, "hw": np.ones(n, np.float32)}
        if kind == "mlstm":
            o = g.mlstm(e["q"], e["k"], e["v"], e["i"], e["f"], g.parameter("state", [lib.mgq_mlstm_state_elements(heads, dim, dim)]), heads, 15.0)
        else:
            params |= {"w2": bf16_round(r.standard_normal((n, rank)).astype(np.float32) * 0.2), "w0": np.full(n, -4, np.float32), "u": np.ones(n, np.float32)}
            decay = g.lora_decay(e["low"], g.parameter_bf16("w2", [n, rank]), g.parameter("w0", [n]))
            o = g.wkv(e["q"], e["k"], e["v"], decay, g.parameter("u", [n]), g.parameter("state", [lib.mgq_wkv_state_elements(heads, dim)]), heads)
        y = _identity(g, g.head_gate(o, e["g"], heads, g.parameter("hw", [n]), 1e-5, GATE_SIGMOID, out_dtype), n, params) if out_dtype == FMT_BF16 else \
            g.head_gate(o, e["g"], heads, g.parameter("hw", [n]), 1e-5, GATE_SIGMOID, out_dtype)
        return session(g, [y], params)

    s, outs = build(4500, FMT_BF16), []
    for portions in ((4500,), (2048, 2048, 404)):
        s.reset_state()
        got, at = [], 0
        for cnt in portions:
            s.set_rows(ROWS_TOKENS, cnt)
            s.set_input_u32("ids", np.arange(at, at + cnt) * 7 % 90)
            got.append(run(s, (cnt, n)))
            at += cnt
        outs.append(np.concatenate(got))
    assert np.isfinite(outs[0]).all() and np.array_equal(outs[0], outs[1])
    del s

    def taken(rows, out_dtype):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        keep = build(rows, out_dtype)
        return before - torch.cuda.mem_get_info()[0]
    grown = {d: taken(40000, d) - taken(8000, d) for d in (FMT_BF16, FMT_F32)}
    buffers = 32000 * n * 2                                   # bf16 output beside an f32 one, and the linear layer behind it
    assert grown[FMT_BF16] <= grown[FMT_F32] + buffers + (8 << 20)
