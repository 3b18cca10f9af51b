"""What users of this framework have it do, as cases that can be timed and checked: quantized matmuls on device
tensors, decode steps of Q4/Q8 decoders through a session, prompts and single tokens of the Petotar and
Tobovik decoders through an engine.

Everything is drawn from a seed on the GPU.  A matmul's weights are what the benchmark configurations describe (codes
uniform, one scale per 32 elements log-uniform in [1e-3, 1e-1]); a decoder's are N(0, 0.02^2) quantized, the row-dynamic
designs' are bf16 with unit gain.
"""
import math
import zlib

import numpy as np
import torch

from meganeura_b200 import ops
from meganeura_b200.decode_model import DecoderConfig, build_decode_graph
from meganeura_b200.engine import Engine
from meganeura_b200.graph import Graph, build_inference_session
from meganeura_b200.petotar import Petotar, PetotarConfig
from meganeura_b200.tobovik import Tobovik, TobovikConfig

FMT = {"q4": ops.FMT_Q4, "q8": ops.FMT_Q8}
PACKED = {"q4": 20, "q8": 36}                       # bytes per block of 32
RANK = {"petotar": 64, "tobovik": 16}               # rows of the low-rank decay projections


# ---------------------------------------------------------------------------------------------- cases

def _matmul(name, fmt, act, m, k, n, addend=False):
    return dict(name=name, kind="matmul", fmt=fmt, act=act, m=m, k=k, n=n, addend=addend)


def _decoder(name, layers, heads, kv_heads, head_dim, ffn, vocab, context, steps, attn, mlp, head):
    return dict(name=name, kind="decoder", layers=layers, heads=heads, kv_heads=kv_heads, head_dim=head_dim, ffn=ffn, vocab=vocab, context=context,
                steps=steps, attn=attn, mlp=mlp, head=head)


def _rows(name, design, layers, width, ff, vocab, prompt, singles, portion, window=2048, dtype="bfloat16"):
    return dict(name=name, kind="rows", design=design, layers=layers, width=width, ff=ff, vocab=vocab, prompt=prompt, singles=singles, portion=portion,
                window=window, dtype=dtype)


def listed():
    return [
        # one token through the gate projection of SmolLM2-135M: the smallest call, latency only
        _matmul("gemv 576x1536 q8", "q8", "f32", 1, 576, 1536),
        # one token's logits of a Qwen3-8B-sized vocabulary: the longest weight stream of a decode step
        _matmul("gemv 4096x151936 q4", "q4", "f32", 1, 4096, 151936),
        # eight sequences decoded together: gate|up of the Qwen3-8B shape
        _matmul("batch8 4096x24576 q4", "q4", "f32", 8, 4096, 24576),
        # a prompt of 512 tokens with bf16 activations through a large up projection
        _matmul("gemm 512x4096x14336 q8 bf16", "q8", "bf16", 512, 4096, 14336),
        # a short prompt of odd length with bf16 activations, and a residual
        _matmul("gemm 203x1536x4100 q4 bf16", "q4", "bf16", 203, 1536, 4100, True),
        # the same with f32 activations, which is what a graph's matmul of a quantized parameter takes: a whole prompt
        _matmul("gemm 512x4096x12288 q4 f32", "q4", "f32", 512, 4096, 12288),
        # a handful of prompt tokens of the SmolLM2-135M shape, f32 activations, residual: the small end of the prefill
        _matmul("gemm 37x1536x576 q8 f32", "q8", "f32", 37, 1536, 576, True),
        # greedy decode of the SmolLM2-135M shape, the pick on the device: 30 small layers, launches and latency
        _decoder("decode smollm2-135m", 30, 9, 3, 64, 1536, 49152, 128, 8, "q8", "q4", "q8"),
        # greedy decode of layers of the Qwen3-8B shape behind a long context
        _decoder("decode 8 layers of 4096", 8, 32, 8, 128, 12288, 32768, 2048, 8, "q4", "q4", "q4"),
        # a long prompt of a Petotar model in one step, its last token's logits
        _rows("petotar prompt 2048", "petotar", "wamwsm", 2048, 6144, 32768, 2048, 0, 2048),
        # a chat turn of a Tobovik model: a prompt of odd length in the default portions, then single tokens one by one
        _rows("tobovik turn 777+12", "tobovik", "pgppgp", 2048, 6144, 32768, 777, 12, 512),
        # a Tobovik model in full f32, a prompt in one step and a few single tokens
        _rows("tobovik f32 100+3", "tobovik", "pg", 1024, 3072, 8192, 100, 3, 512, dtype="float32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matmul"] * 4 + ["decoder", "rows", "rows"])
    if kind == "matmul":
        act = rng.choice(["f32", "f32", "bf16"])
        group = rng.choice([(1, 2), (3, 16), (17, 512)]) if act == "f32" else (33, 512)
        m, k = _log(rng, *group), 32 * _log(rng, 18, 384)
        n = _log(rng, 192, 151936 if m <= 16 else 16384)
        most = 512 * 4096 * 12288
        n = max(192, min(n, most // (m * k)))
        if rng.random() < 0.6:                                  # widths are mostly round, and sometimes not
            n -= n % 64
        case = _matmul("", rng.choice(["q4", "q8"]), act, m, k, n, rng.random() < 0.4)
    elif kind == "decoder":
        head_dim = rng.choice([64, 128])
        kv_heads = rng.choice([1, 2, 3, 4, 8])
        heads = kv_heads * rng.choice([1, 2, 3, 4, 8])
        heads = min(heads, 4096 // head_dim // kv_heads * kv_heads)
        width = heads * head_dim
        layers = rng.randint(2, 30 if width <= 1024 else 8)
        case = _decoder("", layers, heads, kv_heads, head_dim, 32 * _log(rng, max(8, width // 16), max(16, width // 8)), 32 * _log(rng, 256, 1024),
                        _log(rng, 16, 2048), rng.randint(2, 8), rng.choice(["q4", "q8"]), rng.choice(["q4", "q8"]), rng.choice(["q4", "q8"]))
    else:
        design, full = rng.choice([("petotar", "wamwsm"), ("tobovik", "pgppgp")])
        dtype = rng.choice(["bfloat16"] * 4 + ["float32"])
        width = 512 * rng.randint(1, 4 if dtype == "bfloat16" else 2)
        count = rng.randint(2, 6 if dtype == "bfloat16" else 3)
        case = _rows("", design, full[:count], width, 8 * _log(rng, width // 8, 3 * width // 8), 8 * _log(rng, 512, 4096),
                     _log(rng, 2, 2048 if dtype == "bfloat16" else 256), rng.randint(0, 12), rng.choice([256, 512, 2048]), _log(rng, 128, 2048), dtype)
    case.pop("name")
    return case


# ------------------------------------------------------------------------------------------- weights

def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + zlib.crc32(name.encode()))


def _codes(fmt, k, n, seed):
    """Codes [n, k/32, 32] and f16 scales [n, k/32] of a matmul case's weight."""
    g = _gen(seed, "codes")
    lo, hi = math.log(1e-3), math.log(1e-1)
    d = torch.exp(torch.rand((n, k // 32), generator=g, device="cuda") * (hi - lo) + lo).half()
    if fmt == "q4":
        return torch.randint(0, 16, (n, k // 32, 32), generator=g, device="cuda", dtype=torch.uint8), d, (-8.0 * d.float()).half()
    return torch.randint(-127, 128, (n, k // 32, 32), generator=g, device="cuda", dtype=torch.int8), d, torch.zeros_like(d)


def _quantized(fmt, k, n, seed, name):
    """The same for a decoder's weight ~ N(0, 0.02^2)."""
    w = torch.randn((n, k // 32, 32), generator=_gen(seed, name), device="cuda") * 0.02
    if fmt == "q4":
        lo, hi = w.amin(-1), w.amax(-1)
        d = (hi - lo) / 15.0
        return ((w - lo[..., None]) / d[..., None]).round().clamp(0, 15).to(torch.uint8), d.half(), lo.half()
    d = w.abs().amax(-1) / 127.0
    return (w / d[..., None]).round().clamp(-127, 127).to(torch.int8), d.half(), torch.zeros_like(d, dtype=torch.half)


def _pack(fmt, codes, d, m):
    if fmt == "q4":
        header = torch.stack([d, m], -1).contiguous().view(torch.uint8).reshape(-1)
        return torch.cat([header, (codes[..., 0::2] | (codes[..., 1::2] << 4)).reshape(-1)])
    zeros = torch.zeros_like(d)
    return torch.cat([torch.stack([d, zeros], -1).contiguous().view(torch.uint8).reshape(*d.shape, 4), codes.view(torch.uint8)], -1).reshape(-1)


def _times(x, codes, d, m):
    """x [rows, k] . W in 64 bits, for the weight that the codes stand for."""
    out = torch.empty((x.shape[0], codes.shape[0]), dtype=torch.float64, device="cuda")
    for c in range(0, codes.shape[0], 8192):
        w = codes[c:c + 8192].double() * d[c:c + 8192, :, None].double() + m[c:c + 8192, :, None].double()
        out[:, c:c + 8192] = x @ w.reshape(w.shape[0], -1).T
    return out


# ------------------------------------------------------------------------------------ matmul cases

def _matmul_inputs(case, seed):
    g = _gen(seed, "x")
    x = torch.randn((case["m"], case["k"]), generator=g, device="cuda")
    add = torch.randn((case["m"], case["n"]), generator=g, device="cuda") if case["addend"] else None
    return x if case["act"] == "f32" else x.bfloat16(), add


# ----------------------------------------------------------------------------------- decoder cases

def _decoder_config(case):
    return DecoderConfig("decoder", case["vocab"], case["heads"] * case["head_dim"], case["layers"], case["heads"], case["kv_heads"], case["head_dim"],
                         case["ffn"], 1e-5, 1e4, FMT[case["attn"]], FMT[case["mlp"]], FMT[case["head"]])


def _decoder_weights(case):
    """(name, format, k, n) of every quantized weight."""
    hidden, kv, out = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"], []
    for i in range(case["layers"]):
        for name, fmt, k, n in (("self_attn.q_proj", "attn", hidden, hidden), ("self_attn.k_proj", "attn", hidden, kv), ("self_attn.v_proj", "attn", hidden, kv),
                                ("self_attn.o_proj", "attn", hidden, hidden), ("mlp.gate_proj", "mlp", hidden, case["ffn"]),
                                ("mlp.up_proj", "mlp", hidden, case["ffn"]), ("mlp.down_proj", "mlp", case["ffn"], hidden)):
            out.append((f"model.layers.{i}.{name}.weight", case[fmt], k, n))
    return out + [("lm_head.weight", case["head"], hidden, case["vocab"])]


def _decoder_rest(case, seed):
    """Embedding table, norm weights, cached keys and values: name -> f32 tensor."""
    hidden, kv = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    out = {"model.embed_tokens.weight": torch.randn((case["vocab"], hidden), generator=_gen(seed, "embed"), device="cuda")}
    for i in range(case["layers"]):
        for name in (f"model.layers.{i}.input_layernorm.weight", f"model.layers.{i}.post_attention_layernorm.weight"):
            out[name] = 1.0 + 0.1 * torch.randn(hidden, generator=_gen(seed, name), device="cuda")
        for name in (f"kv_cache.layer.{i}.k", f"kv_cache.layer.{i}.v"):
            out[name] = torch.zeros((case["context"] + case["steps"] + 8, kv), device="cuda")
            out[name][:case["context"]] = torch.randn((case["context"], kv), generator=_gen(seed, name), device="cuda")
    out["model.norm.weight"] = 1.0 + 0.1 * torch.randn(hidden, generator=_gen(seed, "norm"), device="cuda")
    return out


def _decoder_prepare(case, seed):
    graph = Graph()
    limit = case["context"] + case["steps"] + 8
    logits, _, _ = build_decode_graph(graph, _decoder_config(case), limit)
    graph.set_outputs([logits])
    s = build_inference_session(graph)
    for name, fmt, k, n in _decoder_weights(case):
        s.upload_param(name, _pack(fmt, *_quantized(fmt, k, n, seed, name)).cpu().numpy())
    for name, value in _decoder_rest(case, seed).items():
        s.set_parameter(name, value.cpu().numpy())
    s.enable_greedy(0, "token_ids", "kv_pos", limit)
    token = int(torch.randint(0, case["vocab"], (1,), generator=_gen(seed, "token"), device="cuda"))
    s.set_input_u32("token_ids", [token])
    s.set_input_u32("kv_pos", [case["context"]])
    s.step()                                                    # a step is captured after it has run once
    s.wait()
    s.capture()
    return {"case": case, "session": s, "token": token}


def _decoder_run(state):
    case, s = state["case"], state["session"]
    s.set_input_u32("token_ids", [state["token"]])
    s.set_input_u32("kv_pos", [case["context"]])
    for _ in range(case["steps"]):
        s.step()
    s.wait()
    return {"tokens": s.read_tokens(case["context"], case["steps"]).astype(np.int64), "logits": s.read_output(case["vocab"])}


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _decoder_exact(case, seed):
    heads, kv_heads, dim, eps = case["heads"], case["kv_heads"], case["head_dim"], 1e-5
    w = {name: _quantized(fmt, k, n, seed, name) for name, fmt, k, n in _decoder_weights(case)}
    r = {name: value.double() for name, value in _decoder_rest(case, seed).items()}
    token = int(torch.randint(0, case["vocab"], (1,), generator=_gen(seed, "token"), device="cuda"))
    # the angle is defined in f32
    freq = torch.pow(torch.tensor(1e4, device="cuda"), -2.0 * torch.arange(dim // 2, device="cuda", dtype=torch.float32) / dim)

    def rope(x, pos):
        a = (float(pos) * freq).double()
        u, v = x.reshape(-1, dim).split(dim // 2, -1)
        return torch.cat([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1)
    for pos in range(case["context"], case["context"] + case["steps"]):
        x = r["model.embed_tokens.weight"][token][None]
        for i in range(case["layers"]):
            p, kc, vc = f"model.layers.{i}", r[f"kv_cache.layer.{i}.k"], r[f"kv_cache.layer.{i}.v"]
            h = _rms(x, r[f"{p}.input_layernorm.weight"], eps)
            q, k, v = (_times(h, *w[f"{p}.self_attn.{s}_proj.weight"]) for s in "qkv")
            q, kc[pos], vc[pos] = rope(q, pos).reshape(kv_heads, -1, dim), rope(k, pos).reshape(-1), v[0]
            keys, values = (c[:pos + 1].reshape(pos + 1, kv_heads, dim).transpose(0, 1) for c in (kc, vc))
            a = torch.softmax(q @ keys.transpose(1, 2) / math.sqrt(dim), -1) @ values
            x = x + _times(a.reshape(1, heads * dim), *w[f"{p}.self_attn.o_proj.weight"])
            h = _rms(x, r[f"{p}.post_attention_layernorm.weight"], eps)
            gate, up = (_times(h, *w[f"{p}.mlp.{s}_proj.weight"]) for s in ("gate", "up"))
            x = x + _times(torch.nn.functional.silu(gate) * up, *w[f"{p}.mlp.down_proj.weight"])
        logits = _times(_rms(x, r["model.norm.weight"], eps), *w["lm_head.weight"])[0]
        token = int(logits.argmax())
    return {"tokens": None, "logits": logits}


# --------------------------------------------------------------------- Petotar and Tobovik cases

def _rows_config(case):
    """config.json of the design at the case's sizes: head sizes are the design benchmark's."""
    w, layers = case["width"], []
    for i, kind in enumerate(case["layers"]):
        if case["design"] == "petotar":
            latent = dict(heads=w // 128, dim=128, rot_dim=64, vdim=128, kv_rank=512, mask={"size": case["window"]}, rot={"base": 1e6, "dims": 64}, scale=192 ** -0.5)
            entry = {"w": dict(type="wkv", mixer=dict(heads=w // 64, dim=64)), "m": dict(type="mlstm", mixer=dict(heads=w // 256, dim=128, vdim=256, gate_cap=15.0)),
                     "a": dict(type="latent_attention", mixer=latent), "s": dict(type="latent_attention", mixer=dict(latent, kv_from=case["layers"].find("a")))}[kind]
            layers.append(dict(entry, mlp={"kind": "dense", "ff": case["ff"], "limit": 7.0}))
        else:
            left = dict(heads=w // 128, kv_heads=max(1, w // 512), dim=128, vdim=128, scale=128 ** -0.5, q_temp={"coef": 0.1, "every": 8192})
            right = dict(heads=w // 256, dim=128, vdim=256, tau=16.0)
            entry = dict(type="parallel", mixer=dict(left=left, right=right, left_scale=0.7, right_scale=1.0)) if kind == "p" else \
                dict(type="gla", mixer=dict(heads=w // 512, dim=256, vdim=512, tau=16.0))
            layers.append(dict(entry, mlp={"kind": "dense", "ff": case["ff"]}))
    out = {"architecture": case["design"].capitalize(), "vocab": case["vocab"], "width": w, "norm": {"eps": 1e-6}, "layers": layers}
    return dict(out, embedding={"scale": 1.0}) if case["design"] == "petotar" else out


def _rows_shapes(case):
    """name -> shape of every weight."""
    w, rank, out = case["width"], RANK[case["design"]], {"embed": (case["vocab"], case["width"])}

    def put(p, **shapes):
        out.update({p + name.replace("_", "."): shape for name, shape in shapes.items()})

    def gla(p, m):
        n, nv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        put(p, q=(n, w), k=(n, w), v=(nv, w), g=(nv, w), a1=(rank, w), a2=(n, rank), a2_b=(n,), norm=(m["vdim"],), o=(w, nv))
    for i, layer in enumerate(_rows_config(case)["layers"]):
        p, m, ff = f"l{i}.mix.", layer["mixer"], layer["mlp"]["ff"]
        put(f"l{i}.", norm1=(w,), norm2=(w,))
        put(f"l{i}.mlp.", gate=(ff, w), up=(ff, w), down=(w, ff))
        if case["design"] == "petotar":
            put(f"l{i}.mlp.", gate_b=(ff,), up_b=(ff,), down_b=(w,))
        if layer["type"] == "wkv":
            n = m["heads"] * m["dim"]
            put(p, mu_r=(w,), mu_k=(w,), mu_v=(w,), mu_g=(w,), mu_w=(w,), r=(n, w), k=(n, w), v=(n, w), g=(n, w), w1=(rank, w), w2=(n, rank), w0=(n,), u=(n,),
                norm=(n,), o=(w, n))
        elif layer["type"] == "mlstm":
            n, nv, h = m["heads"] * m["dim"], m["heads"] * m["vdim"], m["heads"]
            put(p, q=(n, w), k=(n, w), v=(nv, w), g=(nv, w), i=(h, w), f=(h, w), i_b=(h,), f_b=(h,), norm=(nv,), o=(w, nv))
        elif layer["type"] == "latent_attention":
            h, row = m["heads"], m["kv_rank"]
            put(p, q=(h * (m["dim"] + m["rot_dim"]), w), g=(h * m["vdim"], w), uk=(h * m["dim"], row), uv=(h * m["vdim"], row), o=(w, h * m["vdim"]))
            if "kv_from" not in m:
                put(p, dkv=(row + m["rot_dim"], w), dkv_norm=(row,))
        elif layer["type"] == "gla":
            gla(p, m)
        else:
            a = m["left"]
            nq, nk, nv, no = a["heads"] * a["dim"], a["kv_heads"] * a["dim"], a["kv_heads"] * a["vdim"], a["heads"] * a["vdim"]
            put(p + "left.", q=(nq, w), q_b=(nq,), q_norm=(nq,), k=(nk, w), k_b=(nk,), k_norm=(nk,), v=(nv, w), v_b=(nv,), g=(no, w), o=(w, no))
            gla(p + "right.", m["right"])
    out["final.norm"] = (w,)
    if case["design"] == "tobovik":
        out["head"] = (case["vocab"], w)
    return out


def _rows_weight(case, seed, name, shape):
    a = torch.randn(shape, generator=_gen(seed, name), device="cuda")
    if len(shape) == 2:
        return (a * shape[1] ** -0.5).bfloat16()
    if ".mu." in name:
        return torch.sigmoid(a)
    if name.endswith(".a2.b"):
        return a * 1.5 + 2.0
    if "norm" in name.rsplit(".", 1)[-1] and (case["design"] == "tobovik" or ".mix." in name):
        return a * 0.1 + 1.0                                    # the other norm weights are stored around zero
    if name.endswith(".w0"):
        return a * 0.1 - 3.0
    return a * 0.1 + (3.0 if name.endswith(".f.b") else 0.0)


def _rows_tokens(case, seed):
    return torch.randint(0, case["vocab"], (case["prompt"] + case["singles"],), generator=_gen(seed, "tokens"), device="cuda").cpu().numpy()


def _rows_prepare(case, seed):
    config, total, rank = _rows_config(case), case["prompt"] + case["singles"], RANK[case["design"]]
    kw = dict(dtype=case["dtype"], max_rows=case["portion"], max_tokens=total)
    if case["design"] == "petotar":
        model = Petotar(PetotarConfig.from_dict(config), lora_rank={i: rank for i, kind in enumerate(case["layers"]) if kind == "w"}, **kw)
    else:
        model = Tobovik(TobovikConfig.from_dict(config), lora_rank={f"l{i}.mix" + (".right" if kind == "p" else ""): rank for i, kind in enumerate(case["layers"])}, **kw)
    for name, shape, bf16 in model.parameters():
        value = _rows_weight(case, seed, name, shape)
        if bf16:
            model.session.upload_param(name, value.view(torch.int16).cpu().numpy())
        else:
            model.session.set_parameter(name, value.cpu().numpy())
    return {"case": case, "engine": Engine(model, greedy=False), "tokens": _rows_tokens(case, seed)}


def _rows_run(state):
    """A sequence from its start: the prompt's last logits, then those of every single token."""
    case, e, tokens = state["case"], state["engine"], state["tokens"]
    e.end()
    out = [e.feed(tokens[:case["prompt"]], [case["prompt"] - 1])]
    for t in tokens[case["prompt"]:]:
        out.append(e.feed([t], [0]))
    return np.concatenate(out)


class _Exact:
    """The two designs token by token or over all tokens at once, whichever is plain, in 64 bits."""

    def __init__(self, case, seed):
        self.case, self.w = case, {}
        shapes = _rows_shapes(case)
        self.get = lambda name: _rows_weight(case, seed, name, shapes[name]).double()

    def lin(self, x, name, bias=False):
        y = x @ self.get(name).T
        return y + self.get(name + ".b") if bias else y

    def heads(self, x, n):
        return x.reshape(x.shape[0], n, -1)

    def unit(self, x):
        return _rms(x, 1.0, 1e-6)

    def attend(self, q, k, v, scale, window):
        """q [T, H, D], k [T, G, D], v [T, G, V]; head h reads key / value head h // (H / G)."""
        t, ratio = q.shape[0], q.shape[1] // k.shape[1]
        age = torch.arange(t, device="cuda")[:, None] - torch.arange(t, device="cuda")[None]
        hidden = (age < 0) | (age >= window)
        out = torch.empty((t, q.shape[1], v.shape[2]), dtype=torch.float64, device="cuda")
        for h in range(q.shape[1]):
            s = (q[:, h] @ k[:, h // ratio].T * scale).masked_fill(hidden, -math.inf)
            out[:, h] = torch.softmax(s, -1) @ v[:, h // ratio]
        return out.reshape(t, -1)

    def rotate(self, x, base):
        half = x.shape[-1] // 2
        a = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * base ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
        u, v = x[..., :half], x[..., half:]
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)

    def wkv(self, p, m, x, _):
        before = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
        mix = {s: x + (before - x) * self.get(f"{p}mu.{s}") for s in "rkvgw"}
        r, k, v = (self.heads(self.lin(mix[s], p + s), m["heads"]) for s in "rkv")
        w = torch.exp(-torch.exp(torch.tanh(self.lin(mix["w"], p + "w1")) @ self.get(p + "w2").T + self.get(p + "w0"))).reshape(r.shape)
        u, state, out = self.get(p + "u").reshape(m["heads"], -1, 1), torch.zeros((m["heads"], m["dim"], m["dim"]), dtype=torch.float64, device="cuda"), []
        for t in range(len(x)):
            kv = k[t][:, :, None] * v[t][:, None]
            out.append((r[t][:, None] @ (state + u * kv))[:, 0])
            state = w[t][:, :, None] * state + kv
        o = self.unit(torch.stack(out)).reshape(len(x), -1) * self.get(p + "norm")
        return self.lin(o * torch.nn.functional.silu(self.lin(mix["g"], p + "g")), p + "o")

    def mlstm(self, p, m, x, _):
        h, dim, cap = m["heads"], m["dim"], m["gate_cap"]
        q, k, v = (self.heads(self.lin(x, p + s), h) for s in "qkv")
        q = q * dim ** -0.5
        log_i = cap * torch.tanh(self.lin(x, p + "i", True) / cap)
        log_f = torch.nn.functional.logsigmoid(cap * torch.tanh(self.lin(x, p + "f", True) / cap))
        s, n = torch.zeros((h, dim, m["vdim"]), dtype=torch.float64, device="cuda"), torch.zeros((h, dim), dtype=torch.float64, device="cuda")
        top, out = torch.zeros(h, dtype=torch.float64, device="cuda"), []
        for t in range(len(x)):
            new = torch.maximum(log_f[t] + top, log_i[t])
            keep, write = torch.exp(log_f[t] + top - new)[:, None], torch.exp(log_i[t] - new)[:, None]
            s = keep[:, :, None] * s + (write * k[t])[:, :, None] * v[t][:, None]
            n, top = keep * n + write * k[t], new
            out.append((q[t][:, None] @ s)[:, 0] / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-new)) + 1e-6)[:, None])
        o = self.unit(torch.stack(out)).reshape(len(x), -1) * self.get(p + "norm")
        return self.lin(o * torch.sigmoid(self.lin(x, p + "g")), p + "o")

    def latent(self, p, m, x, cache):
        h, dim, rank, base = m["heads"], m["dim"], m["kv_rank"], m["rot"]["base"]
        q = self.heads(self.lin(x, p + "q"), h)
        q = torch.cat([q[..., :dim], self.rotate(q[..., dim:], base)], -1)
        if "kv_from" not in m:
            down = self.lin(x, p + "dkv")
            cache.append((self.unit(down[:, :rank]) * self.get(p + "dkv.norm"), self.rotate(down[:, None, rank:], base)))
        c, kr = cache[0]
        k = torch.cat([self.heads(self.lin(c, p + "uk"), h), kr.expand(-1, h, -1)], -1)
        o = self.attend(q, k, self.heads(self.lin(c, p + "uv"), h), m["scale"], m["mask"]["size"])
        return self.lin(o * torch.sigmoid(self.lin(x, p + "g")), p + "o")

    def gla(self, p, m, x):
        q, k, v = (self.heads(self.lin(x, p + s), m["heads"]) for s in "qkv")
        q = q * m["dim"] ** -0.5
        z = self.lin(x, p + "a1") @ self.get(p + "a2").T + self.get(p + "a2.b")
        decay = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(q.shape)
        s, out = torch.zeros((m["heads"], m["dim"], m["vdim"]), dtype=torch.float64, device="cuda"), []
        for t in range(len(x)):
            s = decay[t][:, :, None] * s + k[t][:, :, None] * v[t][:, None]
            out.append((q[t][:, None] @ s)[:, 0])
        o = (self.unit(torch.stack(out)) * self.get(p + "norm")).reshape(len(x), -1)
        return self.lin(o * torch.nn.functional.silu(self.lin(x, p + "g")), p + "o")

    def parallel(self, p, m, x):
        a, l = m["left"], p + "left."
        q = self.unit(self.lin(x, l + "q", True)) * self.get(l + "q.norm")
        k = self.unit(self.lin(x, l + "k", True)) * self.get(l + "k.norm")
        pos = torch.arange(len(x), device="cuda", dtype=torch.float64)[:, None]
        q = q * (1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / a["q_temp"]["every"]) + 1.0))
        o = self.attend(self.heads(q, a["heads"]), self.heads(k, a["kv_heads"]), self.heads(self.lin(x, l + "v", True), a["kv_heads"]), a["scale"], len(x))
        left = self.lin(o * torch.sigmoid(self.lin(x, l + "g")), l + "o")
        return m["left_scale"] * left + m["right_scale"] * self.gla(p + "right.", m["right"], x)

    def run(self, tokens):
        case, w = self.case, self.case["width"]
        x = self.get("embed")[torch.from_numpy(tokens).cuda()]
        petotar, cache = case["design"] == "petotar", []
        if not petotar:
            angle = torch.arange(len(x), device="cuda", dtype=torch.float64)[:, None] * 1e4 ** (-2.0 * torch.arange((w + 1) // 2, device="cuda", dtype=torch.float64) / w)
            x = x + torch.stack([angle.sin(), angle.cos()], -1).reshape(len(x), -1)[:, :w]
        for i, layer in enumerate(_rows_config(case)["layers"]):
            p, f = f"l{i}.mix.", f"l{i}.mlp."
            if petotar:
                mixer = {"wkv": self.wkv, "mlstm": self.mlstm, "latent_attention": self.latent}[layer["type"]]
                x = x + mixer(p, layer["mixer"], self.unit(x) * (1.0 + self.get(f"l{i}.norm1")), cache)
                h = self.unit(x) * (1.0 + self.get(f"l{i}.norm2"))
                gate, up = self.lin(h, f + "gate", True).clamp(max=7.0), self.lin(h, f + "up", True).clamp(-7.0, 7.0)
                x = x + self.lin(gate * torch.sigmoid(1.702 * gate) * (up + 1.0), f + "down", True)
            else:
                y = (self.parallel if layer["type"] == "parallel" else self.gla)(p, layer["mixer"], x)
                x = x + self.unit(y) * self.get(f"l{i}.norm1")
                y = self.lin(torch.nn.functional.silu(self.lin(x, f + "gate")) * self.lin(x, f + "up"), f + "down")
                x = x + self.unit(y) * self.get(f"l{i}.norm2")
        x = x[case["prompt"] - 1:]
        h = self.unit(x) * (self.get("final.norm") + (1.0 if petotar else 0.0))
        return h @ self.get("embed" if petotar else "head").T


# ------------------------------------------------------------------------------------------ interface

def prepare(case, seed):
    if case["kind"] == "decoder":
        return _decoder_prepare(case, seed)
    if case["kind"] == "rows":
        return _rows_prepare(case, seed)
    x, add = _matmul_inputs(case, seed)
    w = _pack(case["fmt"], *_codes(case["fmt"], case["k"], case["n"], seed))
    return {"case": case, "x": x, "w": w, "add": add, "out": torch.empty((case["m"], case["n"]), device="cuda")}


def run(state):
    case = state["case"]
    if case["kind"] == "decoder":
        return _decoder_run(state)
    if case["kind"] == "rows":
        return _rows_run(state)
    return ops.matmul(FMT[case["fmt"]], state["x"], state["w"], case["k"], case["n"], addend=state["add"], out=state["out"])


def work(case):
    if case["kind"] == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        act = 4 if case["act"] == "f32" else 2
        return {"bytes": k * n // 32 * PACKED[case["fmt"]] + act * m * k + 4 * m * n * (2 if case["addend"] else 1), "flops": 2 * m * k * n}
    if case["kind"] == "decoder":
        kv = 4 * case["kv_heads"] * case["head_dim"]
        weights = sum(k * n // 32 * PACKED[fmt] for _, fmt, k, n in _decoder_weights(case))
        dense = sum(k * n for _, _, k, n in _decoder_weights(case))
        step = weights + case["layers"] * 2 * kv * case["context"] + 4 * case["vocab"]
        flops = 2 * dense + 4 * case["layers"] * case["heads"] * case["head_dim"] * case["context"]
        return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}
    shapes = _rows_shapes(case)
    head = case["vocab"] * case["width"]
    dense = sum(math.prod(s) for name, s in shapes.items() if len(s) == 2 and name not in ("embed", "head"))
    total, passes = case["prompt"] + case["singles"], 1 + case["singles"]
    flops = 2 * dense * total + 2 * head * passes
    for layer in _rows_config(case)["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            seen = sum(min(t + 1, case["window"]) for t in range(total))
            flops += 2 * m["heads"] * seen * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif layer["type"] == "parallel":
            flops += m["left"]["heads"] * total * total * (m["left"]["dim"] + m["left"]["vdim"])
        r = m["right"] if layer["type"] == "parallel" else m
        if layer["type"] != "latent_attention":
            flops += 5 * total * r["heads"] * r["dim"] * r.get("vdim", r["dim"])
    return {"bytes": passes * 2 * (dense + head) + 4 * passes * case["vocab"], "flops": flops}


def tolerance(case):
    """About four times the distance from exact() that was measured: f32 sums 1e-6 off, weights as sums of two bf16 9e-6, a decoder's
    chain of f32 layers 5e-6, bf16 operands of a whole model 1.2e-2."""
    if case["kind"] == "matmul":
        return {"rel": 1e-5} if case["act"] == "f32" else {"rel": 4e-5}
    if case["kind"] == "decoder":
        return {"rel": 3e-5}
    return {"rel": 2e-5} if case["dtype"] == "float32" else {"rel": 3e-2}


def exact(case, seed):
    if case["kind"] == "decoder":
        return _decoder_exact(case, seed)
    if case["kind"] == "rows":
        return _Exact(case, seed).run(_rows_tokens(case, seed))
    x, add = _matmul_inputs(case, seed)
    y = _times(x.double(), *_codes(case["fmt"], case["k"], case["n"], seed))
    return y if add is None else y + add
