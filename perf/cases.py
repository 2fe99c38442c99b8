"""Performance cases of the library: what its users run, over the ranges they run it in.

    call      Linear.forward on host arrays (QuantTensor.matmul_t): one blocking call, x in and y out
    stack     a stack of quantized layers on device buffers, one captured graph per pass: single-token decode
              (m = 1), small batches and the tensor-core range (m >= 64); `relaxed` declares the layers independent
    ffn       SwiGLU feed-forward of a prompt (gate / up / down, each of a block type of its own)
    attend    one decode step's grouped-query attention over a KV cache, sequences of different lengths
    llama     a request to the quantized decoder: a prompt, then tokens chosen by the caller, logits after each
    lugasun, tutezen   the same for the two decoders over dense bf16 weights

Weights are normally distributed values quantized to their block type, so that scales, minima and activations have the
sizes they have in a trained model.  A decoder's layers share one set of values, each in device buffers of its own."""
from __future__ import annotations

import math
import re

import numpy as np
import torch

import skainet_b200 as skn
from skainet_b200 import _ffi
from skainet_b200.llama import LlamaConfig, LlamaDecoder
from skainet_b200.lugasun import LugasunConfig
from skainet_b200.tutezen import TutezenConfig

TYPE_ID = {"q4_0": 2, "q8_0": 8, "q4_k": 12, "q6_k": 14}
BLOCK = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_k": (256, 144), "q6_k": (256, 210)}
VOCAB = 32000
# width: attention heads, kv heads, head width, retention heads, their key and value width, feed-forward, side width
LUGASUN = {1024: (8, 2, 128, 8, 64, 64, 4096, 64), 2048: (16, 4, 128, 8, 128, 128, 8192, 64)}
# width: state-space heads (of 64), attention heads, query and key latents, feed-forward, expert and shared widths
TUTEZEN = {1024: (32, 8, 512, 256, 4096, 512, 1024), 2048: (64, 16, 1024, 512, 8192, 1024, 2048)}
TUTEZEN_PATTERN = ("ssm dense", "ssm moe", "ssm moe", "att dense", "ssm dense", "ssm moe", "ssm dense", "att moe")
EXPERTS, TOP = 32, 4


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # one layer called from host code, as Linear.forward is: latency of a single call
        dict(name="call_q4k_m1", kind="call", type="q4_k", n=4096, k=4096, m=1),
        # decode matvec at batch 1 in stream order: 48 square layers, 453 MB of weights
        dict(name="stack_q4k_m1", kind="stack", type="q4_k", n=4096, k=4096, m=1, layers=48, relaxed=False),
        # four sequences against a feed-forward projection in Q8_0
        dict(name="stack_q80_m4", kind="stack", type="q8_0", n=14336, k=4096, m=4, layers=6, relaxed=False),
        # sixteen sequences against a down projection in Q4_0
        dict(name="stack_q40_m16", kind="stack", type="q4_0", n=4096, k=14336, m=16, layers=8, relaxed=False),
        # prompt of 512 tokens through the feed-forward block, mixed K-quants
        dict(name="ffn_m512", kind="ffn", gate="q4_k", down="q6_k", d=4096, f=14336, m=512),
        # decode attention of eight sequences of 1024 .. 4096 tokens, fp32 cache
        dict(name="attend_b8", kind="attend", batch=8, heads=32, kv_heads=8, dim=128, context=4096, cache="f32"),
        # prompt of 512 tokens, one sampled token: time to the first token
        dict(name="llama_prompt", kind="llama", width=4096, heads=32, kv_heads=8, ffn=14336, layers=8, batch=1, prompt=512, steps=1, cache="f32"),
        # a single user's answer: decoding at batch 1
        dict(name="llama_decode_b1", kind="llama", width=4096, heads=32, kv_heads=8, ffn=14336, layers=8, batch=1, prompt=96, steps=32, cache="f32"),
        # sixteen users' answers in step
        dict(name="llama_decode_b16", kind="llama", width=4096, heads=32, kv_heads=8, ffn=14336, layers=8, batch=16, prompt=20, steps=12, cache="f16"),
        # long prompt through the dense bf16 decoder, and its first token
        dict(name="lugasun_prompt", kind="lugasun", width=2048, layers=8, batch=1, prompt=2048, steps=1),
        # sixteen sequences decoding in step
        dict(name="lugasun_decode_b16", kind="lugasun", width=2048, layers=8, batch=16, prompt=40, steps=12),
        # a whole request to the mixture-of-experts decoder: prompt and answer of one user
        dict(name="tutezen_request", kind="tutezen", width=1024, layers=8, batch=1, prompt=700, steps=24),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["call", "stack", "stack", "stack", "ffn", "attend", "llama", "llama", "lugasun", "tutezen"])
    qtype = rng.choice(sorted(BLOCK))
    # rows of any number; columns in whole super-blocks as in nearly every model, sometimes in 32s where the type allows it
    n = _log(rng, 256, 16384)
    k = 256 * _log(rng, 1, 56) if BLOCK[qtype][0] == 256 or rng.random() < 0.8 else 32 * _log(rng, 8, 256)
    if kind == "call":
        return dict(kind=kind, type=qtype, n=n, k=k, m=_log(rng, 1, 16))
    if kind == "stack":
        n, m = 8 * max(32, n // 8), _log(rng, 1, 300)
        layers = max(2, min(48, 200_000_000 // (n * k // 2) + 1, 6_000_000_000 // (n * k * max(8, m) // 8) + 1))
        return dict(kind=kind, type=qtype, n=n, k=k, m=m, layers=layers, relaxed=rng.random() < 0.3)
    if kind == "ffn":
        return dict(kind=kind, gate=rng.choice(["q4_k", "q4_0", "q8_0"]), down=rng.choice(["q4_k", "q6_k", "q8_0"]), d=256 * _log(rng, 4, 16),
                    f=256 * _log(rng, 8, 56), m=_log(rng, 64, 512))
    if kind == "attend":
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, batch=_log(rng, 1, 12), heads=kv * rng.choice([1, 4, 8]), kv_heads=kv, dim=rng.choice([64, 128, 128]),
                    context=_log(rng, 100, 4096), cache=rng.choice(["f32", "f32", "f16", "q8_0"]))
    long = rng.random() < 0.5
    batch = 1 if long else _log(rng, 1, 16)
    prompt = _log(rng, 128, 512 if kind == "llama" else 2048) if long else _log(rng, 2, 40)
    steps = 1 if long else _log(rng, 4, 24) if batch < 4 else _log(rng, 4, 12)
    if kind == "llama":
        width = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, width=width, heads=width // 128, kv_heads=rng.choice([width // 512, width // 128]), ffn=256 * _log(rng, width // 128, width // 80),
                    layers=_log(rng, 2, 8), batch=batch, prompt=prompt, steps=steps, cache=rng.choice(["f32", "f32", "f16", "q8_0"]))
    return dict(kind=kind, width=rng.choice([1024, 2048] if kind == "lugasun" else [1024]), layers=_log(rng, 4, 8), batch=batch, prompt=prompt, steps=steps)


# ---- block quantization of normal weights, and their exact values ---------------------------------------------------
def _half(x):
    """fp16 bytes [..., 2] and the value they hold."""
    h = x.to(torch.float16)
    return h.view(torch.uint8).reshape(*h.shape, 2), h.float()


def _quantize(qtype, w):
    """fp32 [rows, cols] -> (blocks as bytes [rows, bytes], what they stand for in fp64)."""
    rows, cols = w.shape
    if qtype in ("q4_0", "q8_0"):
        b = w.reshape(rows, cols // 32, 32)
        if qtype == "q4_0":
            at = b.abs().argmax(-1, keepdim=True)
            raw, d = _half(b.gather(-1, at).squeeze(-1) / -8)
            q = (torch.round(b / _away(d)[..., None]) + 8).clamp_(0, 15)
            u = q.to(torch.uint8)
            out, q = torch.cat([raw, u[..., :16] | (u[..., 16:] << 4)], -1), q - 8
        else:
            raw, d = _half(b.abs().amax(-1) / 127)
            q = torch.round(b / _away(d)[..., None]).clamp_(-127, 127)
            out = torch.cat([raw, q.to(torch.int8).view(torch.uint8)], -1)
        return out.reshape(rows, -1), lambda: (d.double()[..., None] * q.double()).reshape(rows, cols)
    b = w.reshape(rows, cols // 256, 256)
    if qtype == "q4_k":
        s = b.reshape(rows, -1, 8, 32)
        low = s.amin(-1).clamp_(max=0.0)
        scale = (s.amax(-1) - low) / 15
        d_raw, d = _half(scale.amax(-1) / 63)
        m_raw, dmin = _half(-low.amin(-1) / 63)
        sc = torch.round(scale / _away(d)[..., None]).clamp_(0, 63)
        mn = torch.round(-low / _away(dmin)[..., None]).clamp_(0, 63)
        q = torch.round((s + (dmin[..., None] * mn)[..., None]) / _away(d[..., None] * sc)[..., None]).clamp_(0, 15)
        a, c, u = sc.to(torch.uint8), mn.to(torch.uint8), q.to(torch.uint8)
        packed = torch.cat([a[..., :4] | (a[..., 4:] >> 4 << 6), c[..., :4] | (c[..., 4:] >> 4 << 6), (a[..., 4:] & 15) | (c[..., 4:] << 4)], -1)
        out = torch.cat([d_raw, m_raw, packed, (u[..., 0::2, :] | (u[..., 1::2, :] << 4)).flatten(-2)], -1)
        return out.reshape(rows, -1), lambda: ((d[..., None] * sc).double()[..., None] * q.double()
                                               - (dmin[..., None] * mn).double()[..., None]).reshape(rows, cols)
    s = b.reshape(rows, -1, 16, 16)
    scale = s.abs().amax(-1) / 31
    raw, d = _half(scale.amax(-1) / 127)
    sc = torch.round(scale / _away(d)[..., None]).clamp_(1, 127)
    q = torch.round(s / _away(d[..., None] * sc)[..., None]).clamp_(-32, 31)
    u = (q + 32).to(torch.uint8).reshape(rows, -1, 2, 4, 32)          # halves of 128, runs of 32
    ql = (u[..., 0:2, :] & 15) | (u[..., 2:4, :] << 4)
    qh = (u[..., 0, :] >> 4) | (u[..., 1, :] >> 4 << 2) | (u[..., 2, :] >> 4 << 4) | (u[..., 3, :] >> 4 << 6)
    out = torch.cat([ql.flatten(-3), qh.flatten(-2), sc.to(torch.int8).view(torch.uint8), raw], -1)
    return out.reshape(rows, -1), lambda: ((d[..., None] * sc).double()[..., None] * q.double()).reshape(rows, cols)


def _away(d):
    """d, with 1 in the place of 0 (a block of zeros)."""
    return torch.where(d == 0, torch.ones_like(d), d)


def _generator(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _normal(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda") * std


def _weight(g, qtype, rows, cols, std=None):
    return _quantize(qtype, _normal(g, rows, cols, std=cols ** -0.5 if std is None else std))


def _host(raw):
    return raw.cpu().numpy()


# ---- linear layers ---------------------------------------------------------------------------------------------------
def _stack_inputs(c, seed):
    """Blocks and exact values of every layer (four sets of values, taken in turn), activations [layers, m, k]."""
    g = _generator(seed)
    layers = c.get("layers", 1)
    w = [_weight(g, c["type"], c["n"], c["k"]) for _ in range(min(4, layers))]
    return [w[i % len(w)] for i in range(layers)], _normal(g, layers, c["m"], c["k"])


def _prepare_call(c, seed):
    (w,), x = _stack_inputs(c, seed)
    ctx = skn.Context(0)
    return dict(ctx=ctx, w=skn.QuantTensor(ctx, (c["n"], c["k"]), TYPE_ID[c["type"]], _host(w[0])), x=_host(x[0]))


def _prepare_stack(c, seed):
    w, x = _stack_inputs(c, seed)
    ctx = skn.Context(0)
    ctx.set_relaxed_order(c["relaxed"])
    raw = [_host(b) for b, _ in w[:4]]
    ts = [skn.QuantTensor(ctx, (c["n"], c["k"]), TYPE_ID[c["type"]], raw[i % len(raw)]) for i in range(len(w))]
    y = torch.empty(len(ts), c["m"], c["n"], device="cuda")

    def layers():
        for t, a, b in zip(ts, x, y):
            t.matmul_t_dev(a, c["m"], b)

    torch.cuda.synchronize()
    layers()                                   # sizes the scratch buffers
    ctx.sync()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    ctx.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        layers()
    return dict(ctx=ctx, w=ts, x=x, y=y, graph=graph, stream=stream)


def _run_stack(s):
    s["graph"].replay()
    return s["y"]


def _ffn_weights(c, g):
    return [_weight(g, c["gate"], c["f"], c["d"]), _weight(g, c["gate"], c["f"], c["d"]), _weight(g, c["down"], c["d"], c["f"])]


def _prepare_ffn(c, seed):
    g = _generator(seed)
    w = _ffn_weights(c, g)
    ctx = skn.Context(0)
    shapes = [(c["f"], c["d"])] * 2 + [(c["d"], c["f"])]
    ts = [skn.QuantTensor(ctx, s, TYPE_ID[c[t]], _host(b)) for s, t, (b, _) in zip(shapes, ("gate", "gate", "down"), w)]
    return dict(ctx=ctx, w=ts, m=c["m"], x=_normal(g, c["m"], c["d"]), y=torch.empty(c["m"], c["d"], device="cuda"))


def _run_ffn(s):
    wg, wu, wd = (t.handle for t in s["w"])
    rc = _ffi.lib().skn_ffn_swiglu_dev(s["ctx"].handle, wg, wu, wd, s["x"].data_ptr(), s["m"], s["y"].data_ptr())
    if rc:
        raise RuntimeError(f"skn_ffn_swiglu_dev: {rc}")
    return s["y"]


def _exact_linear(c, seed):
    w, x = _stack_inputs(c, seed)
    wide = [v() for _, v in w[:4]]
    y = torch.stack([a.double() @ wide[i % len(wide)].T for i, a in enumerate(x)])
    return y[0] if c["kind"] == "call" else y


def _exact_ffn(c, seed):
    g = _generator(seed)
    gate, up, down = (v() for _, v in _ffn_weights(c, g))
    x = _normal(g, c["m"], c["d"]).double()
    return (torch.nn.functional.silu(x @ gate.T) * (x @ up.T)) @ down.T


# ---- decode attention --------------------------------------------------------------------------------------------------
def _attend_inputs(c, seed):
    g = _generator(seed)
    lens = torch.randint(c["context"] // 4 + 1, c["context"] + 1, (c["batch"],), generator=g, device="cuda").cpu().numpy().astype(np.int32)
    k, v = (_normal(g, c["batch"], c["kv_heads"], c["context"], c["dim"]) for _ in range(2))
    return lens, k, v, _normal(g, c["batch"], c["heads"], c["dim"])


def _prepare_attend(c, seed):
    lens, k, v, q = _attend_inputs(c, seed)
    ctx = skn.Context(0)
    kv = skn.KVCache(ctx, c["batch"], c["kv_heads"], c["dim"], c["context"] + 128, dtype=c["cache"])
    kv.load(k.cpu().numpy(), v.cpu().numpy(), lens)
    return dict(ctx=ctx, kv=kv, q=q, heads=c["heads"], out=torch.empty_like(q))


def _run_attend(s):
    s["kv"].attend_dev(s["q"], s["heads"], s["out"])
    return s["out"]


def _cached(x, cache):
    """What a cache of this element type holds of x, in fp64."""
    if cache == "f16":
        return x.to(torch.float16).double()
    if cache == "q8_0":
        b = x.reshape(*x.shape[:-1], -1, 32)
        d = b.abs().amax(-1, keepdim=True) / 127
        return (torch.round(b / _away(d)).double() * d.to(torch.float16).double()).reshape(x.shape)
    return x.double()


def _exact_attend(c, seed):
    lens, k, v, q = _attend_inputs(c, seed)
    out, per = torch.empty(q.shape, dtype=torch.float64, device="cuda"), c["heads"] // c["kv_heads"]
    for b, n in enumerate(lens):
        kb, vb = (_cached(t[b, :, :n], c["cache"]).repeat_interleave(per, 0) for t in (k, v))
        p = torch.softmax((kb @ q[b].double()[:, :, None])[..., 0] * c["dim"] ** -0.5, -1)
        out[b] = (p[:, None] @ vb)[:, 0]
    return out


# ---- decoders ------------------------------------------------------------------------------------------------------------
def _tokens(c, seed):
    return np.random.default_rng(seed).integers(0, VOCAB, size=(c["batch"], c["prompt"] + c["steps"])).astype(np.int32)


LLAMA_SHAPES = ("wq", "wk", "wv", "wo", "w_gate", "w_up", "w_down")


def _llama_weights(c, seed):
    g, d, f = _generator(seed), c["width"], c["ffn"]
    kv = c["kv_heads"] * 128
    shapes = dict(zip(LLAMA_SHAPES, ((d, d), (kv, d), (kv, d), (d, d), (f, d), (f, d), (d, f))))
    layer = {n: _weight(g, "q4_k", *s) for n, s in shapes.items()}
    gains = [1 + _normal(g, d, std=0.1) for _ in range(3)]
    return layer, gains, _weight(g, "q6_k", VOCAB, d, std=1.0), _weight(g, "q6_k", VOCAB, d)


def _prepare_llama(c, seed):
    layer, gains, embed, head = _llama_weights(c, seed)
    ctx = skn.Context(0)
    cfg = LlamaConfig(n_layers=c["layers"], d_model=c["width"], n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=128, ffn_dim=c["ffn"], vocab=VOCAB)
    m = LlamaDecoder(ctx, cfg, batch=c["batch"], max_tokens=c["prompt"], max_ctx=c["prompt"] + c["steps"] + 8, kv_dtype=c["cache"])
    raw, g = {n: _host(b) for n, (b, _) in layer.items()}, [_host(x) for x in gains]
    for i in range(c["layers"]):
        m.set_layer(i, raw, g[0], g[1])
    m.set_head(_host(embed[0]), g[2], _host(head[0]))
    return dict(ctx=ctx, model=m, tokens=_tokens(c, seed), prompt=c["prompt"])


def _run_llama(s):
    m, t, p = s["model"], s["tokens"], s["prompt"]
    m.reset()
    out = [m.forward(t[:, :p], want_logits=True)[1]]
    for i in range(p, t.shape[1] - 1):
        out.append(m.forward(t[:, i:i + 1], want_logits=True)[1])
    return out


def _rms(x, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(u, v, dims, base):
    """The pairs (u, v) [.., T, heads, dims / 2] turned by position * base^(-2i / dims)."""
    a = torch.arange(u.shape[-3], device=u.device, dtype=torch.float64)[:, None] * base ** (-2.0 * torch.arange(dims // 2, device=u.device).double() / dims)
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    return u * c - v * s, v * c + u * s


def _rotate_pairs(x, dims, base=10000.0):
    u, v = _turn(x[..., 0:dims:2], x[..., 1:dims:2], dims, base)
    return torch.cat([torch.stack([u, v], -1).flatten(-2), x[..., dims:]], -1)


def _rotate_half(x, dims, base=10000.0):
    return torch.cat([*_turn(x[..., :dims // 2], x[..., dims // 2:dims], dims, base), x[..., dims:]], -1)


def _softmax_attention(q, k, v, scale, seen, softcap=None, sink=None):
    """q [B, T, H, d], k, v [B, T, G, d] in fp64; seen(i, j) says which keys a query has."""
    per = q.shape[2] // k.shape[2]
    at = torch.arange(q.shape[1], device=q.device)
    hide = ~seen(at[:, None], at[None, :])
    out = []
    for h in range(q.shape[2]):
        s = q[:, :, h] @ k[:, :, h // per].transpose(1, 2) * scale
        s = softcap * torch.tanh(s / softcap) if softcap else s
        s = s.masked_fill(hide, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(*s.shape[:2], 1)], -1)
        out.append(torch.softmax(s, -1)[..., :q.shape[1]] @ v[:, :, h // per])
    return torch.stack(out, 2)


def _causal(i, j):
    return j <= i


def _after(c, x):
    """Rows whose logits a request sees: the last of the prompt, then every token but the last."""
    return x[:, c["prompt"] - 1:c["prompt"] + c["steps"] - 1]


def _heads(x, n):
    return x.reshape(*x.shape[:-1], n, -1)


def _exact_llama(c, seed):
    layer, gains, embed, head = _llama_weights(c, seed)
    w = {n: v() for n, (_, v) in layer.items()}
    g = [x.double() for x in gains]
    x = embed[1]()[torch.from_numpy(_tokens(c, seed)).long().cuda()]
    for _ in range(c["layers"]):
        h = _rms(x) * g[0]
        q, k, v = (_heads(h @ w[n].T, a) for n, a in (("wq", c["heads"]), ("wk", c["kv_heads"]), ("wv", c["kv_heads"])))
        k, v = _cached(_rotate_pairs(k, 128).float(), c["cache"]), _cached(v.float(), c["cache"])
        x = x + _softmax_attention(_rotate_pairs(q, 128), k, v, 128 ** -0.5, _causal).flatten(2) @ w["wo"].T
        h = _rms(x) * g[1]
        x = x + (torch.nn.functional.silu(h @ w["w_gate"].T) * (h @ w["w_up"].T)) @ w["w_down"].T
    y = (_rms(_after(c, x)) * g[2]) @ head[1]().T
    return [y[:, i] for i in range(c["steps"])]


def _dense_config(c):
    """The configuration as a checkpoint's config.json holds it."""
    w = c["width"]
    if c["kind"] == "lugasun":
        H, G, D, RH, RD, RV, F, S = LUGASUN[w]
        layer = {"type": "parallel", "mlp": {"ff": F, "kind": "dense"},
                 "mixer": {"left": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5, "softcap": 50.0, "mask": {"size": 1024},
                                    "rot": {"base": 10000.0, "dims": D}},
                           "right": {"heads": RH, "dim": RD, "vdim": RV, "rot": {"base": 10000.0, "dims": RD},
                                     "decay": [1.0 - 2.0 ** -(5 + 5 * h / RH) for h in range(RH)]},
                           "left_scale": 0.5, "right_scale": 0.5}}
        return {"vocab": VOCAB, "width": w, "norm": {"eps": 1e-5}, "layers": [layer] * c["layers"], "token_side": {"dim": S}}
    SH, H, QR, KR, F, EF, SF = TUTEZEN[w]
    part = {"dense": {"kind": "dense", "ff": F},
            "moe": {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP}, "expert": {"ff": EF}, "shared": {"ff": SF}},
            "ssm": {"type": "mamba2", "mixer": {"heads": SH, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}},
            "att": {"type": "latent_attention", "mixer": {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": QR, "kv_rank": KR,
                                                          "scale": 192 ** -0.5, "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 64}}}}
    layers = [dict(part[a], mlp=part[b]) for a, b in map(str.split, TUTEZEN_PATTERN[:c["layers"]])]
    return {"vocab": VOCAB, "width": w, "norm": {"eps": 1e-5}, "residual_mult": 0.5, "layers": layers}


def _dense_classes(kind):
    return (LugasunConfig, skn.LugasunDecoder) if kind == "lugasun" else (TutezenConfig, skn.TutezenDecoder)


def _key(c, name):
    """The name under which layers share a tensor: without the layer, mixers by their kind."""
    at = re.match(r"l(\d+)\.(.*)", name)
    if not at:
        return name
    return TUTEZEN_PATTERN[int(at[1])][:4].replace(" ", ".") + at[2] if c["kind"] == "tutezen" and at[2].startswith("mix.") else at[2]


def _dense_weights(c, seed):
    """shared name -> bf16 tensor; vectors around what training leaves them at, matrices of unit gain."""
    g, out = _generator(seed), {}
    for name, shape in _dense_classes(c["kind"])[0].from_dict(_dense_config(c)).tensor_shapes().items():
        key = _key(c, name)
        if key in out:
            continue
        if key.endswith("A_log"):
            t = torch.log(1 + 15 * torch.rand(*shape, generator=g, device="cuda"))
        elif key.endswith("dt_bias"):
            t = _normal(g, *shape) - 3
        elif key.endswith(("conv.b", "sink")):
            t = _normal(g, *shape, std=0.1)
        elif len(shape) == 1:
            t = 1 + _normal(g, *shape, std=0.1)
        else:
            t = _normal(g, *shape, std=1.0 if "embed" in key else (3.0 if key.endswith("router") else 1.0) * shape[1] ** -0.5)
        if key == "embed":
            t = t * c["width"] ** -0.5           # the output layer's weights too
        out[key] = t.to(torch.bfloat16)
    return out


def _prepare_dense(c, seed):
    bits = {k: v.view(torch.int16).cpu().numpy().view(np.uint16) for k, v in _dense_weights(c, seed).items()}
    conf, cls = _dense_classes(c["kind"])
    ctx = skn.Context(0)
    m = cls(ctx, conf.from_dict(_dense_config(c)), max_seqs=c["batch"], max_tokens=c["batch"] * c["prompt"], max_ctx=c["prompt"] + c["steps"] + 8)
    m.load(lambda name, shape: bits[_key(c, name)])
    return dict(ctx=ctx, model=m, tokens=_tokens(c, seed), prompt=c["prompt"])


def _run_dense(s):
    m, t, p = s["model"], s["tokens"], s["prompt"]
    n = t.shape[0]
    m.reset()
    out = [m.forward(t[:, :p], want=[p * (b + 1) - 1 for b in range(n)])[1]]
    for i in range(p, t.shape[1] - 1):
        out.append(m.forward(t[:, i:i + 1], want=range(n))[1])
    return out


def _exact_dense(c, seed):
    w = {k: v.double() for k, v in _dense_weights(c, seed).items()}
    cfg, tokens = _dense_config(c), torch.from_numpy(_tokens(c, seed)).long().cuda()
    x = w["embed"][tokens]
    for i, layer in enumerate(cfg["layers"]):
        h = _rms(x) * w["norm1"]
        if c["kind"] == "lugasun":
            m, d = layer["mixer"], cfg["token_side"]["dim"]
            x = x + m["left_scale"] * _chunk_mixer(w, m["left"], h) + m["right_scale"] * _retention_mixer(w, m["right"], h)
            h = _rms(x) * w["norm2"]
            x = x + torch.relu(h @ w["mlp.up"].T) ** 2 @ w["mlp.down"].T
            g = torch.nn.functional.gelu(x @ w["side.gate"].T, approximate="tanh") * w["side.embed"][tokens][..., i * d:(i + 1) * d]
            x = x + _rms(g @ w["side.proj"].T) * w["side.norm"]
        else:
            y = (_ssm_mixer if layer["type"] == "mamba2" else _latent_mixer)(w, layer["mixer"], h)
            x = x + cfg["residual_mult"] * (y + (_experts if layer["mlp"]["kind"] == "moe" else _dense_ff)(w, h))
    y = (_rms(_after(c, x)) * w["final.norm"]) @ w["embed"].T
    return [y[:, i] for i in range(c["steps"])]


def _chunk_mixer(w, m, h):
    p, n = "mix.left.", m["mask"]["size"]
    q, k, v = (_heads(h @ w[p + a].T, m["heads"] if a == "q" else m["kv_heads"]) for a in "qkv")
    q, k = (_rotate_half(_rms(a) * w[p + b + ".norm"], m["rot"]["dims"]) for a, b in ((q, "q"), (k, "k")))
    o = _softmax_attention(q, k, v, m["scale"], lambda i, j: (j <= i) & (i // n == j // n), m["softcap"])
    return o.flatten(2) @ w[p + "o"].T


def _retention_mixer(w, m, h):
    p = "mix.right."
    q, k, v = (_heads(h @ w[p + a].T, m["heads"]) for a in "qkv")
    q, k = (_rotate_half(a, m["rot"]["dims"]) for a in (q, k))
    at = torch.arange(h.shape[1], device=h.device).double()
    apart = at[:, None] - at[None, :]
    o = []
    for n in range(m["heads"]):
        fade = torch.where(apart >= 0, m["decay"][n] ** apart.clamp(min=0), 0.0)
        o.append((q[:, :, n] @ k[:, :, n].transpose(1, 2) * m["dim"] ** -0.5 * fade) @ v[:, :, n])
    o = _rms(torch.stack(o, 2)).flatten(2)
    return (o * torch.nn.functional.silu(h @ w[p + "g"].T)) @ w[p + "o"].T


def _ssm_mixer(w, m, h):
    H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    B, T = h.shape[:2]
    z, u, dt = torch.split(h @ w["ssm.mix.in"].T, [H * V, H * V + 2 * G * N, H], -1)
    conv = w["ssm.mix.conv"]
    u = torch.nn.functional.pad(u, (0, 0, conv.shape[1] - 1, 0))
    u = torch.nn.functional.silu(sum(conv[:, t] * u[:, t:t + T] for t in range(conv.shape[1])) + w["ssm.mix.conv.b"])
    x, b, k = torch.split(u, [H * V, G * N, G * N], -1)
    x, b, k = _heads(x, H), _heads(b, G).repeat_interleave(H // G, 2), _heads(k, G).repeat_interleave(H // G, 2)
    dt = torch.nn.functional.softplus(dt + w["ssm.mix.dt_bias"])
    fade = torch.exp(-torch.exp(w["ssm.mix.A_log"]) * dt)
    S, y = torch.zeros(B, H, N, V, dtype=h.dtype, device=h.device), []
    for t in range(T):
        S = fade[:, t, :, None, None] * S + (dt[:, t, :, None] * b[:, t])[..., None] * x[:, t, :, None]
        y.append((k[:, t, :, None] @ S)[:, :, 0])
    y = (torch.stack(y, 1) + w["ssm.mix.D"][:, None] * x).flatten(2) * torch.nn.functional.silu(z)
    return (_rms(_heads(y, m["norm_groups"])).flatten(2) * w["ssm.mix.norm"]) @ w["ssm.mix.o"].T


def _latent_mixer(w, m, h):
    H, D, R, K, n = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["mask"]["size"]
    q = _heads((_rms(h @ w["att.mix.dq"].T) * w["att.mix.dq.norm"]) @ w["att.mix.uq"].T, H)
    u = h @ w["att.mix.dkv"].T
    c = _rms(u[..., :K]) * w["att.mix.dkv.norm"]
    turned = _rotate_pairs(u[..., None, K:], m["rot"]["dims"]).expand(*u.shape[:2], H, R)
    q = torch.cat([q[..., :D], _rotate_pairs(q[..., D:], m["rot"]["dims"])], -1)
    k, v = torch.cat([_heads(c @ w["att.mix.uk"].T, H), turned], -1), _heads(c @ w["att.mix.uv"].T, H)
    o = _softmax_attention(q, k, v, m["scale"], lambda i, j: (j <= i) & (i - j < n), sink=w["att.mix.sink"])
    return (o.flatten(2) * torch.sigmoid(h @ w["att.mix.g"].T)) @ w["att.mix.o"].T


def _dense_ff(w, h):
    return torch.nn.functional.gelu(h @ w["mlp.up"].T, approximate="tanh") @ w["mlp.down"].T


def _gated(w, p, h):
    return (torch.nn.functional.silu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T


def _experts(w, h):
    s, chosen = torch.topk(torch.softmax(h @ w["mlp.router"].T, -1), TOP, -1)
    s = torch.zeros(*h.shape[:2], EXPERTS, dtype=h.dtype, device=h.device).scatter_(-1, chosen, s / s.sum(-1, keepdim=True))
    return sum(s[..., e:e + 1] * _gated(w, f"mlp.e{e}.", h) for e in range(EXPERTS)) + _gated(w, "mlp.shared.", h)


# ---- the interface ----------------------------------------------------------------------------------------------------
KINDS = {
    "call": (_prepare_call, lambda s: s["w"].matmul_t(s["x"]), _exact_linear),
    "stack": (_prepare_stack, _run_stack, _exact_linear),
    "ffn": (_prepare_ffn, _run_ffn, _exact_ffn),
    "attend": (_prepare_attend, _run_attend, _exact_attend),
    "llama": (_prepare_llama, _run_llama, _exact_llama),
    "lugasun": (_prepare_dense, _run_dense, _exact_dense),
    "tutezen": (_prepare_dense, _run_dense, _exact_dense),
}


def prepare(case, seed):
    state = KINDS[case["kind"]][0](case, seed)
    torch.cuda.synchronize()
    return dict(state, kind=case["kind"])


def run(state):
    return KINDS[state["kind"]][1](state)


def exact(case, seed):
    return KINDS[case["kind"]][2](case, seed)


def work(case):
    """Weights and inputs read once, outputs written once; two operations per weight and row."""
    c, kind = case, case["kind"]

    def size(t, n, k):
        return n * (k // BLOCK[t][0]) * BLOCK[t][1]

    if kind in ("call", "stack"):
        layers = c.get("layers", 1)
        return dict(bytes=layers * (size(c["type"], c["n"], c["k"]) + 4 * c["m"] * (c["n"] + c["k"])), flops=2 * layers * c["m"] * c["n"] * c["k"])
    if kind == "ffn":
        return dict(bytes=2 * size(c["gate"], c["f"], c["d"]) + size(c["down"], c["d"], c["f"]) + 8 * c["m"] * c["d"], flops=6 * c["m"] * c["d"] * c["f"])
    if kind == "attend":
        tokens = c["batch"] * c["context"] * 5 / 8         # lengths are uniform between a quarter and all of the context
        per = {"f32": 4.0, "f16": 2.0, "q8_0": 1.0625}[c["cache"]]
        return dict(bytes=2 * tokens * c["kv_heads"] * c["dim"] * per + 8 * c["batch"] * c["heads"] * c["dim"], flops=4 * tokens * c["heads"] * c["dim"])
    # decoders: the layers' weights once for the prompt and once for each of the tokens that follow, the head for each row that it is asked for
    B, P, steps = c["batch"], c["prompt"], c["steps"]
    rows, d = B * (P + steps - 1), c["width"]
    if kind == "llama":
        kv = c["kv_heads"] * 128
        n = c["layers"] * (2 * d * d + 2 * kv * d + 3 * d * c["ffn"])
        near, dots = n, 2 * c["layers"] * c["heads"] * 128 * B * (P + steps) ** 2
        layer_bytes, head_bytes = n // 256 * 144, size("q6_k", VOCAB, d)
    else:
        conf = _dense_classes(kind)[0].from_dict(_dense_config(c))
        sizes = {k: math.prod(s) for k, s in conf.tensor_shapes().items() if k[0] == "l" and k[1].isdigit()}
        routed = sum(v for k, v in sizes.items() if ".mlp.e" in k)
        n, near = sum(sizes.values()), sum(sizes.values()) - routed + routed * TOP // EXPERTS
        shared = near if B * P == 1 else n                 # experts that a prompt's rows meet, taken as all of them
        dots, head_bytes = 0, 2 * VOCAB * d
        layer_bytes = (2 * shared + 2 * (steps - 1) * (near if B == 1 else n)) / steps
    return dict(bytes=steps * (layer_bytes + head_bytes) + 4 * B * steps * VOCAB, flops=2 * near * rows + 2 * VOCAB * d * B * steps + dots)


def tolerance(case):
    c, kind = case, case["kind"]
    if kind == "attend":
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("call", "stack") and c["m"] < 64:
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("call", "stack", "ffn"):
        return {"rel": 1e-2, "max": 0.1}                   # bf16 operands
    if kind == "llama" and c["batch"] * c["prompt"] < 64:
        return {"rel": 1e-4, "max": 1e-3}                  # fp32 throughout
    return {"rel": 0.03, "max": 0.4}                       # bf16 operands through all layers
