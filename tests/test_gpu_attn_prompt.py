"""Causal attention of many queries against fp64 on what the cache holds, on the tensor cores (three bf16 terms per fp32 operand) and where the rule
leaves it to the split kernels: edges of tiles of 64 (query, head) rows and 32 keys, rings that wrap, queries before the first key, operands
without finite bf16 terms, few queries over many keys."""
import ctypes
import math

import numpy as np
import pytest
import torch

import skainet_b200 as skn
from skainet_b200 import _ffi, synth

pytestmark = pytest.mark.gpu


def causal(ctx, kv, q, T, scale):
    qd = torch.from_numpy(q).cuda()
    out = torch.full_like(qd, np.nan)
    torch.cuda.synchronize()
    rc = _ffi.lib().skn_attn_causal_dev(kv.handle, qd.data_ptr(), q.shape[2], T, ctypes.c_float(scale), out.data_ptr(), None)
    assert rc == 0
    ctx.sync()
    return out.cpu().numpy()


def routed(ctx, kv, q, T, scale):
    """The same with the caller's scratch memory, and whether the tensor-core kernel took the call: it leaves that alone."""
    qd = torch.from_numpy(q).cuda()
    out, scratch = torch.full_like(qd, np.nan), torch.full((T * kv.scratch_bytes(q.shape[2]) // 4,), 7.0, device="cuda")
    torch.cuda.synchronize()
    rc = _ffi.lib().skn_attn_causal_dev(kv.handle, qd.data_ptr(), q.shape[2], T, ctypes.c_float(scale), out.data_ptr(), scratch.data_ptr())
    assert rc == 0
    ctx.sync()
    return out.cpu().numpy(), bool((scratch == 7.0).all())


def faster(B, Hkv, G, D, dtype, T, keys):
    """The rule of skn_attn_prompt_faster: estimated microseconds of the split kernels and of the tensor-core kernel."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    heads, seen, q8, f16 = B * Hkv, keys - T / 2, dtype == "q8_0", dtype == "f16"
    per = {(64, 0): (.061, .037, .025, .024), (128, 0): (.075, .047, .031, .031), (64, 1): (.081, .045, .028, .021), (128, 1): (.093, .053, .034, .032)}[D, q8]
    split = 14 + heads * G * T / 1000 * (seen * per[int(math.log2(G))] + 4 * min(1, keys / 256))
    key = {"f32": (.057, .108), "f16": (.055, .115), "q8_0": (.071, .131)}[dtype][D == 128] * (1.4 if f16 and heads * keys * D * 4 > 48e6 else 1)
    ctas = heads * -(-T * G // 64)
    return heads * G * T >= 2048 and 12 + key * max(keys, 32, -(-ctas // sms) * seen) + 1 <= split


def held(kv):
    """What the cache holds, per sequence: k, v [kv heads, len, dim] in fp64."""
    lens, _ = kv.lengths()
    return [tuple(torch.from_numpy(x.astype(np.float64)) for x in kv.gather(b, 0, int(n))) for b, n in enumerate(lens)]


def expected(pairs, q, scale):
    """fp64 outputs, and the weighted sums of |v| that their errors are measured by."""
    B, T, Hq, D = q.shape
    ref, size = (np.zeros((B, T, Hq, D)) for _ in range(2))
    for b, (k, v) in enumerate(pairs):
        per, n = Hq // k.shape[0], k.shape[1]
        s = torch.einsum("thd,hjd->htj", torch.from_numpy(q[b].astype(np.float64)), k.repeat_interleave(per, 0)) * scale
        seen = torch.arange(n)[None] <= n - T + torch.arange(T)[:, None]
        some = seen.any(1).numpy()
        p = torch.softmax(s.masked_fill(~seen, -np.inf), -1)
        for to, x in ((ref, v), (size, v.abs())):
            to[b][some] = torch.einsum("htj,hjd->thd", p, x.repeat_interleave(per, 0)).numpy()[some]
    return ref, size


def check(out, pairs, q, scale):
    """Scores: a chain of six products per 16 elements and one addition each, every one within 2^-23 of sums of |q k| (at most `big` here);
    an error of a score moves a weight by as much, relatively, and the outputs' own sums add a few 2^-23 more."""
    ref, size = expected(pairs, q, scale)
    big = max(float((torch.from_numpy(q[b]).double().abs().amax((0, 1)) * k.abs().amax((0, 1))).sum()) * scale for b, (k, _) in enumerate(pairs) if k.shape[1])
    assert np.all(np.abs(out - ref) <= (2 * big + 32) * 2.0 ** -23 * size)
    assert np.linalg.norm(out - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("dtype", ["f32", "f16", "q8_0"])
@pytest.mark.parametrize("B,Hkv,G,D,T,cap,lens", [
    (1, 8, 4, 128, 64, 64, [64]), (1, 8, 4, 128, 65, 400, [97]), (2, 4, 8, 64, 33, 300, [33, 260]), (3, 8, 1, 64, 129, 161, [161, 130, 129]),
    (4, 8, 2, 128, 47, 96, [96, 48, 47, 50]), (1, 32, 1, 128, 64, 1000, [1000]), (16, 8, 8, 128, 2, 70, [2 + 4 * i for i in range(16)]),
    (9, 8, 4, 128, 20, 32, [20, 32, 31, 21, 32, 25, 24, 30, 32]), (5, 4, 8, 64, 17, 31, [17, 31, 18, 30, 24])])
def test_prompt_attention(ctx, B, Hkv, G, D, T, cap, lens, dtype):
    g = synth.rng(T + cap + D)
    kv = skn.KVCache(ctx, B, Hkv, D, cap, dtype=dtype)
    k, v = (g.standard_normal((B, Hkv, cap, D), dtype=np.float32) for _ in range(2))
    kv.load(k, v, np.array(lens, dtype=np.int32))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32)
    check(causal(ctx, kv, q, T, D ** -0.5), held(kv), q, D ** -0.5)
    for _ in range(5):                                     # rings that were full go on: their first token is not in slot 0 any more
        kv.append(*(g.standard_normal((B, Hkv, D), dtype=np.float32) for _ in range(2)))
    check(causal(ctx, kv, q, T, D ** -0.5), held(kv), q, D ** -0.5)
    kv.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "q8_0"])
@pytest.mark.parametrize("B,Hkv,G,D,T,cap,lens", [
    (2, 8, 4, 128, 64, 64, [64, 64]), (2, 8, 4, 128, 65, 400, [97, 400]), (4, 4, 8, 64, 33, 300, [33, 260, 299, 64]), (3, 8, 1, 128, 129, 161, [161, 130, 129]),
    (4, 8, 2, 128, 47, 96, [96, 48, 47, 50]), (1, 32, 1, 128, 64, 1000, [1000]), (16, 8, 8, 128, 5, 70, [5 + 4 * i for i in range(16)]),
    (9, 8, 4, 128, 20, 32, [20, 32, 31, 21, 32, 25, 24, 30, 32]), (9, 8, 4, 128, 20, 33, [20, 33, 31, 21, 32, 25, 24, 30, 32]),
    (9, 4, 8, 64, 17, 31, [17, 31, 18, 30, 24, 31, 31, 17, 20]), (1, 8, 4, 128, 200, 1300, [1300])])
def test_prompt_attention_on_the_tensor_cores(ctx, B, Hkv, G, D, T, cap, lens, dtype):
    g = synth.rng(T + cap + D)
    kv = skn.KVCache(ctx, B, Hkv, D, cap, dtype=dtype)
    k, v = (g.standard_normal((B, Hkv, cap, D), dtype=np.float32) for _ in range(2))
    kv.load(k, v, np.array(lens, dtype=np.int32))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32)
    out, taken = routed(ctx, kv, q, T, D ** -0.5)
    assert taken
    check(out, held(kv), q, D ** -0.5)
    assert np.array_equal(out, causal(ctx, kv, q, T, D ** -0.5))
    for _ in range(5):                                     # rings that were full go on: their first token is not in slot 0 any more
        kv.append(*(g.standard_normal((B, Hkv, D), dtype=np.float32) for _ in range(2)))
    check(causal(ctx, kv, q, T, D ** -0.5), held(kv), q, D ** -0.5)
    kv.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "q8_0"])
@pytest.mark.parametrize("B,Hkv,G,D,T,keys,taken", [
    (1, 8, 4, 128, 64, 4000, False), (1, 8, 4, 128, 100, 2000, False), (1, 8, 4, 128, 256, 2000, True), (1, 4, 8, 128, 64, 1500, False), (4, 8, 4, 128, 16, 2000, False),
    (4, 8, 4, 128, 64, 1000, True), (16, 8, 8, 128, 2, 500, False), (1, 8, 2, 128, 128, 1000, False), (1, 8, 2, 128, 256, 1000, True), (1, 8, 1, 64, 256, 1500, True),
    (1, 2, 1, 128, 1024, 1024, False), (1, 2, 4, 128, 256, 1000, False), (1, 8, 4, 128, 63, 100, False)])
def test_few_queries_over_many_keys_are_left_to_the_split_kernels(ctx, B, Hkv, G, D, T, keys, dtype, taken):
    """A CTA of the tensor-core kernel walks all keys whatever the number of CTAs: which kernel runs, and that both are right."""
    assert faster(B, Hkv, G, D, dtype, T, keys) == taken
    g = synth.rng(T + keys + D)
    kv = skn.KVCache(ctx, B, Hkv, D, keys, dtype=dtype)
    k, v = (g.standard_normal((B, Hkv, keys, D), dtype=np.float32) for _ in range(2))
    kv.load(k, v, np.full(B, keys, dtype=np.int32))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32)
    out, tensor_cores = routed(ctx, kv, q, T, D ** -0.5)
    assert tensor_cores == taken
    check(out, held(kv), q, D ** -0.5)
    check(causal(ctx, kv, q, T, D ** -0.5), held(kv), q, D ** -0.5)
    kv.close()


def test_a_captured_call_without_scratch_memory():
    """While a graph is captured nothing can be allocated: the tensor-core kernel takes what the rule would leave to the split kernels."""
    with skn.Context(0) as own:
        g = synth.rng(21)
        Hkv, G, D, T, keys = 8, 4, 128, 64, 2000
        kv = skn.KVCache(own, 1, Hkv, D, keys)
        kv.load(*(g.standard_normal((1, Hkv, keys, D), dtype=np.float32) for _ in range(2)), np.array([keys], dtype=np.int32))
        q = g.standard_normal((1, T, Hkv * G, D), dtype=np.float32)
        qd = torch.from_numpy(q).cuda()
        out = torch.full_like(qd, np.nan)
        torch.cuda.synchronize()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        own.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
            rc = _ffi.lib().skn_attn_causal_dev(kv.handle, qd.data_ptr(), Hkv * G, T, ctypes.c_float(D ** -0.5), out.data_ptr(), None)
        assert rc == 0
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        check(out.cpu().numpy(), held(kv), q, D ** -0.5)
        kv.close()


def test_queries_before_the_first_key_are_zero(ctx):
    g = synth.rng(3)
    B, Hkv, G, D, T, cap = 3, 8, 4, 128, 70, 100
    kv = skn.KVCache(ctx, B, Hkv, D, cap)
    k, v = (g.standard_normal((B, Hkv, cap, D), dtype=np.float32) for _ in range(2))
    kv.load(k, v, np.array([0, 3, 69], dtype=np.int32))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32)
    out = causal(ctx, kv, q, T, 0.1)
    assert not out[0].any() and not out[1, :67].any() and not out[2, 0].any()
    check(out, held(kv), q, 0.1)
    kv.close()


@pytest.mark.parametrize("T", [80, 128])
@pytest.mark.parametrize("size_q,size_k,size_v", [(1.0, 1.0, 1e30), (1e-12, 1e12, 1e-30), (30.0, 1.0, 1.0)])
def test_sizes_of_values(ctx, size_q, size_k, size_v, T):
    """One element in eight is a thousand times the others: every term keeps its own 24 bits."""
    g = synth.rng(7)
    B, Hkv, G, D = 1, 8, 4, 128
    kv = skn.KVCache(ctx, B, Hkv, D, T)
    k, v = (g.standard_normal((B, Hkv, T, D), dtype=np.float32) * size for size in (size_k, size_v))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32) * size_q
    k[..., ::8] *= 1e-3
    v[..., ::8] *= 1e3
    kv.load(k.astype(np.float32), v.astype(np.float32), np.array([T], dtype=np.int32))
    q = q.astype(np.float32)
    check(causal(ctx, kv, q, T, D ** -0.5), held(kv), q, D ** -0.5)
    kv.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3.4e38])
@pytest.mark.parametrize("where", ["k", "v"])
def test_what_is_not_finite_reaches_no_earlier_query(ctx, where, value):
    g = synth.rng(11)
    B, Hkv, G, D, T, at = 1, 8, 4, 128, 100, 70
    assert faster(B, Hkv, G, D, "f32", T, T)
    k, v = (g.standard_normal((B, Hkv, T, D), dtype=np.float32) for _ in range(2))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32)
    (k if where == "k" else v)[0, 2, at, 5] = value
    kv = skn.KVCache(ctx, B, Hkv, D, T)
    kv.load(k, v, np.array([T], dtype=np.int32))
    out = causal(ctx, kv, q, T, D ** -0.5)
    kv.close()
    pair = lambda a, b: [tuple(torch.from_numpy(x[0].astype(np.float64)) for x in (a, b))]
    with np.errstate(all="ignore"):
        ref, size = expected(pair(k, v), q, D ** -0.5)
    k[0, 2, at, 5] = v[0, 2, at, 5] = 0.0                                           # (a reference's own zero weight would not keep NaN away)
    early, early_size = expected(pair(k, v), q, D ** -0.5)
    ref[:, :at], size[:, :at] = early[:, :at], early_size[:, :at]
    fp32 = np.abs(ref) < 3e38
    hit = np.zeros(out.shape, dtype=bool)                                           # heads 8 .. 11 from token 70 on
    hit[:, at:, 8:12] = True
    assert np.isfinite(out[~hit]).all()
    assert np.all(np.abs(out - ref)[~hit] <= 2.0 ** -17 * size[~hit])
    if where == "v":
        col = np.zeros_like(hit)
        col[:, at:, 8:12, 5] = True
        if np.isfinite(value):
            assert np.all((np.abs(out - ref) <= 2.0 ** -17 * size)[hit & fp32])
        else:                                                                      # its own column alone, of the value's kind
            assert np.all((np.abs(out - ref) <= 2.0 ** -17 * size)[hit & ~col])
            assert np.isnan(out[col]).all() if np.isnan(value) else np.all((out[col] == value) | np.isnan(out[col]))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3.4e38, -3.4e38])
@pytest.mark.parametrize("B,Hkv,G,D,T,keys,dtype", [(1, 8, 4, 128, 100, 100, "f32"), (1, 8, 4, 64, 128, 700, "f16"), (1, 8, 4, 128, 200, 700, "q8_0"), (9, 8, 4, 128, 20, 32, "f32")])
def test_what_is_not_finite_in_a_query_reaches_no_other(ctx, B, Hkv, G, D, T, keys, dtype, value):
    """A query off the range that three bf16 terms have: the scores of one that is finite are those of fp32, against keys so small there that they are ordinary."""
    assert faster(B, Hkv, G, D, dtype, T, keys)
    g, at = synth.rng(12), T // 2
    k, v = (g.standard_normal((B, Hkv, keys, D), dtype=np.float32) for _ in range(2))
    q = g.standard_normal((B, T, Hkv * G, D), dtype=np.float32) * np.float32(0.1)
    k[..., 5] *= 1e-38
    q[0, at, 9, 5] = value
    kv = skn.KVCache(ctx, B, Hkv, D, keys, dtype=dtype)
    kv.load(k, v, np.full(B, keys, dtype=np.int32))
    out, pairs = causal(ctx, kv, q, T, 1.0), held(kv)
    kv.close()
    rows = np.ones(out.shape, dtype=bool)
    if not np.isfinite(value):
        rows[0, at, 9] = False
        assert np.isnan(out[~rows]).all()
        q[0, at, 9, 5] = 0.0
    ref, size = expected(pairs, q, 1.0)
    assert np.isfinite(out[rows]).all()
    assert np.all(np.abs(out - ref)[rows] <= 2.0 ** -17 * size[rows])
