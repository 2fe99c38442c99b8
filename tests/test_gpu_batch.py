"""Batches of 9 to 63 activation rows (tcgen05 with exact fp16 integers) against the fp64 oracle, at the edges of chunks, tiles,
launches and parts of K; the tolerance of the single-row kernels."""
import threading

import numpy as np
import pytest
import torch

import skainet_b200 as skn
from conftest import FP32_TOL, assert_close_dot
from oracle import oracle
from skainet_b200 import synth
from skainet_b200.llama import LlamaConfig, LlamaDecoder
from test_gpu_matvec import _zero_weight_at as zero_weight_at

pytestmark = pytest.mark.gpu
TYPES = [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K]


def check(ctx, qt, w, x, N, K, bias=None):
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y = t.matmul_t(x, bias)
    t.close()
    ref, absdot = oracle.matmul(qt, w, N, K, x)
    if bias is not None:
        ref, absdot = ref + bias.astype(np.float64), absdot + np.abs(bias.astype(np.float64))
    assert_close_dot(y, ref, absdot, FP32_TOL, f"type {qt} {N}x{K} M={x.shape[0]}")


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("M,N,K", [(9, 1, 256), (16, 127, 512), (17, 130, 768), (24, 128, 2304), (25, 300, 1024), (32, 16, 4096), (33, 257, 256), (63, 40, 1792)])
def test_batch_edges(ctx, qt, M, N, K):
    g = synth.rng(M + N + K)
    check(ctx, qt, synth.make_weight(g, qt, N, K), synth.make_activations(g, M, K), N, K, g.standard_normal(N).astype(np.float32) if M % 2 else None)


@pytest.mark.parametrize("M", [9, 16, 17])
@pytest.mark.parametrize("N,K", [(16 * 148, 512), (16 * 148 + 1, 512), (333, 768), (333, 1024)])
def test_short_rows_on_both_sides_of_the_rule(ctx, N, K, M):
    """Q4_K rows of two and three super-blocks, one group of 16 weight rows per SM and 16 activation rows at most: the many-row kernel."""
    g = synth.rng(N + K + M)
    check(ctx, synth.Q4_K, synth.make_weight(g, synth.Q4_K, N, K), synth.make_activations(g, M, K), N, K, g.standard_normal(N).astype(np.float32))


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("zero_weight", [False, True])
def test_batch_outliers_zeros_and_scales(ctx, qt, zero_weight):
    """Rows of zeros, of one element, of very different sizes, and of two outliers in every 256 elements, up to 1e6 times the others.  They meet
    ordinary weights (an outlier's own product), or zero weights: then the bound is that of the others alone, which a fixed-point
    form with the outliers left in would miss by far (2^-30 of 4e6)."""
    g = synth.rng(5)
    M, N, K = 12, 48, 1024
    w = synth.make_weight(g, qt, N, K)
    cols = np.sort(np.concatenate([np.arange(5, K, 256), np.arange(130, K, 256)]))
    if zero_weight:
        e = synth.GEOMETRY[qt][0]
        for first in (5, 130):
            pos = np.full(K // e, -1)
            pos[np.arange(first, K, 256) // e] = first % e
            keep, w0 = pos < 0, w.reshape(N, K // e, -1).copy()
            w = zero_weight_at(qt, w, N, K, np.where(keep, 0, pos))
            w.reshape(N, K // e, -1)[:, keep] = w0[:, keep]
        assert np.all(oracle.dequant(qt, w).reshape(N, K)[:, cols] == 0.0)
    x = synth.make_activations(g, M, K)
    x[0] = 0
    x[1] = 0
    x[1, 700] = 3.5
    for m, size in ((2, 1e3), (3, 1e4), (4, 1e6)):
        x[m, 5::256] *= size
        x[m, 130::256] *= -size
    x[5] *= 1e-20
    x[6] *= 1e20
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y = t.matmul_t(x)
    t.close()
    ref, absdot = oracle.matmul(qt, w, N, K, x)
    for m in range(M):
        assert_close_dot(y[m], ref[m], absdot[m], FP32_TOL, f"type {qt} row {m}")


@pytest.mark.parametrize("qt", TYPES)
def test_batch_rows_that_are_not_finite_stay_apart(ctx, qt):
    g = synth.rng(6)
    M, N, K = 10, 33, 512
    w, x = synth.make_weight(g, qt, N, K), synth.make_activations(g, M, K)
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    clean = t.matmul_t(x)
    x[3, 17], x[7, 300] = np.inf, np.nan
    y = t.matmul_t(x)
    t.close()
    assert not np.isfinite(y[3]).any() and not np.isfinite(y[7]).any()
    keep = [m for m in range(M) if m not in (3, 7)]
    assert np.array_equal(y[keep], clean[keep])


def _near_the_largest(g, qt, n, k):
    """Blocks of positive weights whose quants and integer scales are at or near their largest, d a power of two."""
    half = np.frombuffer(np.float16(2.0 ** -6).tobytes(), dtype=np.uint8)
    nibbles = lambda *shape: (0xEE | g.integers(0, 2, shape) | g.integers(0, 2, shape) << 4).astype(np.uint8)        # 14 and 15
    if qt == synth.Q4_K:
        b = np.zeros((n, k // 256, 144), dtype=np.uint8)
        sc = g.integers(61, 64, (n, k // 256, 8)).astype(np.uint8)
        b[..., 0:2], b[..., 16:] = half, nibbles(n, k // 256, 128)
        b[..., 4:8], b[..., 12:16] = sc[..., :4] | sc[..., 4:] >> 4 << 6, sc[..., 4:] & 15
    elif qt == synth.Q6_K:
        b = np.full((n, k // 256, 210), 0xFF, dtype=np.uint8)
        b[..., 208:], b[..., :128], b[..., 192:208] = half, nibbles(n, k // 256, 128), g.integers(118, 128, (n, k // 256, 16))
    elif qt == synth.Q4_0:
        b = np.zeros((n, k // 32, 18), dtype=np.uint8)
        b[..., :2], b[..., 2:] = half, nibbles(n, k // 32, 16)
    else:
        b = np.zeros((n, k // 32, 34), dtype=np.uint8)
        b[..., :2], b[..., 2:] = half, g.integers(118, 128, (n, k // 32, 32))
    return b.reshape(-1)


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("K", [256, 4096])
@pytest.mark.parametrize("digit", [0, -128, 127])
def test_batch_sums_of_one_sign_are_exact(ctx, qt, K, digit):
    """Activations and weights of one sign near their largest, with the second byte digit of the activations near `digit`: the integer sums
    are the largest there are.  They are exact, so what is left are roundings to nearest: joining the digits (3), sums of x and
    offset, scale and accumulation of a super-block (4) and the parts of K (2), each at most 2^-24 of a sum of terms of one sign --
    and without a preferred direction: the mean over some thousand outputs is far below one of them."""
    g = synth.rng(K + digit + 200)
    M, N = 12 if K == 256 else 30, 256
    w = _near_the_largest(g, qt, N, K)
    top, low = g.integers(56, 63, (M, K)), g.integers(-128, 128, (M, K))
    second = np.clip(digit + g.integers(-3, 4, (M, K)), -128, 127)
    x = ((top * 2.0 ** 24 + second * 2.0 ** 16 + low * 2.0 ** 8) * 2.0 ** -29).astype(np.float32)       # at most 23 bits: exact
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y = t.matmul_t(x)
    t.close()
    ref, _ = oracle.matmul(qt, w, N, K, x)
    err = (y - ref) / ref
    assert np.abs(err).max() <= (9 + K // 256 / 8) * 2.0 ** -24
    assert abs(err.mean()) <= 2.0 ** -26


def _captured(ctx, t, x, y):
    """A graph of one product on a stream of its own."""
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    ctx.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        t.matmul_t_dev(x, x.shape[0], y)
    ctx.set_stream(None)
    return graph


@pytest.mark.parametrize("qt,M", [(synth.Q4_K, 30), (synth.Q6_K, 30), (synth.Q8_0, 9)])
def test_batch_captured_before_its_buffer_is_large_enough(qt, M):
    """Nothing can be allocated while a graph is captured: a route takes the call that needs no larger buffer than there is.  Q6_K has one
    without any; the others' takes up to 16 rows a launch and has what a call of five rows left."""
    g = synth.rng(11)
    N, K = 256, 8192
    w, x = synth.make_weight(g, qt, N, K), torch.from_numpy(synth.make_activations(g, M, K)).cuda()
    ctx = skn.Context(0)
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y = torch.zeros(M, N, device="cuda")
    if qt != synth.Q6_K:
        torch.cuda.synchronize()
        t.matmul_t_dev(x, 5, y)
        ctx.sync()
    graph = _captured(ctx, t, x, y)
    graph.replay()
    torch.cuda.synchronize()
    ref, absdot = oracle.matmul(qt, w, N, K, x.cpu().numpy())
    assert_close_dot(y.cpu().numpy(), ref, absdot, FP32_TOL, f"type {qt}")
    del graph
    t.close()
    ctx.close()


@pytest.mark.parametrize("qt", TYPES)
def test_batch_graph_outlives_a_larger_call(qt):
    """A later call whose prepared activations need a larger buffer leaves the one a captured graph works in."""
    g = synth.rng(12)
    ctx = skn.Context(0)
    small, large = (skn.QuantTensor(ctx, s, qt, synth.make_weight(g, qt, *s)) for s in ((256, 512), (16, 32768)))
    x, big = (torch.from_numpy(synth.make_activations(g, *s)).cuda() for s in ((16, 512), (32, 32768)))
    y, y_big = torch.zeros(16, 256, device="cuda"), torch.zeros(32, 16, device="cuda")
    torch.cuda.synchronize()
    small.matmul_t_dev(x, 16, y)
    ctx.sync()
    want = y.clone()
    graph = _captured(ctx, small, x, y)
    large.matmul_t_dev(big, 32, y_big)
    ctx.sync()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    del graph
    small.close()
    large.close()
    ctx.close()


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("M", [17, 24, 32])
@pytest.mark.parametrize("N,K", [(14336, 2560), (1000, 14336)])
def test_batch_rings_wrap(ctx, qt, N, K, M):
    """Enough super-blocks per CTA (ten; seven of eight parts of K) that every ring is refilled several times, three and four chunks of rows; sampled outputs."""
    g = synth.rng(N + M)
    some = synth.make_weight(g, qt, 256, K).reshape(256, -1)
    w = np.ascontiguousarray(some[np.arange(N) % 256])
    x = synth.make_activations(g, M, K)
    t = skn.QuantTensor(ctx, (N, K), qt, w.reshape(-1))
    y = t.matmul_t(x)
    t.close()
    rows = np.unique(np.concatenate([g.choice(N, size=60, replace=False), [0, N - 1]]))
    ref, absdot = oracle.matmul(qt, np.ascontiguousarray(w[rows]), rows.size, K, x)
    assert_close_dot(y[:, rows], ref, absdot, FP32_TOL, f"type {qt} {N}x{K} M={M}")
    assert np.array_equal(y[:, 256:512], y[:, :256])                 # the same weights in other tiles: the same bits


def test_batch_at_the_longest_row(ctx):
    g = synth.rng(13)
    check(ctx, synth.Q4_K, synth.make_weight(g, synth.Q4_K, 3, 1 << 18), synth.make_activations(g, 32, 1 << 18), 3, 1 << 18)


@pytest.mark.parametrize("qt", TYPES)
def test_batch_in_relaxed_order_and_on_another_stream(qt):
    """Products of different sizes share the buffer of prepared activations: declared independent, or on a stream of the caller's, they give the same bits."""
    g = synth.rng(14)
    ctx = skn.Context(0)
    shapes = [(512, 2048, 16), (300, 512, 31), (4096, 4096, 9), (40, 8192, 24)]
    ts = [skn.QuantTensor(ctx, (n, k), qt, synth.make_weight(g, qt, n, k)) for n, k, _ in shapes]
    xs = [torch.from_numpy(synth.make_activations(g, m, k)).cuda() for _, k, m in shapes]
    ys = [[torch.zeros(m, n, device="cuda") for n, _, m in shapes] for _ in range(3)]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    for way in range(3):
        ctx.set_relaxed_order(way == 1)
        ctx.set_stream(stream.cuda_stream if way == 2 else None)
        for _ in range(5):
            for t, x, y in zip(ts, xs, ys[way]):
                t.matmul_t_dev(x, x.shape[0], y)
        ctx.sync()
    for way in (1, 2):
        assert all(torch.equal(a, b) for a, b in zip(ys[0], ys[way]))
    for t in ts:
        t.close()
    ctx.close()


def test_batch_from_two_threads():
    """A context per thread: buffers and plans are the context's, what is kept for the device is the same for both."""
    def work(seed, out):
        g = synth.rng(seed)
        ctx = skn.Context(0)
        for i, qt in enumerate(TYPES * 3):
            n, k, m = 128 + 40 * i, 512 + 256 * (i % 5), 9 + 2 * i
            w, x = synth.make_weight(g, qt, n, k), synth.make_activations(g, m, k)
            t = skn.QuantTensor(ctx, (n, k), qt, w)
            out.append((qt, w, n, k, x, [t.matmul_t(x) for _ in range(5)]))
            t.close()
        ctx.close()

    got = [[], []]
    threads = [threading.Thread(target=work, args=(20 + i, got[i])) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out in got:
        assert len(out) == 3 * len(TYPES)
        for qt, w, n, k, x, ys in out:
            ref, absdot = oracle.matmul(qt, w, n, k, x)
            assert_close_dot(ys[0], ref, absdot, FP32_TOL, f"type {qt} {n}x{k}")
            assert all(np.array_equal(y, ys[0]) for y in ys)


@pytest.mark.parametrize("qt,batch", [(synth.Q4_0, 30), (synth.Q8_0, 24), (synth.Q4_K, 31), (synth.Q6_K, 25)])
def test_decoder_gate_and_up_of_many_sequences(ctx, qt, batch):
    """Gate and up interleaved, three and four chunks of rows, a tile for every SM and more super-blocks than a ring holds: a batch of sequences
    against some of them one by one; fp32 sums, 1e-5 a product."""
    d, f = 2560, 9472
    g = synth.rng(batch)
    cfg = LlamaConfig(n_layers=1, d_model=d, n_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=f, vocab=320, proj_type=qt)

    def weight(n, k):
        some = synth.make_weight(g, qt, 128, k).reshape(128, -1)
        return np.ascontiguousarray(some[np.arange(n) % 127]).reshape(-1)

    shapes = dict(wq=(256, d), wk=(128, d), wv=(128, d), wo=(d, 256), w_gate=(f, d), w_up=(f, d), w_down=(d, f))
    layer = {n: weight(*s) for n, s in shapes.items()}
    embed, head = (synth.make_weight(g, synth.Q6_K, 320, d) for _ in range(2))
    gain = np.ones(d, dtype=np.float32)
    tokens = g.integers(0, 320, size=(batch, 2)).astype(np.int32)

    def logits(rows):
        m = LlamaDecoder(ctx, cfg, batch=len(rows), max_tokens=1, max_ctx=8)
        m.set_layer(0, layer, gain, gain)
        m.set_head(embed, gain, head)
        out = np.stack([m.forward(np.ascontiguousarray(rows[:, i:i + 1]), want_logits=True)[1] for i in range(rows.shape[1])])
        m.close()
        return out.astype(np.float64)

    many = logits(tokens)
    assert np.isfinite(many).all()
    for b in (0, 17, batch - 1):
        one = logits(tokens[b:b + 1])[:, 0]
        assert np.linalg.norm(many[:, b] - one) <= 1e-3 * np.linalg.norm(one)


@pytest.mark.parametrize("batch", [9, 20, 40])
def test_decoder_batch_agrees_with_single_sequences(ctx, batch):
    """Q/K/V grouped, gate / up / SwiGLU interleaved, residuals and folded norms: a batch of sequences against the same
    sequences one by one (single-row kernels), both in fp32 sums: 1e-5 a product, a few dozen in a row."""
    g = synth.rng(batch)
    cfg = LlamaConfig(n_layers=2, d_model=512, n_heads=4, n_kv_heads=2, head_dim=128, ffn_dim=768, vocab=320)
    shapes = dict(wq=(512, 512), wk=(256, 512), wv=(256, 512), wo=(512, 512), w_gate=(768, 512), w_up=(768, 512), w_down=(512, 768))
    layers = [{n: synth.make_weight(g, synth.Q4_K, *s) for n, s in shapes.items()} for _ in range(2)]
    embed, head = (synth.make_weight(g, synth.Q6_K, 320, 512) for _ in range(2))
    gain = np.ones(512, dtype=np.float32)
    tokens = g.integers(0, 320, size=(batch, 3)).astype(np.int32)

    def logits(rows):
        m = LlamaDecoder(ctx, cfg, batch=len(rows), max_tokens=1, max_ctx=8)
        for i, l in enumerate(layers):
            m.set_layer(i, l, gain, gain)
        m.set_head(embed, gain, head)
        out = np.stack([m.forward(np.ascontiguousarray(rows[:, i:i + 1]), want_logits=True)[1] for i in range(rows.shape[1])])
        m.close()
        return out.astype(np.float64)

    many = logits(tokens)
    assert np.isfinite(many).all()
    for b in (0, 8, batch - 1):
        one = logits(tokens[b:b + 1])[:, 0]
        assert np.linalg.norm(many[:, b] - one) <= 1e-3 * np.linalg.norm(one)
