"""Batches of 9 to 63 activation rows (tcgen05 with exact fp16 integers) against the fp64 oracle, at the edges of chunks, tiles,
launches and parts of K; the tolerance of the single-row kernels."""
import numpy as np
import pytest
import torch

import skainet_b200 as skn
from conftest import FP32_TOL, assert_close_dot
from oracle import oracle
from skainet_b200 import synth
from skainet_b200.llama import LlamaConfig, LlamaDecoder

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
def test_batch_outliers_zeros_and_scales(ctx, qt):
    """Rows of zeros, of one element, of outliers up to 1e6 in the block, of very different sizes; the towering elements meet zero weights."""
    g = synth.rng(5)
    M, N, K = 12, 48, 1024
    w = synth.make_weight(g, qt, N, K)
    x = synth.make_activations(g, M, K)
    x[0] = 0
    x[1] = 0
    x[1, 700] = 3.5
    for m, size in ((2, 1e3), (3, 1e4), (4, 1e6)):
        x[m, 5::256] *= size
        x[m, 130::256] *= -size
    x[5] *= 1e-20
    x[6] *= 1e20
    check(ctx, qt, w, x, N, K)


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
