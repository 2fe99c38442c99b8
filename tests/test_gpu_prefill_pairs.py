"""Prefill matmul at the edges of its plan: token blocks, accumulators, feature tiles, parts of K, short last super-blocks.

The reference rounds weights and activations to bf16 as the kernel does and multiplies them in fp64, so what is left is the
fp32 accumulation: one rounding (at most an ulp, 2^-23, as the tensor cores truncate) per K step of 16, a few more inside a
step and for the parts of K, each of a partial sum that sum |w x| bounds."""
import numpy as np
import pytest
import torch

import skainet_b200 as skn
from skainet_b200 import synth

pytestmark = pytest.mark.gpu


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(torch.bfloat16).double().numpy()


@pytest.mark.parametrize("qt", [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("M,N,K", [(64, 8, 64), (65, 264, 320), (256, 256, 256), (257, 520, 1024), (288, 128, 1280), (512, 776, 768),
                                   (513, 136, 2304), (1030, 40, 512)])
def test_matmul_at_plan_edges(ctx, qt, M, N, K):
    e, _ = synth.GEOMETRY[qt]
    K = -(-K // e) * e
    g = synth.rng(M + N + K)
    t = skn.QuantTensor(ctx, (N, K), qt, synth.make_weight(g, qt, N, K))
    x = synth.make_activations(g, M, K)
    b = g.standard_normal(N).astype(np.float32) if M % 2 else None
    y = t.matmul_t(x, b)
    w, x = bf16(t.dequantize()), bf16(x)
    t.close()
    ref, absdot = x @ w.T, np.abs(x) @ np.abs(w).T
    if b is not None:
        ref, absdot = ref + b.astype(np.float64), absdot + np.abs(b)
    assert np.all(np.abs(y - ref) <= (K / 16 + 16) * 2.0 ** -23 * absdot)


@pytest.mark.parametrize("gate,down,M,F,K", [(synth.Q4_K, synth.Q6_K, 96, 72, 512), (synth.Q8_0, synth.Q4_0, 300, 320, 256), (synth.Q4_0, synth.Q8_0, 513, 128, 1088)])
def test_ffn_at_plan_edges(ctx, gate, down, M, F, K):
    if F % synth.GEOMETRY[down][0]:
        F = -(-F // 256) * 256
    g = synth.rng(F + K)
    ts = [skn.QuantTensor(ctx, s, q, synth.make_weight(g, q, *s)) for q, s in ((gate, (F, K)), (gate, (F, K)), (down, (40, F)))]
    x = synth.make_activations(g, M, K)
    y = skn.ffn_swiglu(ctx, *ts, x)
    wg, wu, wd = (bf16(t.dequantize()) for t in ts)
    for t in ts:
        t.close()
    a = bf16(x) @ wg.T
    h = bf16(a / (1 + np.exp(-np.clip(a, -700, 700))) * (bf16(x) @ wu.T))
    # the intermediate may round to the neighbouring bf16 (2^-8 of it): fp32 sums against fp64 sums
    assert np.all(np.abs(y - h @ wd.T) <= 2.0 ** -8 * (np.abs(h) @ np.abs(wd).T))
