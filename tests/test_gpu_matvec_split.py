"""Single-row matvec with K over two CTAs of a cluster: rows per CTA and super-chunks of K at the edges of the rule, against the fp64 oracle."""
import numpy as np
import pytest
import torch

import skainet_b200 as skn
from conftest import FP32_TOL, assert_close_dot
from oracle import oracle
from skainet_b200 import synth

pytestmark = pytest.mark.gpu
KS = {synth.Q4_K: 16, synth.Q4_0: 16, synth.Q8_0: 8, synth.Q6_K: 8}


@pytest.mark.parametrize("qt", list(KS))
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,halves", [(2, 4), (3, 4), (147, 3), (149, 5), (300, 2), (16 * 148, 4), (16 * 148 + 1, 3), (48 * 148, 2), (48 * 148 + 1, 2), (64 * 148 + 1, 2)])
def test_split_rows(ctx, qt, M, N, halves):
    """halves: K in half super-chunks (3: two chunks, the upper one short and within the rule; 5: three)."""
    K = KS[qt] * 128 * halves
    if N * K > 30_000_000 and qt != synth.Q4_K:
        pytest.skip("the largest sizes once")
    g = synth.rng(N + M + halves)
    w, x = synth.make_weight(g, qt, N, K), synth.make_activations(g, M, K)
    x[0, K // 2 + 5] *= 3000.0                             # an outlier in the upper half
    b = g.standard_normal(N).astype(np.float32)
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y, again = t.matmul_t(x, b), t.matmul_t(x, b)
    t.close()
    ref, absdot = oracle.matmul(qt, w, N, K, x)
    assert_close_dot(y, ref + b.astype(np.float64), absdot + np.abs(b.astype(np.float64)), FP32_TOL, f"type {qt} {N}x{K} M={M}")
    assert np.array_equal(y, again)


def test_split_keeps_the_bits_of_a_row(ctx):
    """A row's sum does not depend on how K was shared: rows of a weight that is split against the same rows inside one that is not (as many
    rows per CTA, an odd number of them)."""
    g = synth.rng(8)
    K, N = 8192, 148 - 1                                   # one row a CTA either way: 147 CTAs are no pairs
    w = synth.make_weight(g, synth.Q4_K, N + 1, K)
    x = torch.from_numpy(synth.make_activations(g, 1, K)[0].copy()).cuda()
    out = []
    for n in (N, N + 1):
        t = skn.QuantTensor(ctx, (n, K), synth.Q4_K, w.reshape(-1)[: n * (K // 256) * 144])
        y = torch.empty(n, device="cuda")
        t.matmul_t_dev(x, 1, y)
        ctx.sync()
        out.append(y.cpu().numpy()[:N])
        t.close()
    assert np.array_equal(out[0], out[1])
