"""Single-row matvec with K over two CTAs of a cluster: rows per CTA and super-chunks of K on both sides of the rule, against the fp64 oracle."""
import numpy as np
import pytest
import torch

import skainet_b200 as skn
from conftest import FP32_TOL, assert_close_dot
from oracle import oracle
from skainet_b200 import synth

pytestmark = pytest.mark.gpu
KS = {synth.Q4_K: 16, synth.Q4_0: 16, synth.Q8_0: 8, synth.Q6_K: 8}
STAGE = {synth.Q4_K: (144, 32), synth.Q4_0: (144, 16), synth.Q8_0: (272, 32), synth.Q6_K: (210, 0)}       # bytes of a super-block, padding of a row


def is_split(sms, qt, N, K, M):
    """The launch rule of skn_matvec_mma.cu (mm_plan) for one or two activation rows, without norm, rotary epilogue or exchange."""
    ks, nb, grid = KS[qt], K // 256, min(sms, N)
    chunks, rows_per_cta = -(-nb // ks), -(-N // grid)
    half, tiles = (chunks + 1) // 2, (rows_per_cta + 15) // 16
    if chunks < 2 or grid % 2 or tiles > 2 + M or half * ks * 4 > nb * 3 or (qt == synth.Q6_K and tiles * chunks > 4):
        return False
    # digit planes, scales, group sums, outliers and partial sums of half of K, beside two stages of weights
    blocks, slots = half * ks, -(-half * ks // 4) * 4
    most = -(-N // (grid // 2))
    planes = -(-M * (4 * (blocks * 256 + 32) + 64) // 128) * 128 + M * slots * 4 + M * blocks * (16 if qt == synth.Q6_K else 8) * 4
    planes += M * slots * 20 + -(-M * slots // 16) * 16 + M * ((most + 1) // 2 + 1) * chunks * 8 * 4 + 64
    sb, pad = STAGE[qt]
    budget = 200 if (rows_per_cta + 2 + 15) // 16 * chunks >= 6 else 110
    return planes + 2 * (16 * (ks * sb + pad) + 16) <= budget * 1024


def check(ctx, qt, M, N, K, seed):
    g = synth.rng(seed)
    w, x = synth.make_weight(g, qt, N, K), synth.make_activations(g, M, K)
    x[0, K // 2 + 5] *= 3000.0                             # an outlier in the upper half
    b = g.standard_normal(N).astype(np.float32)
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    y, again = t.matmul_t(x, b), t.matmul_t(x, b)
    t.close()
    ref, absdot = oracle.matmul(qt, w, N, K, x)
    assert_close_dot(y, ref + b.astype(np.float64), absdot + np.abs(b.astype(np.float64)), FP32_TOL, f"type {qt} {N}x{K} M={M}")
    assert np.array_equal(y, again)


# rows as (multiple of the SMs, more), K in half super-chunks -> for which (type, M) the rows are split
ALL, NONE = lambda qt, M: True, lambda qt, M: False
EDGES = [((0, 2), 4, ALL), ((0, 147), 4, NONE), ((0, 300), 3, ALL), ((0, 300), 5, NONE), ((0, 300), 6, lambda qt, M: M == 1 or KS[qt] == 8),
         ((0, 300), 7, lambda qt, M: M == 1 or KS[qt] == 8), ((16, 0), 4, ALL), ((16, 1), 3, ALL), ((32, 0), 4, ALL), ((32, 1), 4, lambda qt, M: qt != synth.Q6_K),
         ((48, 0), 4, lambda qt, M: qt != synth.Q6_K), ((48, 1), 4, lambda qt, M: M == 2 and qt != synth.Q6_K),
         ((64, 0), 4, lambda qt, M: M == 2 and qt != synth.Q6_K), ((64, 1), 4, NONE)]


@pytest.mark.parametrize("qt", list(KS))
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("rows,halves,split", EDGES)
def test_both_sides_of_the_rule(ctx, qt, M, rows, halves, split):
    """One to five row tiles per CTA, two to four super-chunks of K: three and seven halves end with a short one, of three chunks (six halves) the
    second CTA has two; there two rows of x leave no room for Q4_K's and Q4_0's planes."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N, K = rows[0] * sms + rows[1], KS[qt] * 128 * halves
    assert is_split(sms, qt, N, K, M) == split(qt, M)
    check(ctx, qt, M, N, K, N + M + halves)


@pytest.mark.parametrize("qt", list(KS))
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,halves", [(2, 4), (3, 4), (147, 3), (149, 5), (300, 2), (16 * 148, 4), (16 * 148 + 1, 3), (48 * 148, 2), (48 * 148 + 1, 2), (64 * 148 + 1, 2)])
def test_split_rows(ctx, qt, M, N, halves):
    """halves: K in half super-chunks.  Most of these sizes are not split (one super-chunk, an odd number of CTAs, 5: more than three quarters of K in one half)."""
    K = KS[qt] * 128 * halves
    if N * K > 30_000_000 and qt != synth.Q4_K:
        pytest.skip("the largest sizes once")
    check(ctx, qt, M, N, K, N + M + halves)


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
