"""Blocking calls on host buffers of any kind: results in one piece and in several, from and to pageable and page-locked memory."""

import numpy as np
import pytest
import torch

import skainet_b200 as skn
from conftest import FP32_TOL, assert_close_dot
from oracle import oracle
from skainet_b200 import synth
from skainet_b200.lugasun import LugasunConfig
from tests import lugasun_models as lm

pytestmark = pytest.mark.gpu


def pinned(a):
    return torch.from_numpy(a.copy()).pin_memory().numpy()


@pytest.mark.parametrize("kind", ["pageable", "pinned", "pinned and odd"])
@pytest.mark.parametrize("qt,M,N,K", [(synth.Q4_K, 1, 257, 512), (synth.Q8_0, 2, 4096, 96), (synth.Q4_K, 5, 7001, 256), (synth.Q4_0, 3, 12290, 512), (synth.Q4_K, 70, 16401, 256)])
def test_matmul_from_any_host_memory(ctx, qt, M, N, K, kind):
    """Results of 1 KB to 4.6 MB: beside the status word, staged through page-locked memory, and in pieces; a bias of any length."""
    g = synth.rng(M + N)
    w, x, bias = synth.make_weight(g, qt, N, K), synth.make_activations(g, M, K), g.standard_normal(N + 1).astype(np.float32)
    if kind == "pinned and odd":                           # a bias that starts 4 bytes off a 16-byte boundary
        x, b = pinned(x), pinned(bias)[1:]
    else:
        b = bias[1:]
        if kind == "pinned":
            x, b = pinned(x), pinned(b)
    t = skn.QuantTensor(ctx, (N, K), qt, w)
    ref, absdot = oracle.matmul(qt, w, N, K, x)
    for add in (None, b):
        y = t.matmul_t(x, add)
        r, a = (ref, absdot) if add is None else (ref + add.astype(np.float64), absdot + np.abs(add.astype(np.float64)))
        if M < 64:
            assert_close_dot(y, r, a, FP32_TOL, f"{kind} {N}x{K} M={M}")
        else:                                              # bf16 activations: 2**-9 of every term at most
            assert (np.abs(y - r) <= 2.0 ** -8 * a).all()
    t.close()


def test_rows_that_are_the_last_of_their_sequences(ctx):
    """The logits of the last rows come from the step itself, those of other rows from a product of their own: the same either way."""
    cfg = lm.config([lm.layer(heads=4, kv_heads=2, dim=64, vdim=64, chunk=96, rheads=2, rdim=64, rvdim=64, ff=512)], width=512, side=0)
    bits = lm.weights(cfg, 3)
    tokens = np.random.default_rng(4).integers(0, cfg["vocab"], (3, 7)).astype(np.int32)
    got = []
    for want in ([6, 13, 20], [20, 13, 6], range(21)):
        m = skn.LugasunDecoder(ctx, LugasunConfig.from_dict(cfg), max_seqs=3, max_tokens=21, max_ctx=8)
        m.load(lm.getter(bits))
        got.append(m.forward(tokens, want=want))
        m.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][0], got[2][0])
    assert np.array_equal(got[0][1].argmax(1), got[0][0])
    scale = np.abs(got[2][1]).max()
    assert np.abs(got[0][1] - got[1][1][::-1]).max() < 1e-5 * scale      # (fp32 sums of the same bf16 rows, in another order at most)
    assert np.abs(got[0][1] - got[2][1][[6, 13, 20]]).max() < 1e-5 * scale
