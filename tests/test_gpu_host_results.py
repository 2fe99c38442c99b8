"""Blocking calls on host buffers of any kind: results in one piece and in several, from and to pageable and page-locked memory."""

import ctypes

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


def managed(n):
    """n floats of managed memory and what frees them."""
    rt, p = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p()
    assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(4 * n), 1) == 0
    return np.ctypeslib.as_array((ctypes.c_float * n).from_address(p.value)), lambda: rt.cudaFree(p)


@pytest.mark.parametrize("role", ["x", "bias"])
@pytest.mark.parametrize("kind", ["pinned", "pinned, read off 16 bytes", "pinned, written off 16 bytes", "managed", "pageable"])
def test_blocking_call_on_a_result_that_is_still_to_come(ctx, role, kind):
    """A result of skn_matmul_async is the next, blocking call's x or bias while the GPU is milliseconds behind: stream order, whatever memory
    it lies in.  As a bias of 513 and four rows of x it does not come in fours either."""
    g = synth.rng(5)
    N1, K, N2, K2, M = 520, 512, 513, 512, 4
    w1, w2, w = synth.make_weight(g, synth.Q4_K, N1, K), synth.make_weight(g, synth.Q4_K, N2, K2), synth.make_weight(g, synth.Q4_K, 4096, 4096)
    t1, t2, t = (skn.QuantTensor(ctx, s, synth.Q4_K, b) for s, b in (((N1, K), w1), ((N2, K2), w2), ((4096, 4096), w)))
    x, x2, bias = synth.make_activations(g, 1, K)[0], synth.make_activations(g, M, K2), g.standard_normal(N2).astype(np.float32)
    busy = [torch.zeros(2048, 4096, device="cuda") for _ in range(2)]
    free = None
    if kind == "managed":
        buf, free = managed(M * N1 + 8)
    else:
        buf = np.zeros(M * N1 + 8, dtype=np.float32) if kind == "pageable" else torch.zeros(M * N1 + 8).pin_memory().numpy()
    out = buf[1:1 + M * N1] if kind.endswith("written off 16 bytes") else buf[:M * N1]
    at = 1 if kind.endswith("read off 16 bytes") else 0
    first = np.concatenate([t1.matmul_t(np.roll(x, i)) for i in range(M)])             # blocking, on memory of its own
    part = lambda a: a[at:at + M * K2].reshape(M, K2) if role == "x" else a[at:at + N2]
    call = lambda a: t2.matmul_t(part(a), bias) if role == "x" else t2.matmul_t(x2, part(a))
    want = call(first.copy())
    rows = [np.roll(x, i) if kind == "pageable" else pinned(np.roll(x, i)) for i in range(M)]
    for _ in range(3):
        buf[:] = 0
        ctx.sync()
        for _ in range(20):
            t.matmul_t_dev(busy[0], 2048, busy[1])
        for i in range(M):
            t1.matmul_t_async(rows[i], out[i * N1:(i + 1) * N1])
        got = call(out)
        assert np.array_equal(got, want)
        assert np.array_equal(out, first)
    ctx.sync()
    for q in (t1, t2, t):
        q.close()
    if free:
        free()


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
