"""Retention in chunks on the tensor cores at the edges of its shared memory: keys in several pieces of 128 columns, values in several blocks of
128, the widest that fit (the last block of outputs lies over the operands) and the first that do not (which run in fp32 on the CUDA cores)."""
import numpy as np
import pytest

from skainet_b200.mixers import RecurrentState
from tests.test_gpu_lugasun import rel, retention_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,D,V", [(2, 128, 129), (1, 129, 128), (1, 256, 256), (1, 257, 255), (1, 192, 384), (1, 256, 384), (1, 6, 2), (1, 128, 512), (2, 97, 385), (1, 193, 260),
                                   (1, 352, 256), (1, 257, 129), (1, 192, 512), (1, 193, 512), (1, 353, 200)])
def test_retention_widths(ctx, H, D, V):
    g = np.random.default_rng(D * 3 + V)
    T, decay = 131, [0.998, 0.9][:H]
    q, k, v, gate = (g.standard_normal((T, H, d)).astype(np.float32) for d in (D, D, V, V))
    want, S = retention_reference(q, k, v, gate, decay, None, 1e-5)
    st = RecurrentState(ctx, 1, H, D, V)
    out = np.concatenate([st.retain(*(a[None, i:j] for a in (q, k, v, gate)), [i], decay)[0] for i, j in ((0, 67), (67, T))])
    # sums of at most 64 + D products in fp32, the errors walking at random (2**-24 * sqrt(450) = 1.3e-6), and the norm of rows that can be ten
    # times smaller than the largest
    assert rel(out, want) < 2e-5
    assert rel(st.read(0), S) < 2e-5
    st.close()


@pytest.mark.parametrize("D,V,tc", [(128, 512, True), (97, 385, True), (256, 384, True), (193, 257, True), (352, 256, True), (257, 129, True), (192, 512, True), (193, 512, False), (353, 200, False)])
def test_which_widths_run_on_the_tensor_cores(ctx, D, V, tc):
    """By their bits: sums of split operands are not those of the fp32 form, which `exact` asks for."""
    g = np.random.default_rng(D + V)
    T, decay = 64, [0.99]
    q, k, v, gate = (g.standard_normal((1, T, 1, d)).astype(np.float32) for d in (D, D, V, V))
    out = []
    for exact in (False, True):
        st = RecurrentState(ctx, 1, 1, D, V)
        out.append(st.retain(q, k, v, gate, [0], decay, exact=exact)[0])
        st.close()
    assert np.array_equal(out[0], out[1]) != tc
