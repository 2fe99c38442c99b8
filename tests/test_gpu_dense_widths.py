"""Tensor-core products of more than 128 rows, whose token tiles have any multiple of 16 between 128 and 256: sizes that are no multiple of a
tile, and the decoders' epilogues against the same model in steps of one narrow tile."""
import numpy as np
import pytest

import skainet_b200 as skn
from skainet_b200.lugasun import LugasunConfig
from skainet_b200.tensor import from_bf16_bits, to_bf16_bits
from skainet_b200.tutezen import TutezenConfig
from tests import lugasun_models as lm, tutezen_models as tm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(129, 18500, 712), (300, 4226, 1100), (515, 7170, 1288), (2048, 2050, 520), (257, 9473, 1032)])
def test_ragged_products(ctx, M, N, K):
    g = np.random.default_rng(M + N)
    w = to_bf16_bits(g.standard_normal((N, K)).astype(np.float32))
    x = g.standard_normal((M, K)).astype(np.float32)
    t = skn.DenseTensor(ctx, w)
    y = t.matmul_t(x)
    t.close()
    exact = from_bf16_bits(to_bf16_bits(x)).astype(np.float64) @ from_bf16_bits(w).astype(np.float64).T      # exact in the bf16-rounded rows
    assert np.linalg.norm(y - exact) < 2e-6 * np.linalg.norm(exact)
    assert np.abs(y - exact).max() < 1e-5 * np.abs(exact).max()


LUGASUN = lm.config([lm.layer(heads=8, kv_heads=2, dim=64, vdim=64, chunk=96, rheads=4, rdim=64, rvdim=64, ff=4098)], width=1030, side=0)
TUTEZEN = tm.config([tm.ssm(heads=16, vdim=64, state=64, groups=1, norm_groups=1, mlp=tm.dense(4104)),
                     tm.latent(heads=16, dim=128, rot_dim=64, vdim=64, q_rank=1024, kv_rank=64, window=120, mlp=tm.moe(experts=4, top=2, ff=64, shared=2056))],
                    width=1032)


@pytest.mark.parametrize("models,cfg,config,decoder", [(lm, LUGASUN, LugasunConfig, skn.LugasunDecoder), (tm, TUTEZEN, TutezenConfig, skn.TutezenDecoder)])
def test_prompt_at_once_and_in_short_steps(ctx, models, cfg, config, decoder):
    bits, T = models.weights(cfg, 5), 417
    tokens = np.random.default_rng(2).integers(0, cfg["vocab"], T).astype(np.int32)
    out = []
    for most in (T, 96):
        m = decoder(ctx, config.from_dict(cfg), max_seqs=1, max_tokens=most, max_ctx=T + 1)
        m.load(models.getter(bits))
        out.append(m.forward(tokens, want=range(T))[1])
        m.close()
    assert np.quantile(models.errors(out[0], out[1].astype(np.float64)), 0.98) < models.TOL["bfloat16"]
