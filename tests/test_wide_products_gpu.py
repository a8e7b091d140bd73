"""bf16 products of layer-plan designs at widths of real models, where a step of more than 32 rows shares the K range of a tile among the
blocks of a cluster (on 148 SMs: 17 to 73 weight tiles, two to eight parts of unequal length): several output ranges, sums into the
stream, gated units, norms in the epilogue. Against the plain restatements; a part lost or added twice is off by a tenth and more."""
import numpy as np
import pytest

import fatilix_models
import revelix_models
import tedelix_models
from oracle import fatilix, revelix, tedelix
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


def _tedelix():
    M = tedelix_models
    return M, tedelix, M.config([M.delta(heads=32, dim=64, rank=64, ff=5000), M.attention(heads=16, kv_heads=4, dim=128, vdim=128, rot=64, window=150, ff=2500)], width=2056)


def _fatilix():
    M = fatilix_models
    return M, fatilix, M.config([M.shared_kv(heads=16, kv_heads=4, dim=128, mlp=M.dense(2500)),
                                 M.biased(heads=16, kv_heads=4, dim=128, vdim=128, bias_max=200, rows=20, mlp=M.dense(9216))], width=2056)


def _revelix():
    M = revelix_models
    a = M.left(heads=16, kv_heads=4, dim=128, vdim=128, rot=64, window=150)
    return M, revelix, M.config([M.retention(heads=16, dim=128, vdim=128, rot=64, ff=2500), M.parallel(a, M.right(heads=16, dim=64, vdim=64), ff=5000)], width=2056)


# The distance of bf16 engines from these models' restatements is 0.01 to 0.02 of the logits' spread at any number of rows: every
# sublayer rounds its operands to 2^-9, and the stream sums some ten of them.
@pytest.mark.parametrize("make", [_tedelix, _fatilix, _revelix], ids=lambda f: f.__name__[1:])
def test_k_shared_above_32_rows(make):
    M, oracle, cfg = make()
    W = M.weights(cfg, seed=9)
    ids = M.tokens(cfg, 300)
    want, _ = oracle.forward(cfg, W, ids)
    eng = ForwardEngine.from_config(cfg, W, dtype="bfloat16", max_ctx=512, max_batch=1, max_tokens=512)
    worst = {}
    for rows in (33, 64, 65, 100, 129, 250, 300):
        eng.reset_cache()
        got = eng.forward_mixed([(0, ids[:rows], list(range(rows)))])
        eng.reset_cache()
        again = eng.forward_mixed([(0, ids[:rows], list(range(rows)))])
        worst[rows] = float(M.error(got, want[:rows]).max())
        assert np.array_equal(got, again), rows  # parts are added in their order
    eng.close()
    assert max(worst.values()) < 0.04, worst
