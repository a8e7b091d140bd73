"""bf16 products whose rows are dealt out evenly over tiles that are no power of two high and share their K range: where the model of the
time promises a tenth (on 148 SMs: 1024 x 4096 as tiles of 80 rows in eight parts, gated 1024 x 3072 as tiles of 48 and 80). Against the
plain restatements; a row or a part lost or taken twice is off by a tenth and more."""
import numpy as np
import pytest

import fatilix_models
import tedelix_models
from oracle import fatilix, tedelix
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


def _plain():
    M = tedelix_models
    return M, tedelix, M.config([M.attention(heads=8, kv_heads=2, dim=64, vdim=64, rot=32, window=150, ff=4096)], width=1024), (257, 301, 400)


def _gated():
    M = fatilix_models
    return M, fatilix, M.config([M.shared_kv(heads=8, kv_heads=2, dim=64, mlp=M.dense(1024))], width=3072), (129, 300, 389)


@pytest.mark.parametrize("make", [_plain, _gated], ids=lambda f: f.__name__[1:])
def test_rows(make):
    """The bar of the other tests of these models' products: 0.01 to 0.02 of the logits' spread is what bf16 operands move."""
    M, oracle, cfg, counts = make()
    W = M.weights(cfg, seed=5)
    ids = M.tokens(cfg, max(counts))
    want, _ = oracle.forward(cfg, W, ids)
    eng = ForwardEngine.from_config(cfg, W, dtype="bfloat16", max_ctx=512, max_batch=1, max_tokens=512)
    for rows in counts:
        got = []
        for _ in range(2):
            eng.reset_cache()
            got.append(eng.forward_mixed([(0, ids[:rows], list(range(rows)))]))
        assert np.array_equal(*got), rows  # parts are added in their order
        assert float(M.error(got[0], want[:rows]).max()) < 0.04, rows
    eng.close()
