"""bf16 products of more than 32 rows in tiles of any multiple of 16 rows: counts that leave one, two and more tiles with a short last
one, heights whose accumulators are no power of two of tensor-memory columns. Against the plain restatements; a row lost or
stored twice is off by all of it."""
import pytest

from sapient_b200.engine import ForwardEngine
from test_wide_products_gpu import _fatilix, _revelix, _tedelix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [_tedelix, _fatilix, _revelix], ids=lambda f: f.__name__[1:])
def test_heights(make):
    """The bar of the other test of these models' products: 0.01 to 0.02 of the logits' spread is what bf16 operands move."""
    M, oracle, cfg = make()
    W = M.weights(cfg, seed=4)
    ids = M.tokens(cfg, 400)
    want, _ = oracle.forward(cfg, W, ids)
    eng = ForwardEngine.from_config(cfg, W, dtype="bfloat16", max_ctx=512, max_batch=1, max_tokens=512)
    worst = {}
    for rows in (47, 80, 81, 113, 145, 161, 177, 209, 241, 257, 400):
        eng.reset_cache()
        worst[rows] = float(M.error(eng.forward_mixed([(0, ids[:rows], list(range(rows)))]), want[:rows]).max())
    eng.close()
    assert max(worst.values()) < 0.04, worst
