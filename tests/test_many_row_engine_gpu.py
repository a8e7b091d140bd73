"""Engines whose steps have at most 16 rows, on the many-row GEMV by choice."""
import numpy as np
import pytest

from helpers import tiny_model
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_llama", "tiny_qwen", "tiny_llama_wide"])
@pytest.mark.parametrize("rows", [11, 13, 16])
def test_small_engines_share_the_columns_too(name, rows):
    """The same bits as an engine for longer steps, which has the scratch for columns shared by blocks: without it the sums have another
    order. Against passes of the tile-row kernel: the same integer products, f32 sums in another order, the bar of tests that compare kernels."""
    cfg, W = tiny_model(name)
    ids = np.random.default_rng(rows).integers(0, cfg["vocab"], rows).astype(np.uint32)
    got = []
    for max_tokens, many in ((16, True), (64, True), (16, False)):
        eng = ForwardEngine.from_weights(cfg, W, max_tokens=max_tokens)
        eng.set_kv_rounding(False)
        eng.set_many_row_gemv(many)
        got.append(eng.forward_all_logits(ids))
        eng.close()
    assert np.array_equal(got[0], got[1])
    assert np.abs(got[0] - got[2]).max() < 2e-3
