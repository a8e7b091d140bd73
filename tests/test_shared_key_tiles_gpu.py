"""Prompts whose key tiles two blocks of a cluster share: row tiles with one, two and more key tiles, so that the second block has none, one
and as many as the first or one less; the last rows short; portions that start inside and past a tile."""
import numpy as np
import pytest

from helpers import oracle_engine, tiny_model
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_phi2_wide", "tiny_llama"])
@pytest.mark.parametrize("first,n", [(0, 129), (0, 193), (0, 257), (63, 130), (64, 66), (128, 150), (190, 70)])
def test_portions(oracle, name, first, n):
    """Against the oracle with a continuous cache: the bar between kernels, 3e-3 of the logits (f32 sums in another order, and an fp16
    rounding of a cached value here and there)."""
    cfg, W = tiny_model(name, max_ctx=320)
    ids = np.random.default_rng(first + n).integers(0, cfg["vocab"], first + n).astype(np.uint32)
    eng, ref = ForwardEngine.from_weights(cfg, W, max_tokens=320, fast_large_m=True), oracle_engine(oracle, cfg, W, kv_mode=1)
    exact = ForwardEngine.from_weights(cfg, W, max_tokens=320)
    for e, bar in ((eng, 1e-2), (exact, 3e-3)):  # (products of fp16-rounded operands, and of both parts)
        e.set_graphs(False)
        e.set_kv_rounding(False)
        if first:
            e.forward_logits(ids[:first], True)
        got = e.forward_all_logits_cached(ids[first:])
        want = ref.forward_all_logits(ids)[first:]
        assert np.abs(got - want).max() < bar, np.abs(got - want).max()
        again = e.truncate_cache(first) is not None and e.forward_all_logits_cached(ids[first:])
        assert np.array_equal(got, again)
        e.close()
