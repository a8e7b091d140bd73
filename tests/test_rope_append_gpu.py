"""Rotation and cache append of many tokens: whole and partial rotation, head sizes with and without 32-blocks, with the reference's cache
rounding and without, token counts around the switch of kernels, on the same prompts as the oracle."""
import numpy as np
import pytest

from helpers import oracle_engine, tiny_model
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_llama", "tiny_qwen", "tiny_phi2", "tiny_phi2_wide", "tiny_llama_wide"])
@pytest.mark.parametrize("n", [31, 32, 33, 70])
@pytest.mark.parametrize("rounded", [False, True])
def test_prompts_then_decode(oracle, name, n, rounded):
    """A value near the edge of a step of the rounded cache may take the other step (0.8 % of its block's largest): the bar of the
    reference's own configuration, 2e-2 of the logits; a continuous cache keeps the one between kernels, 3e-3."""
    cfg, W = tiny_model(name, max_ctx=128)
    ids = np.random.default_rng(n).integers(0, cfg["vocab"], n + 2).astype(np.uint32)
    eng = ForwardEngine.from_weights(cfg, W, max_tokens=128)
    eng.set_kv_rounding(rounded)
    ref = oracle_engine(oracle, cfg, W, kv_mode=0 if rounded else 1)
    bar = 2e-2 if rounded else 3e-3
    assert np.abs(eng.forward_logits(ids[:n], True) - ref.forward_logits(ids[:n], True)).max() < bar
    for t in ids[n:]:
        assert np.abs(eng.forward_logits([t], True) - ref.forward_logits([t], True)).max() < bar
    eng.close()
