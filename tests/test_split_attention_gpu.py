"""Attention with a token per block: key counts at the edges of a warp's round, of a split and of a page, for every width of the lanes,
and steps whose first keys are requested while the step's own are still being appended."""
import numpy as np
import pytest

from helpers import f16_round, rel_l2, tiny_model
from sapient_b200 import ops
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [32, 64, 80, 128, 160, 256])
@pytest.mark.parametrize("sq,sk", [(1, 1), (1, 7), (1, 8), (1, 31), (1, 33), (2, 128), (1, 129), (3, 257), (1, 641), (20, 37)])
def test_key_counts(oracle, hd, sq, sk):
    rng = np.random.default_rng(hd + sk)
    q = rng.standard_normal((4, sq, hd)).astype(np.float32)
    k, v = (f16_round(rng.standard_normal((4, sk, hd))) for _ in range(2))  # (unshared heads: never the grouped kernel)
    # f32 sums of up to 641 terms against f32 sums in another order
    assert rel_l2(ops.gqa_attention(q, k, v), oracle.attention(q, k, v, oracle.causal_mask(sq, sk))) < 1e-5


@pytest.mark.parametrize("hd,H,Hkv", [(64, 8, 2), (128, 16, 8), (80, 6, 3)])
@pytest.mark.parametrize("sq,sk", [(16, 257), (16, 400), (40, 161), (111, 130), (160, 170)])
def test_grouped_kernel_with_few_and_many_blocks(oracle, hd, H, Hkv, sq, sk):
    """(Query rows, cached heads) below and above two blocks per SM: four and three warps a block, which share the pages out differently."""
    rng = np.random.default_rng(hd + sk)
    q = rng.standard_normal((H, sq, hd)).astype(np.float32)
    k, v = (f16_round(rng.standard_normal((Hkv, sk, hd))) for _ in range(2))
    # queries and weights in two fp16 parts (2^-22), f32 sums
    assert rel_l2(ops.gqa_attention(q, k, v), oracle.attention(q, k, v, oracle.causal_mask(sq, sk))) < 1e-5


@pytest.mark.parametrize("name", ["tiny_llama", "tiny_phi2"])
def test_rows_of_a_step_see_each_other(name):
    """Five rows at once and one after the other, from lengths around pages and rounds: the rows of a step are keys of the later ones."""
    cfg, W = tiny_model(name, max_ctx=256)
    rng = np.random.default_rng(3)
    many, single = (ForwardEngine.from_weights(cfg, W) for _ in range(2))
    for e in (many, single):
        e.set_kv_rounding(False)  # a continuous cache: this test is about the kernels
    for n in (1, 3, 11, 12, 15, 16, 17, 64, 65, 127, 130):
        ids, more = rng.integers(0, cfg["vocab"], n).astype(np.uint32), rng.integers(0, cfg["vocab"], 5).astype(np.uint32)
        for e in (many, single):
            e.reset_cache()
            e.forward_logits(ids, True)
        rows = many.forward_all_logits_cached(more)
        # (other splits of the keys, other passes of the products: the bar of the other tests that compare kernels)
        for i, t in enumerate(more):
            assert np.abs(rows[i] - single.forward_logits([t], True)).max() < 2e-3, (n, i)
    many.close()
    single.close()
