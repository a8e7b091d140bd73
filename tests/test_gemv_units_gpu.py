"""Edges of the tile-row GEMV's prefetch (gemv_imma.cu): Q8_0 in units of 128 columns, three deep (one row or two) or two deep, over
eight warps; Q6_K tiles two deep; and decode steps of 11 to 16 rows, whose digits one launch makes for two passes."""
import numpy as np
import pytest

from helpers import tiny_model
from sapient_b200 import ops, synth
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu

# fewer units than warps, a warp's first, second and third, one more than all in flight (25 units), tiles of eight and of four blocks
Q8_K = [128, 256, 896, 1152, 2048, 2304, 3072, 3200, 4352, 6272]
# Q6_K: 8 warps x 1, 2, 3 tiles and one more
Q6_K_COLUMNS = [256, 2048, 2304, 4096, 4352, 6400]


@pytest.mark.parametrize("dtype,k", [(synth.Q8_0, k) for k in Q8_K] + [(synth.Q6_K, k) for k in Q6_K_COLUMNS])
@pytest.mark.parametrize("m", [1, 3, 6])
def test_prefetched_tiles_at_their_edges(dtype, k, m):
    """Against the dequantised weights in float64: activations keep 2^-23 of a block's maximum, products are exact integers and the
    sums of k / 32 blocks are f32, 2^-24 each: 2e-6 of a row's norm."""
    n, (be, _) = 40, synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, k, synth.random_bit_blocks(dtype, n * k // be, seed=k + m))
    try:
        x = np.random.default_rng(k + m).standard_normal((m, k)).astype(np.float32)
        got = w.matmul_nt(x).astype(np.float64)
        want = x.astype(np.float64) @ w.dequant().astype(np.float64).T
    finally:
        w.free()
    assert np.all(np.linalg.norm(got - want, axis=1) < 2e-6 * np.linalg.norm(want, axis=1))


@pytest.mark.parametrize("name", ["tiny_llama_wide", "tiny_qwen", "tiny_phi2_wide"])
@pytest.mark.parametrize("b", [11, 13, 16])
def test_steps_of_two_passes_equal_each_sequence_alone(name, b):
    """A row's digits and sums do not depend on the rows beside it; the attention kernel may (f32 sums in another order), and with
    it the fp16 rounding of a cached value here and there: 2e-4 of logits near 1."""
    cfg, W = tiny_model(name, max_ctx=64)
    rng = np.random.default_rng(b)
    prompts = [rng.integers(0, cfg["vocab"], 3 + s).astype(np.uint32) for s in range(b)]
    ids = rng.integers(0, cfg["vocab"], b).astype(np.uint32)
    both = ForwardEngine.from_weights(cfg, W, max_batch=b, max_tokens=64)
    alone = ForwardEngine.from_weights(cfg, W, max_tokens=64)
    for e in (both, alone):
        e.set_kv_rounding(False)
    for s, p in enumerate(prompts):
        both.forward_slot(s, p)
    got, _ = both.decode_batch(ids, list(range(b)))
    for s, p in enumerate(prompts):
        alone.reset_cache()
        alone.forward_logits(p)
        assert np.abs(got[s] - alone.forward_logits(ids[s:s + 1])).max() < 2e-4, s
    both.close()
    alone.close()
