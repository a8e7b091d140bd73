"""One and two rows on matrices of 1024 tile rows and more, whose warps hold one tile each: fewer tiles than warps, as many, one more, several."""
import numpy as np
import pytest

from sapient_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("n,k", [(16384, 256), (16385, 768), (16370, 2048), (16384, 2304), (16391, 4352)])
def test_deep_grids(dtype, n, k):
    """Against the dequantised weights in float64, on rows of the first, some middle and the last tiles: activations keep 2^-23 of a block's
    maximum, products are exact integers, sums f32: 2e-6 of a row's norm."""
    be, _ = synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, k, synth.random_bit_blocks(dtype, n * k // be, seed=k))
    rows = np.r_[0:40, 8000:8040, n - 40:n]
    values = w.dequant()[rows].astype(np.float64).T
    x = np.random.default_rng(n).standard_normal((2, k)).astype(np.float32)
    for m in (1, 2):
        got, want = w.matmul_nt(x[:m]).astype(np.float64)[:, rows], x[:m].astype(np.float64) @ values
        assert np.all(np.linalg.norm(got - want, axis=1) < 2e-6 * np.linalg.norm(want, axis=1)), m
    w.free()
