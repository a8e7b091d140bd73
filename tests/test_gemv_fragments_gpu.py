"""The tile-row GEMV with digits in fragments: every number of 8-column n-tiles (1 to 6) and its last row, rows that start a new one,
columns for fewer and more pieces than eight and sixteen warps, tile rows fewer than SMs, as many, and more."""
import numpy as np
import pytest

from sapient_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,k", [(synth.Q4_K, 40, 256), (synth.Q4_K, 40, 2048), (synth.Q4_K, 2400, 4096), (synth.Q6_K, 40, 4096), (synth.Q4_K, 72, 2304), (synth.Q4_K, 40, 4352), (synth.Q4_K, 2384, 2304),
                                       (synth.Q6_K, 40, 2304), (synth.Q6_K, 24, 4608), (synth.Q8_0, 40, 1024), (synth.Q8_0, 40, 1152),
                                       (synth.Q8_0, 72, 2304), (synth.Q8_0, 40, 96), (synth.Q8_0, 2384, 1152)])
def test_every_row_count_of_a_pass(dtype, n, k):
    """Against the dequantised weights in float64: activations keep 2^-23 of a block's maximum, products are exact integers and the
    sums of k / 32 blocks are f32, 2^-24 each: 2e-6 of a row's norm."""
    be, _ = synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, k, synth.random_bit_blocks(dtype, n * k // be, seed=k))
    try:
        values = w.dequant().astype(np.float64).T
        x = np.random.default_rng(k).standard_normal((17, k)).astype(np.float32)
        x[3, : k // 2] *= 1e-3  # (blocks of unequal size beside one another)
        ops.set_large_m_gemm(0)  # 17 rows: a pass of sixteen and one of one
        for m in range(1, 18):
            got, want = w.matmul_nt(x[:m]).astype(np.float64), x[:m].astype(np.float64) @ values
            assert np.all(np.linalg.norm(got - want, axis=1) < 2e-6 * np.linalg.norm(want, axis=1)), m
        # one row may make its digits itself, two never: the same digits, products and sums
        assert np.array_equal(w.matmul_nt(x[3:4]), w.matmul_nt(x[3:5])[:1])
    finally:
        ops.set_large_m_gemm(2)
        w.free()
