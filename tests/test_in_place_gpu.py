"""Matmuls whose outputs take the place of their inputs."""
import numpy as np
import pytest

from sapient_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n", [(synth.Q4_K, 256), (synth.Q4_K, 1536), (synth.Q4_K, 4096), (synth.Q6_K, 256), (synth.Q6_K, 4096), (synth.Q8_0, 96),
                                     (synth.Q8_0, 1152), (synth.Q4_K, 4352)])
@pytest.mark.parametrize("rows", [1, 2, 5, 16, 17, 40])
def test_square_matmul(dtype, n, rows):
    """The same sums in the same order as into a buffer of its own; up to 16 rows also where outputs start inside
    the inputs or inputs inside the outputs. One row of these formats may make its digits in the product's own launch, but not then: blocks that are done would overwrite what others read."""
    import torch

    be, _ = synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, n, synth.random_bit_blocks(dtype, n * n // be, seed=n))
    x = torch.from_numpy(np.random.default_rng(rows).standard_normal((rows, n)).astype(np.float32)).cuda()
    y = torch.empty_like(x)
    stream = torch.cuda.current_stream().cuda_stream

    def launches(src, dst):
        before = ops.launch_count()
        w.matmul_nt_dev(src.data_ptr(), rows, dst.data_ptr(), stream)
        return ops.launch_count() - before

    launches(x, y)
    apart = launches(x, y)
    last = rows * n - 32
    for at, to in ((0, 0), (0, 32), (32, 0), (0, last), (last, 0)) if rows <= 16 else ((0, 0),):
        both = torch.zeros(2 * rows * n, device="cuda")
        src, dst = both[at:at + rows * n], both[to:to + rows * n]
        src.copy_(x.reshape(-1))
        n_launches = launches(src, dst)
        assert torch.equal(dst.reshape(rows, n), y), (at, to)
        assert n_launches >= 2
    assert apart == 1 or rows > 1 or dtype == synth.Q8_0 or n > 4096
    w.free()
