"""Quantised products of 17 rows and more at sizes where the plan takes lower tiles than need be, clusters that nearly fill their places, a
walk and shared tiles, with one to eight parts; the last rows and tiles short."""
import pytest

from sapient_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [synth.Q4_K, synth.Q6_K, synth.Q8_0])
@pytest.mark.parametrize("m,n,k", [(17, 1000, 1024), (33, 1000, 1024), (64, 512, 2048), (112, 3000, 2048), (129, 3000, 2048), (192, 1536, 1536), (300, 1152, 768),
                                   (389, 2560, 2560), (512, 500, 2048), (700, 512, 2048), (400, 6144, 1024), (1025, 1100, 512)])
def test_plans(dtype, m, n, k):
    """Of the size of a result, its products' absolute sum: operands as two fp16 parts and f32 sums leave 4e-6 at most."""
    import torch

    be, _ = synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, k, synth.random_bit_blocks(dtype, n * k // be, seed=m))
    x = torch.randn(m, k, device="cuda", generator=torch.Generator("cuda").manual_seed(k))
    y = [torch.full((m, n), float("nan"), device="cuda") for _ in range(2)]
    for out in y:
        w.matmul_nt_dev(x.data_ptr(), m, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    values = torch.from_numpy(w.dequant()).cuda().double()
    want, size = x.double() @ values.T, x.double().abs() @ values.abs().T
    assert torch.equal(y[0], y[1])
    assert float(((y[0].double() - want).abs() / size).max()) < 4e-6
    w.free()
