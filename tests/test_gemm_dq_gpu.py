"""The GEMM with exact-class operands inside engine steps: several matrices of different formats in one launch, biases, sums into the
residual stream, tiles walked over and tiles shared by clusters, and the kernels that make its operands at every number of pieces
per thread. The same steps on the integer-digit GEMV (other kernels, exact products) are the reference."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from sapient_b200 import ops, synth
from sapient_b200._lib import check, lib
from sapient_b200.engine import ForwardEngine
from sapient_b200.synth import Q4_K, Q6_K, Q8_0

pytestmark = pytest.mark.gpu

BASE = dict(n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, vocab=320, norm_eps=1e-5, rope_theta=1e4, tied=False)


def _compare(shape, formats, tokens):
    cfg, W = synth.build_model(dict(BASE, **shape), seed=3, device="cuda", max_ctx=512)
    g = torch.Generator(device="cuda").manual_seed(4)
    for name, (dt, dims, _) in list(W.items()):
        role = name.split(".")[-2]
        if len(dims) == 2 and role in formats:
            w = torch.randn(*dims, generator=g, device="cuda") * 0.02
            W[name] = (formats[role], dims, synth.quantize(formats[role], w).reshape(-1))
        if role in ("k_proj", "v_proj") and len(dims) == 2:
            # keys and values are their biases: one near an edge of the cache's fp16 would move by 2^-11 of itself, and with it every
            # later row by 1e-4
            W[name] = (W[name][0], dims, torch.zeros_like(W[name][2]))
    W = synth.weights_to_numpy(W)
    ids = np.random.default_rng(tokens).integers(0, cfg["vocab"], tokens).astype(np.uint32)
    out = []
    for mode in (2, 0):
        eng = ForwardEngine.from_weights(cfg, W, max_tokens=512)
        eng.set_large_m_gemm(mode)
        eng.set_graphs(False)
        eng.set_kv_rounding(False)
        out.append(eng.forward_all_logits(ids))
        eng.close()
    # A product differs by some 1e-6 of a row's norm (operands to 2^-22, f32 sums; tests/test_gemm_tc5_gpu.py) and a layer has four in a row,
    # each through a norm or an activation: 1e-5 of a row of logits, held to four times that.
    rows = np.linalg.norm(out[0] - out[1], axis=1) / np.linalg.norm(out[1], axis=1)
    assert rows.max() < 4e-5, rows.max()
    assert rel_l2(out[0], out[1]) < 1e-5


# gate and up: 152 tiles and more for 148 SMs, so that a block walks from a tile of one format into one of another
@pytest.mark.parametrize("tokens", [40, 300])
@pytest.mark.parametrize("gate,up", [(Q4_K, Q8_0), (Q8_0, Q4_K), (Q6_K, Q4_K), (Q4_K, Q6_K)])
def test_matrices_of_different_formats_in_one_launch(gate, up, tokens):
    _compare(dict(arch="qwen2", hidden=512, ffn=9728, qkv_bias=True),
             {"gate_proj": gate, "up_proj": up, "down_proj": up, "q_proj": up, "k_proj": gate, "v_proj": Q8_0, "o_proj": gate}, tokens)


# norms of two and four pieces per thread and of rows that do not fit; sums into the residual stream from as many tiles as hidden / 128
@pytest.mark.parametrize("hidden,tokens", [(6144, 33), (12288, 20), (19200, 17), (19200, 150)])
def test_wide_rows_and_sums_into_the_stream(hidden, tokens):
    _compare(dict(arch="qwen2", hidden=hidden, ffn=256, qkv_bias=True), {"down_proj": Q8_0, "o_proj": Q4_K}, tokens)


@pytest.mark.parametrize("hidden,ffn,tokens", [(6400, 1280, 40), (9216, 512, 18), (640, 19456, 70)])
def test_layer_norms_of_wide_rows_and_biases_of_many_tiles(hidden, ffn, tokens):
    _compare(dict(arch="phi2", hidden=hidden, ffn=ffn, n_kv_heads=4, rotary_dim=32), {}, tokens)


# rows x weight rows x columns by how launch_gemm_dq deals them out on 148 SMs: one wave of clusters; whole rounds walked over; a walk and a
# few tiles shared (of one, two and three rounds); clusters in several waves
@pytest.mark.parametrize("dtype", [Q4_K, Q6_K, Q8_0])
@pytest.mark.parametrize("m,n,k", [(20, 512, 4096), (100, 17920, 512), (192, 17920, 512), (20, 19077, 2560), (130, 19100, 2304), (257, 19077, 1536), (300, 4096, 5120)])
def test_every_way_of_dealing_out_tiles(dtype, m, n, k):
    """Element by element against float64: within 4e-6 of sum |x w| (operands 2^-22, at most 48 truncated additions of 2^-24 before a
    sum leaves the tensor core, an f32 sum of 2^-24 per 256 columns after it)."""
    be, _ = synth.BLOCK[dtype]
    w = ops.Weight(dtype, n, k, synth.random_bit_blocks(dtype, n * k // be, seed=m + n + dtype))
    W = torch.from_numpy(w.dequant()).cuda().double()
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(m)).cuda()
    y = [torch.full((m, n), 7.0, device="cuda") for _ in range(2)]
    for t in y:
        w.matmul_nt_dev(x.data_ptr(), m, t.data_ptr())
    check(lib().sp_cuda_check_kernels(0))
    w.free()
    want, size = x.double() @ W.T, x.double().abs() @ W.abs().T
    assert torch.equal(y[0], y[1])
    assert float(((y[0].double() - want).abs() / size).max()) < 4e-6
