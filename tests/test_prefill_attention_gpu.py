"""Prefill attention on tensor cores (attention_prefill_kernel): engines that put a whole prompt through the tiled
kernel (one sequence, more than 16 tokens per step, launched directly) against engines that feed the same prompt in
chunks of 32 tokens through replayed step graphs (the per-token kernel, which reads positions from device memory),
and against the oracle."""
import numpy as np
import pytest

from helpers import oracle_engine, rel_l2, tiny_model
from sapient_b200 import ops, synth
from sapient_b200.engine import ForwardEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_llama", "tiny_qwen", "tiny_llama_tp"])
@pytest.mark.parametrize("n_prompt", [33, 64, 100, 150])
def test_tiled_prefill_attention_matches_per_token_kernel_and_oracle(oracle, name, n_prompt):
    cfg, W = tiny_model(name, max_ctx=256)
    ids = np.random.default_rng(n_prompt).integers(0, cfg["vocab"], n_prompt).astype(np.uint32)
    big = ForwardEngine.from_weights(cfg, W, max_tokens=256, fast_large_m=True)     # whole prompt in one chunk: tiled kernel + tcgen05 GEMM
    small = ForwardEngine.from_weights(cfg, W, max_tokens=32)    # chunks of 32: per-token kernel
    big.set_graphs(False)  # direct launches: the tiled kernel takes the first position as an argument
    for e in (big, small):
        e.set_kv_rounding(False)  # continuous cache rounding: this test is about the kernels
    a = big.forward_all_logits(ids)
    b = small.forward_all_logits(ids)
    ref = oracle_engine(oracle, cfg, W, kv_mode=1).forward_all_logits(ids)
    assert np.abs(a - b).max() < 2e-3, np.abs(a - b).max()
    assert np.abs(a - ref).max() < 3e-3, np.abs(a - ref).max()
    # a second chunk on top of a non-empty cache (pos0 > 0), then a decode step reading what prefill wrote
    more = np.random.default_rng(1).integers(0, cfg["vocab"], 40).astype(np.uint32)
    a2 = big.forward_all_logits_cached(more)
    b2 = small.forward_all_logits_cached(more)
    assert np.abs(a2 - b2).max() < 2e-3
    assert np.abs(big.forward_logits([5], True) - small.forward_logits([5], True)).max() < 2e-3
    big.close()
    small.close()


def test_replayed_step_graphs_do_not_freeze_positions():
    """The same number of rows at two different cache positions: the second call replays the step graph captured by
    the first, so nothing in it may depend on the positions the first call had."""
    cfg, W = tiny_model("tiny_llama", max_ctx=256)
    rng = np.random.default_rng(9)
    first, second = (rng.integers(0, cfg["vocab"], 40).astype(np.uint32) for _ in range(2))
    graphs = ForwardEngine.from_weights(cfg, W, max_tokens=64, fast_large_m=True)
    direct = ForwardEngine.from_weights(cfg, W, max_tokens=64, fast_large_m=True)
    direct.set_graphs(False)
    for e in (graphs, direct):
        e.set_kv_rounding(False)
    assert np.abs(graphs.forward_all_logits(first) - direct.forward_all_logits(first)).max() < 2e-3
    assert np.abs(graphs.forward_all_logits_cached(second) - direct.forward_all_logits_cached(second)).max() < 2e-3


@pytest.mark.parametrize("name,n_prompt", [("tiny_phi2_wide", 75), ("tiny_phi2_wide", 129), ("tiny_phi2_wide", 191), ("tiny_llama", 300), ("tiny_llama", 321)])
def test_tiled_attention_with_exact_operands(oracle, name, n_prompt):
    """Engines with exact-class operands: a prompt in one chunk (tiled kernel with leading parts and remainders) against chunks of 32
    (the f32 and grouped kernels), a second portion at a position that starts no tile, and a mixed step in which decoded tokens
    stand before and after a prompt's portion. The two differ by f32 sums and the remainders' 2^-22, and where such a difference
    crosses an edge of the cache's fp16 rounding a key or value moves by 2^-11 of itself: one in some thousand does, of 64 or more
    that a score adds up, which leaves 1e-4 of logits near 1."""
    cfg, W = tiny_model(name, max_ctx=1024)
    rng = np.random.default_rng(n_prompt)
    ids, more = (rng.integers(0, cfg["vocab"], n).astype(np.uint32) for n in (n_prompt, 163))
    big = ForwardEngine.from_weights(cfg, W, max_tokens=512, max_batch=3)
    small = ForwardEngine.from_weights(cfg, W, max_tokens=32, max_batch=3)
    for e in (big, small):
        e.set_kv_rounding(False)  # continuous cache rounding: this test is about the kernels
    tol = 1e-4
    a, b = big.forward_slot(1, ids), small.forward_slot(1, ids)
    assert np.abs(a - b).max() < tol, np.abs(a - b).max()
    more = np.concatenate([more, ids])
    a, b = big.forward_slot(1, more), small.forward_slot(1, more)
    assert np.abs(a - b).max() < tol, np.abs(a - b).max()
    for e in (big, small):
        e.forward_slot(0, ids[:9])
    step = [(0, [5], [0]), (2, ids, [n_prompt - 1]), (1, [7], [0])]
    a, b = big.forward_mixed(step), small.forward_mixed(step)
    assert np.abs(a - b).max() < tol, np.abs(a - b).max()
    ref = oracle_engine(oracle, cfg, W, kv_mode=1).forward_logits(ids, False)
    assert np.abs(a[1] - ref).max() < 3e-3
    big.close()
    small.close()


@pytest.mark.parametrize("heads,depth", [(8, 18.4), (8, 16.0), (4, 12.0)])
def test_long_flat_tails_keep_their_weight(oracle, heads, depth):
    """The first token has all of the weight but e^-depth per other token, and a value of zero: what comes out of the attention is the sum
    of up to 900 weights far below fp16's range (e^-18.4 = 2^-26.5). Queries and keys are one coordinate each, of a pair that the
    rotation leaves where it is (base 1e30). Scores of size depth in f32: 2^-23 depth per weight and the same in the reference, 1e-5;
    remainders of small weights are whole multiples of 2^-38 of the largest weight, so each may be 2^-39 off."""
    import torch

    hid = 256
    shape = dict(arch="qwen2", n_layers=1, hidden=hid, n_heads=heads, n_kv_heads=heads, head_dim=64, ffn=256, vocab=320, norm_eps=1e-5, rope_theta=1e30,
                 tied=False, qkv_bias=True)
    cfg, W = synth.build_model(shape, seed=5, device="cpu", max_ctx=1024)

    def put(name, m):
        dt, dims, _ = W[name]
        W[name] = (dt, dims, synth.quantize(dt, m).reshape(-1) if dt != synth.F32 else m.contiguous().view(torch.uint8).reshape(-1))

    n, p = heads * 64, "model.layers.0."
    embed = torch.randn(320, hid, generator=torch.Generator().manual_seed(1)) * 0.02
    embed[:2] = 0.0
    embed[0, 0] = embed[1, 1] = 1.0  # after the norm: 16 in this column
    put("model.embed_tokens.weight", embed)
    put(p + "input_layernorm.weight", torch.ones(hid))
    k, v, at = torch.zeros(n, hid), torch.zeros(n, hid), torch.arange(20, n, 64)
    k[at, 0] = depth / 16
    v[:, 1] = 30000.0 / 16
    qb = torch.zeros(n)
    qb[at] = 8.0
    put(p + "self_attn.q_proj.weight", torch.zeros(n, hid))
    put(p + "self_attn.k_proj.weight", k)
    put(p + "self_attn.v_proj.weight", v)
    put(p + "self_attn.q_proj.bias", qb)
    for name in ("self_attn.k_proj.bias", "self_attn.v_proj.bias"):
        put(p + name, torch.zeros(n))
    W = synth.weights_to_numpy(W)
    dt, dims, raw = W[p + "self_attn.k_proj.weight"]
    depth = 16.0 * float(ops.Weight(dt, *dims, raw).dequant().max())  # as quantised
    ids = np.array([0] + [1] * 899, np.uint32)
    eng = ForwardEngine.from_weights(cfg, W, max_tokens=1024)
    eng.set_kv_rounding(False)
    got = eng.forward_logits(ids, False)
    ref = oracle_engine(oracle, cfg, W, kv_mode=1).forward_logits(ids, True)  # (from the cache, with its fp16 rounding)
    assert rel_l2(got, ref) < 3e-5 + 2.0 ** -39 * np.exp(depth), rel_l2(got, ref)
    eng.close()


@pytest.mark.parametrize("later", [40, 300])
def test_portions_on_either_kernel_by_their_position(oracle, later):
    """Shared heads: 300 tokens from position 0 on take tiles, 40 from 300 on a token per block, 300 from 300 on tiles again; decoded tokens
    read what they left. Against chunks of 32, which never take tiles; the tolerance is that of the test above."""
    shape = dict(synth.CONFIGS["tiny_llama"], hidden=512, n_heads=16, n_kv_heads=8, head_dim=64)
    cfg, W = synth.build_model(shape, seed=6, device="cpu", max_ctx=1024)
    W = synth.weights_to_numpy(W)
    rng = np.random.default_rng(later)
    ids, more = (rng.integers(0, cfg["vocab"], n).astype(np.uint32) for n in (300, later))
    big, small = (ForwardEngine.from_weights(cfg, W, max_tokens=n) for n in (512, 32))
    for e in (big, small):
        e.set_kv_rounding(False)
    for step in (ids, more, [3], [4]):
        a, b = big.forward_logits(step, True), small.forward_logits(step, True)
        assert np.abs(a - b).max() < 1e-4, np.abs(a - b).max()
    ref = oracle_engine(oracle, cfg, W, kv_mode=1)
    for step in (ids, more, [3], [4]):
        want = ref.forward_logits(np.asarray(step, np.uint32), True)
    assert np.abs(a - want).max() < 3e-3
    big.close()
    small.close()
