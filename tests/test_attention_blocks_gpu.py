"""Grouped attention in blocks of three warps."""
import numpy as np
import pytest

from helpers import f16_round, rel_l2
from sapient_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,H,Hkv,sq,sk", [(128, 16, 8, 63, 97), (96, 8, 4, 125, 161), (80, 16, 8, 81, 90), (64, 16, 8, 100, 113), (128, 16, 8, 64, 300)])
def test_three_warps(oracle, hd, H, Hkv, sq, sk):
    """(Query rows, cached heads) in one round of the SMs as blocks of three warps and in two as blocks of four."""
    rng = np.random.default_rng(hd + sk)
    q = rng.standard_normal((H, sq, hd)).astype(np.float32)
    k, v = (f16_round(rng.standard_normal((Hkv, sk, hd))) for _ in range(2))
    # queries and weights in two fp16 parts (2^-22), f32 sums
    assert rel_l2(ops.gqa_attention(q, k, v), oracle.attention(q, k, v, oracle.causal_mask(sq, sk))) < 1e-5
