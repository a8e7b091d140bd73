"""Decode attention over long key ranges, whose pages are looked up ahead of their rows, and grouped attention in blocks of three warps."""
import numpy as np
import pytest

from helpers import f16_round, rel_l2
from sapient_b200 import _lib, ops

pytestmark = pytest.mark.gpu
KV_PAGE = 16


@pytest.mark.parametrize("hd", [32, 64, 80, 128, 256])
@pytest.mark.parametrize("lengths,n_splits", [((700, 17, 1), 1), ((700, 33, 2), 3), ((1501, 16, 49), 7), ((65, 31, 15), 2)])
def test_ranges_over_scattered_pages(hd, lengths, n_splits):
    """Ranges that begin inside a round and a page, many rounds long and shorter than one; every sequence's pages lie in any order."""
    import torch

    rng = np.random.default_rng(hd + n_splits)
    H = Hkv = 3  # (unshared heads: never the grouped kernel)
    max_pages = (max(lengths) + KV_PAGE - 1) // KV_PAGE
    table = rng.permutation(len(lengths) * max_pages).astype(np.int32).reshape(len(lengths), max_pages)
    pool = rng.standard_normal((table.size, 2, Hkv, KV_PAGE, hd)).astype(np.float16)
    q = rng.standard_normal((len(lengths), H, hd)).astype(np.float32)
    dev = {n: torch.from_numpy(a).cuda() for n, a in (("q", q), ("pool", pool), ("table", table), ("slot", np.arange(len(lengths), dtype=np.int32)),
                                                      ("pos", np.array(lengths, np.int32) - 1))}
    out = torch.full((len(lengths), H * hd), float("nan"), device="cuda")
    _lib.check(_lib.lib().sp_cuda_attention_paged_static(0, dev["q"].data_ptr(), H * hd, out.data_ptr(), H * hd, len(lengths), H, Hkv, hd, dev["slot"].data_ptr(),
                                                         dev["pos"].data_ptr(), dev["pool"].data_ptr(), dev["table"].data_ptr(), table.size, max_pages, 0, n_splits, None))
    got = out.cpu().numpy().reshape(len(lengths), H, hd)
    for s, n in enumerate(lengths):
        k, v = (pool[table[s], i].transpose(1, 0, 2, 3).reshape(Hkv, -1, hd)[:, :n].astype(np.float64) for i in (0, 1))
        w = np.einsum("hd,hkd->hk", q[s].astype(np.float64), k) * hd ** -0.5
        w = np.exp(w - w.max(1, keepdims=True))
        want = np.einsum("hk,hkd->hd", w / w.sum(1, keepdims=True), v)
        assert rel_l2(got[s], want) < 1e-5, n  # f32 scores and sums of up to 1501 terms


@pytest.mark.parametrize("hd,H,Hkv,sq,sk", [(128, 16, 8, 63, 97), (96, 8, 4, 125, 161), (80, 16, 8, 81, 90), (64, 16, 8, 100, 113), (128, 16, 8, 64, 300)])
def test_three_warps(oracle, hd, H, Hkv, sq, sk):
    """(Query rows, cached heads) in one round of the SMs as blocks of three warps and in two as blocks of four."""
    rng = np.random.default_rng(hd + sk)
    q = rng.standard_normal((H, sq, hd)).astype(np.float32)
    k, v = (f16_round(rng.standard_normal((Hkv, sk, hd))) for _ in range(2))
    # queries and weights in two fp16 parts (2^-22), f32 sums
    assert rel_l2(ops.gqa_attention(q, k, v), oracle.attention(q, k, v, oracle.causal_mask(sq, sk))) < 1e-5
