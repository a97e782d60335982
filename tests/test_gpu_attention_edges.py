"""GPU tests of the attention kernels at the edges of their tiles, pages and row splits, against the numpy oracle."""
import numpy as np
import pytest
import torch

from oracle import q40_oracle as O

pytestmark = pytest.mark.gpu

# fp16 operands and result, fp32 sums and softmax: an fp16 step of the result and the hardware's 2^x (2 ulp of fp32)
TOL = dict(rtol=2e-3, atol=1e-3)


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from spec_mcts_b200 import kernels
    return kernels


def normal(rng, *shape):
    return rng.standard_normal(shape).astype(np.float16)


# rows on either side of every split of warps (32 heads: 296, 444, 592, 740 rows), page sizes that are and are not powers of two
@pytest.mark.parametrize("B,L,Hkv,page,idx", [(1, 1, 32, 1, np.int16), (9, 130, 32, 16, np.int32), (10, 65, 8, 3, np.int32), (14, 129, 32, 1, np.int16),
                                              (19, 128, 32, 5, np.int32), (19, 140, 32, 1, np.int16), (24, 33, 32, 20, np.int32)])
def test_paged_rows(K, B, L, Hkv, page, idx):
    rng = np.random.default_rng(B * 7 + L)
    H, pages = 32, -(-L // page)
    P = B * pages * page
    table = rng.permutation(B * pages).reshape(B, pages).astype(idx)
    lens = rng.integers(0, L + 1, B).astype(np.int32)
    lens[0], lens[-1] = L, L
    q, k, v = normal(rng, B, H, 128), normal(rng, Hkv, P, 128), normal(rng, Hkv, P, 128)
    d = lambda x: torch.from_numpy(x).cuda()
    o = K.page_flash_attn(d(table), d(q), d(k), d(v), P, B, L, H, 128, page_size=page, seq_lens=d(lens)).float().cpu().numpy()
    for b in range(B):
        n = int(lens[b])
        if n == 0:
            assert not o[b].any()
            continue
        at = np.arange(n)
        slot = table[b].astype(np.int64)[at // page] * page + at % page
        kb, vb = (np.repeat(x[:, slot].astype(np.float64), H // Hkv, axis=0) for x in (k, v))
        s = np.einsum("hd,hnd->hn", q[b].astype(np.float64), kb) / np.sqrt(128.0)
        w = np.exp(s - s.max(axis=1, keepdims=True))
        np.testing.assert_allclose(o[b], np.einsum("hn,hnd->hd", w / w.sum(axis=1, keepdims=True), vb), **TOL)


# one tile, a tile's last and first key, ragged splits; one row block, its edge (64 rows) and two, with branches of no own keys
@pytest.mark.parametrize("B,prefix,Hkv", [(1, 1, 2), (3, 64, 2), (5, 65, 1), (64, 130, 2), (65, 63, 2), (130, 500, 2)])
def test_prefix_beside_own_keys(K, B, prefix, Hkv):
    rng = np.random.default_rng(B + prefix)
    H, page, pages = 2, 16, 3
    q, pk, pv = normal(rng, B, H, 128), normal(rng, prefix, Hkv, 128), normal(rng, prefix, Hkv, 128)
    kp, vp = normal(rng, Hkv, B * pages * page, 128), normal(rng, Hkv, B * pages * page, 128)
    table = rng.permutation(B * pages).reshape(B, pages).astype(np.int32)
    lens = rng.integers(0, pages * page + 1, B).astype(np.int32)
    d = lambda x: torch.from_numpy(x).cuda()
    args = (d(q), d(pk), d(pv), prefix, d(table), d(lens), d(kp), d(vp))
    want = O.attn_shared_prefix(q, pk, pv, prefix, table, lens, kp, vp, page)
    outs = [K.shared_prefix_attn(*args, page_size=page) for _ in range(3)]      # the scratch of one is the next one's
    for o in outs:
        np.testing.assert_allclose(o.float().cpu().numpy(), want.astype(np.float32), **TOL)
        assert torch.equal(o, outs[0])


@pytest.mark.parametrize("S", [1, 16, 63, 65, 127, 193])
def test_causal_blocks(K, S):
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn((S, h, 128), generator=g, device="cuda").half() for h in (4, 2, 2))
    s = torch.einsum("ihd,jhd->hij", q.double(), k.double().repeat_interleave(2, 1)) / 128 ** 0.5
    s = s.masked_fill(torch.ones((S, S), device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = torch.einsum("hij,jhd->ihd", torch.softmax(s, -1), v.double().repeat_interleave(2, 1))
    np.testing.assert_allclose(K.causal_attn(q, k, v).float().cpu().numpy(), want.float().cpu().numpy(), **TOL)


def test_causal_rows_whose_first_tile_of_scores_is_minus_infinity(K):
    """Rows with a finite score later on attend to those keys alone; rows without one are zero."""
    g = torch.Generator(device="cuda").manual_seed(3)
    S, blocked = 193, 70                              # more than a tile of 64 keys
    q, k, v = (torch.randn((S, h, 128), generator=g, device="cuda").half() for h in (4, 2, 2))
    q[..., 0], k[:blocked, :, 0] = 1.0, float("-inf")
    got = K.causal_attn(q, k, v)
    s = torch.einsum("ihd,jhd->hij", q[blocked:].double(), k[blocked:].double().repeat_interleave(2, 1)) / 128 ** 0.5
    n = S - blocked
    s = s.masked_fill(torch.ones((n, n), device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = torch.einsum("hij,jhd->ihd", torch.softmax(s, -1), v[blocked:].double().repeat_interleave(2, 1))
    np.testing.assert_allclose(got[blocked:].float().cpu().numpy(), want.float().cpu().numpy(), **TOL)
    assert not got[:blocked].any()


@pytest.mark.parametrize("blocked", [70, 130])        # of 130 shared keys: a split of 64 and part of the next, then all
def test_shared_keys_whose_scores_are_minus_infinity(K, blocked):
    """They weigh nothing beside a branch's own keys and the other shared ones; a branch without any has zeros."""
    rng = np.random.default_rng(blocked)
    B, H, prefix = 3, 4, 130
    q, pk, pv = normal(rng, B, H, 128), normal(rng, prefix, H, 128), normal(rng, prefix, H, 128)
    kp, vp = normal(rng, H, 32, 128), normal(rng, H, 32, 128)
    q[..., 0], pk[:blocked, :, 0] = 1.0, -np.inf
    table, lens = np.arange(6, dtype=np.int32).reshape(3, 2) % 4, np.array([0, 5, 16], dtype=np.int32)
    d = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    got = K.shared_prefix_attn(d(q), d(pk), d(pv), prefix, d(table), d(lens), d(kp), d(vp), page_size=8).float().cpu().numpy()
    some = slice(1, None) if blocked == prefix else slice(None)       # branches with a finite score
    want = O.attn_shared_prefix(q[some], pk[blocked:], pv[blocked:], prefix - blocked, table[some], lens[some], kp, vp, 8)
    np.testing.assert_allclose(got[some], want.astype(np.float32), **TOL)
    assert blocked < prefix or not got[0].any()
