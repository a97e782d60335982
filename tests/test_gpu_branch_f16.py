"""Attention of branches over their own fp16 keys where several heads, or warps, share a row, at the edges of the 16 keys a warp takes at a time,
against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 191, 255, 256, 257]


def _case(B, H, Hkv, L, page, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    q = normal(B, H, 128)
    if page == 0:
        return q, normal(B, Hkv, L, 128), normal(B, Hkv, L, 128), None
    pages = -(-L // page)
    table = torch.randperm(B * pages, generator=g, device="cuda").view(B, pages)
    return q, normal(Hkv, B * pages * page, 128), normal(Hkv, B * pages * page, 128), table


def _want(q, k, v, table, page, L, lens, prefix=None):
    """Sums in float64, and what each would be of absolute values"""
    B, H, Hkv = q.shape[0], q.shape[1], k.shape[0 if page else 1]
    out = []
    for b in range(B):
        n = int(lens[b])
        at = (table[b, torch.arange(n, device="cuda") // page] * page + torch.arange(n, device="cuda") % page) if page else torch.arange(n, device="cuda")
        kb, vb = ((x[:, at] if page else x[b][:, at]).double() for x in (k, v))
        if prefix is not None:
            kb, vb = torch.cat((prefix[0].double().transpose(0, 1), kb), 1), torch.cat((prefix[1].double().transpose(0, 1), vb), 1)
        s = torch.einsum("grd,gkd->grk", q[b].double().view(Hkv, H // Hkv, 128), kb) / math.sqrt(128)
        w = torch.softmax(s, -1)
        out.append((torch.einsum("grk,gkd->grd", w, vb).reshape(H, 128), torch.einsum("grk,gkd->grd", w, vb.abs()).reshape(H, 128)))
    return torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out])


def _check(got, want, size, prompt):
    # the result is rounded to fp16, a prompt's weights are too; scores are fp32 sums of 128 products of some ten: as a relative error of a weight
    # 2^-24 times 128 times those
    bound = (2 ** -11 + (2 ** -11 if prompt else 0) + 2 ** -24 * 128 * 16) * size + 2 ** -25
    assert ((got.double() - want).abs() <= bound).all()


# B, H, Hkv, L, page size (0: contiguous), id type: by heads and warps of a row
@pytest.mark.parametrize("B,H,Hkv,L,page,ids", [
    (10, 32, 8, 257, 0, None), (10, 32, 8, 257, 16, "int16"), (3, 64, 1, 300, 3, "int32"),          # 4 heads, 8 warps
    (20, 32, 8, 100, 0, None), (20, 32, 8, 257, 1, "int16"),                                        # 4 warps, three stages
    (40, 32, 8, 129, 0, None), (40, 32, 8, 257, 5, "int32"), (29, 32, 8, 20, 16, "int16"),          # 4 warps
    (70, 32, 8, 97, 0, None), (70, 32, 8, 160, 16, "int32"), (150, 32, 8, 65, 0, None), (150, 32, 8, 97, 1, "int16"),      # 2, 1
    (7, 32, 8, 130, 0, None), (29, 12, 2, 160, 16, "int32"), (29, 32, 16, 255, 1, "int16"), (40, 32, 16, 33, 0, None), (60, 20, 10, 97, 8, "int32"),     # 2 heads
    (3, 32, 32, 300, 0, None), (4, 24, 8, 400, 16, "int32"), (5, 32, 8, 64, 0, None), (10, 32, 32, 257, 0, None), (29, 12, 12, 160, 16, "int16"),     # 1 head
    (25, 32, 32, 49, 0, None), (29, 28, 28, 160, 1, "int32"), (29, 48, 16, 257, 16, "int16"), (38, 32, 32, 129, 0, None), (38, 32, 32, 401, 0, None)])
def test_own_keys_against_float64(B, H, Hkv, L, page, ids):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    q, k, v, table = _case(B, H, Hkv, L, page, B + L)
    out, st = torch.full_like(q, 9.0), torch.cuda.current_stream().cuda_stream
    if page:
        lens = torch.tensor([min(n, L) for n in (LENS * (B // len(LENS) + 1))[:B]], dtype=torch.int32, device="cuda")
        t = table.to(getattr(torch, ids))
        check(lib.q40_attn_paged(t.data_ptr(), t.element_size(), t.stride(0), lens.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), k.shape[1],
                                 B, L, H, Hkv, 128, page, st))
    else:
        lens = [L] * B
        check(lib.q40_attn_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, L, H, Hkv, 128, st))
    _check(out, *_want(q, k, v, table, page, L, lens), False)


@pytest.mark.parametrize("B,H,Hkv,L,plen", [(29, 32, 8, 64, 70), (20, 32, 8, 129, 300), (29, 32, 8, 160, 513), (58, 32, 8, 97, 64), (13, 32, 8, 33, 1), (13, 32, 16, 160, 130),
                                            (4, 32, 32, 257, 70), (29, 6, 6, 160, 64), (29, 12, 12, 257, 600), (29, 28, 28, 256, 200), (29, 32, 32, 257, 128),
                                            # up to 16 and up to 32 rows a kv head, whose warps share a tile's keys: 1, 15 to 17, 63 to 65 keys, none in the last part
                                            (1, 4, 4, 33, 1), (2, 32, 4, 33, 15), (16, 4, 4, 33, 16), (5, 12, 4, 33, 17), (17, 4, 4, 33, 63), (4, 32, 4, 33, 65), (8, 16, 4, 33, 33), (16, 4, 4, 33, 600), (32, 4, 4, 33, 1100), (33, 4, 4, 33, 65)])
def test_behind_a_prompt_against_float64(B, H, Hkv, L, plen):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    q, k, v, table = _case(B, H, Hkv, L, 16, B + L)
    g = torch.Generator(device="cuda").manual_seed(plen)
    pk, pv = (torch.randn((plen, Hkv, 128), generator=g, device="cuda").half() for _ in range(2))
    lens = torch.tensor([min(n, L) for n in (LENS * (B // len(LENS) + 1))[:B]], dtype=torch.int32, device="cuda")
    t, out = table.to(torch.int32), torch.full_like(q, 9.0)
    ws = torch.empty(lib.q40_attn_shared_prefix_workspace_bytes(B, H, 128, plen), dtype=torch.uint8, device="cuda")
    check(lib.q40_attn_shared_prefix(q.data_ptr(), pk.data_ptr(), pv.data_ptr(), plen, pk.stride(0), pk.stride(1), t.data_ptr(), 4, t.stride(0), lens.data_ptr(), k.data_ptr(),
                                     v.data_ptr(), out.data_ptr(), k.shape[1], B, L, H, Hkv, 128, 16, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    _check(out, *_want(q, k, v, table, 16, L, lens, (pk, pv)), True)


@pytest.mark.parametrize("B,Hkv", [(10, 32), (10, 8), (40, 8)])
@pytest.mark.parametrize("lead", [0.0, 9.0, 36.0])    # the infinite value's weight: 1, 2^-13, 2^-52 of the largest
def test_infinities(B, Hkv, lead):
    """An infinite value makes its dim infinite, whatever its weight; a key with a score of -inf counts for nothing."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    H, L, z = 32, 300, lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    q, k, v, out = z(B, H, 128), z(B, Hkv, L, 128), z(B, Hkv, L, 128) + 1, z(B, H, 128)
    q[..., 0] = 1
    k[:, :, 7, 0], k[:, :, 40, 0] = lead * math.sqrt(128), -math.inf
    v[:, :, 21, 3], v[:, :, 21, 100] = -math.inf, math.inf
    check(lib.q40_attn_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, L, H, Hkv, 128, torch.cuda.current_stream().cuda_stream))
    assert (out[..., 3] == -math.inf).all() and (out[..., 100] == math.inf).all()
    out[..., 3] = out[..., 100] = 1
    assert (out == 1).all()


@pytest.mark.parametrize("B,H,Hkv", [(1, 32, 32), (4, 32, 32), (5, 32, 32), (7, 32, 32), (9, 32, 32), (12, 32, 32), (16, 32, 32), (20, 32, 32), (23, 32, 32), (27, 32, 32),
                                     (30, 32, 32), (40, 32, 32), (60, 32, 32), (70, 32, 32), (4, 32, 8), (6, 32, 8), (12, 32, 8), (18, 32, 8), (20, 32, 8), (30, 32, 8),
                                     (39, 32, 8), (70, 32, 8), (30, 32, 16), (3, 24, 8)])
def test_bits_do_not_depend_on_what_only_bounds_the_lengths(B, H, Hkv):
    """With lengths, neither the table's width, nor max_suffix, nor the pool's size changes a bit; but behind a prompt of eight tiles and more
    max_suffix says how many splits it has."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as K
    page, pages, longest = 16, 3, 48
    q, k, v, table = _case(B, H, Hkv, longest, page, B)
    g = torch.Generator(device="cuda").manual_seed(B)
    lens = torch.randint(0, longest + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    P = k.shape[1]
    k2, v2 = (torch.zeros((Hkv, 40 * P, 128), dtype=torch.float16, device="cuda") for _ in range(2))
    k2[:, :P], v2[:, :P] = k, v
    k1, v1 = (t[:, :max(page, int(table[:, :].max()) * page + page)].contiguous() for t in (k, v))
    tables = []
    for width in (pages, 8, 9, 16, 17, 40):               # 48, 128, 144, 256, 272 and 640 keys
        t = torch.zeros((B, width), dtype=torch.int32, device="cuda")
        t[:, :pages] = table
        tables.append(t)
    for plen in (0, 20, 400, 512, 1300):
        pk, pv = (torch.randn((max(plen, 1), Hkv, 128), generator=g, device="cuda").half() for _ in range(2))
        want = None
        for t in tables if plen < 449 else tables[-1:]:
            for kk, vv in ((k, v), (k2, v2), (k1, v1)):
                n = t.shape[1] * page
                if plen:
                    got = K.shared_prefix_attn(q, pk, pv, plen, t, lens, kk, vv, page_size=page, max_suffix=n)
                else:
                    got = K.page_flash_attn(t, q, kk, vv, kk.shape[1], B, n, H, 128, page_size=page, seq_lens=lens)
                want = got if want is None else want
                assert torch.equal(got, want), (plen, n, kk.shape[1])
