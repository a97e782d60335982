"""Attention of branches over their packed Q4_0 rows (q40_attn_tree_decode) at the edges of a warp's chunks of 32 keys and 16-key products,
for one, two and four warps a row, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160]


# rows up to 444, up to 1480 and above; grouped heads; scales at two-byte addresses; no prompt, one key, a longer one; scales of usual and of
# subnormal size
@pytest.mark.parametrize("B,H,Hkv,plen,cur,shift,size", [(25, 4, 4, 0, True, 0, 0.3), (25, 8, 2, 1, False, 0, 0.3), (50, 16, 16, 70, True, 0, 1e-5), (50, 24, 8, 0, False, 0, 8.0),
                                                         (100, 16, 16, 0, True, 0, 0.3), (75, 32, 8, 130, True, 0, 0.05), (25, 4, 4, 5, True, 1, 0.3), (100, 16, 16, 0, False, 1, 0.3)])
def test_own_keys_against_float64(B, H, Hkv, plen, cur, shift, size):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    D, maxP, maxT, rep = 128, 144, 160, H // Hkv
    g = torch.Generator(device="cuda").manual_seed(B * H + plen)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    q, ck, cv, pk, pv = normal(B, H * D), normal(B, Hkv * D), normal(B, Hkv * D), normal(maxP, Hkv, D), normal(maxP, Hkv, D)
    codes = [torch.randint(-128, 128, (B, maxT, Hkv, 64), generator=g, device="cuda", dtype=torch.int8) for _ in range(2)]
    flat = [torch.zeros(B * maxT * Hkv * 2 + shift, dtype=torch.float16, device="cuda")[shift:] for _ in range(2)]
    scales = [f.view(B, maxT, Hkv, 2).copy_(torch.rand((B, maxT, Hkv, 2), generator=g, device="cuda") * s) for f, s in zip(flat, (0.3, size))]
    lens = torch.tensor((LENS * (B // len(LENS) + 1))[:B], dtype=torch.int32, device="cuda")
    plen_d, pos, out = torch.tensor([plen], dtype=torch.int32, device="cuda"), lens + plen, torch.full((B, H * D), 9.0, dtype=torch.float16, device="cuda")
    ws = torch.empty(lib.q40_attn_shared_prefix_workspace_bytes(B, H, D, maxP), dtype=torch.uint8, device="cuda")
    check(lib.q40_attn_tree_decode(q.data_ptr(), H * D, pk.data_ptr(), pv.data_ptr(), maxP, plen_d.data_ptr(), pk.stride(0), pk.stride(1),
                                   codes[0].data_ptr(), scales[0].data_ptr(), codes[1].data_ptr(), scales[1].data_ptr(), maxT, pos.data_ptr(),
                                   ck.data_ptr() if cur else None, cv.data_ptr() if cur else None, Hkv * D, out.data_ptr(), B, H, Hkv, D,
                                   ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))

    def rows(c, s):                               # high nibbles: dims 0 .. 63
        return torch.cat(((c >> 4).double() * s[..., :1].double(), ((c << 4) >> 4).double() * s[..., 1:].double()), -1)

    parts = []
    for p, c, s, own in ((pk, codes[0], scales[0], ck), (pv, codes[1], scales[1], cv)):
        x = [p[:plen].double().expand(B, -1, -1, -1), rows(c, s)] + ([own.view(B, 1, Hkv, D).double()] if cur else [])
        parts.append(torch.cat(x, 1).repeat_interleave(rep, 2))
    k, v = parts
    at = torch.arange(k.shape[1], device="cuda")[None]
    there = (at < plen + lens[:, None]) | (at == plen + maxT)
    score = torch.einsum("bhd,bkhd->bhk", q.view(B, H, D).double(), k) / math.sqrt(D)
    w = torch.softmax(score.masked_fill(~there[:, None], -math.inf), -1).nan_to_num(0.0)      # no key at all: zeros
    want, size_of = torch.einsum("bhk,bkhd->bhd", w, v), torch.einsum("bhk,bkhd->bhd", w, v.abs())
    got = out.view(B, H, D).double()
    # a value's code * scale and the result are rounded to fp16 (2^-11, at least a subnormal's half step of 2^-25); a prompt's weights are too;
    # scores are fp32 sums over 128 dims of products up to some hundred: 2^-24 times 128 times those, as a relative error of a weight
    bound = (2 * 2 ** -11 + (2 ** -11 if plen else 0) + 1e-3 * 2 ** -4) * size_of + 2 * 2 ** -25
    assert ((got - want).abs() <= bound).all()


def test_own_keys_of_scales_off_four_bytes_by_two_warps_a_row():
    test_own_keys_against_float64(50, 16, 8, 70, True, 1, 0.3)


@pytest.mark.parametrize("H", [4, 64])                # four and two warps a row
@pytest.mark.parametrize("code", [-1, 2])             # of the infinite value; its weight: 1, 2^-13, 2^-52 of the largest
@pytest.mark.parametrize("lead", [0.0, 9.0, 36.0])
def test_infinities(H, code, lead):
    """A value of infinite scale makes its dims infinite, whatever its weight; the token's own key with a score of -inf counts for nothing."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    B, D, n = 20, 128, 40
    q = torch.zeros(B, H, D, dtype=torch.float16, device="cuda")
    q[..., 0] = 1
    z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    kq, vq = torch.zeros(B, n, H, 64, dtype=torch.int8, device="cuda"), torch.full((B, n, H, 64), 0x11, dtype=torch.int8, device="cuda")
    ks, vs = z(B, n, H, 2), z(B, n, H, 2) + 1
    kq[:, 7, :, 0], ks[:, 7, :, 0] = 16, lead * math.sqrt(D)             # key 7 leads
    vq[:, 21], vs[:, 21, :, 0] = (code & 15) * 17 - (256 if code < 0 else 0), math.inf
    pos, zero, out = torch.full((B,), n, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), z(B, H * D)
    ck, cv = z(B, H, D), z(B, H * D) + 1
    ck[..., 0] = -math.inf
    pk, ws = z(64, H, D), torch.empty(lib.q40_attn_shared_prefix_workspace_bytes(B, H, D, 64), dtype=torch.uint8, device="cuda")
    check(lib.q40_attn_tree_decode(q.data_ptr(), H * D, pk.data_ptr(), pk.data_ptr(), 64, zero.data_ptr(), pk.stride(0), pk.stride(1), kq.data_ptr(),
                                   ks.data_ptr(), vq.data_ptr(), vs.data_ptr(), n, pos.data_ptr(), ck.data_ptr(), cv.data_ptr(), H * D, out.data_ptr(), B, H, H, D,
                                   ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    out = out.view(B, H, 2, 64)
    assert (out[:, :, 0] == math.copysign(math.inf, code)).all()
    assert out[:, :, 1].isfinite().all()
