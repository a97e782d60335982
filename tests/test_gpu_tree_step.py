"""q40_attn_tree_step against q40_rope_kv_append followed by q40_attn_tree_decode: the same bits in cache and output, the inputs left alone."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# both widths of the prefix pass and the forms of the branch pass by rows; grouped heads; no shared keys, no own keys, the last slot, a slot
# beyond the cache (nothing is appended), positions beyond the tables (clamped)
@pytest.mark.parametrize("B,H,Hkv,plen,own", [(1, 4, 4, 77, 5), (3, 8, 2, 512, 0), (20, 32, 32, 130, 33), (70, 4, 4, 64, 39), (40, 32, 8, 1, 20),
                                              (5, 4, 1, 200, 40), (2, 2, 2, 0, 7), (9, 4, 4, 512, 60)])
def test_same_bits_as_two_calls(B, H, Hkv, plen, own):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    D, maxP, maxT, n_pos = 128, 512, 40, 560
    g = torch.Generator(device="cuda").manual_seed(B + plen)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    W = (H + 2 * Hkv) * D
    qkv, pk, pv = normal(B, W), normal(maxP, Hkv, D), normal(maxP, Hkv, D)
    ang = torch.rand((n_pos, 64), generator=g, device="cuda") * 6.28
    cos, sin = ang.cos().half(), ang.sin().half()
    plen_d = torch.tensor([plen], dtype=torch.int32, device="cuda")
    pos = plen + own - torch.arange(B, device="cuda", dtype=torch.int32) % 3          # lengths differ a little
    ws = torch.zeros(lib.q40_attn_shared_prefix_workspace_bytes(B, H, D, maxP), dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    cache = [torch.randint(-128, 128, (B, maxT, Hkv, 64), generator=g, device="cuda", dtype=torch.int8),
             (torch.rand((B, maxT, Hkv, 2), generator=g, device="cuda") * 0.3).half()]
    cache += [cache[0].flip(0).contiguous(), cache[1].flip(0).contiguous()]
    two, one = [c.clone() for c in cache], [c.clone() for c in cache]
    x = qkv.clone()
    q, k, v = x[:, :H * D], x[:, H * D:(H + Hkv) * D], x[:, (H + Hkv) * D:]
    p = lambda c: [t.data_ptr() for t in c]
    o2, o1 = torch.empty((B, H * D), dtype=torch.float16, device="cuda"), torch.full((B, H * D), 9.0, dtype=torch.float16, device="cuda")
    check(lib.q40_rope_kv_append(q.data_ptr(), W, k.data_ptr(), W, v.data_ptr(), W, pos.data_ptr(), plen_d.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                 n_pos, *p(two), B, H, Hkv, D, maxT, st))
    check(lib.q40_attn_tree_decode(q.data_ptr(), W, pk.data_ptr(), pv.data_ptr(), maxP, plen_d.data_ptr(), pk.stride(0), pk.stride(1), *p(two), maxT,
                                   pos.data_ptr(), k.data_ptr(), v.data_ptr(), W, o2.data_ptr(), B, H, Hkv, D, ws.data_ptr(), ws.numel(), st))
    y = qkv.clone()
    q, k, v = y[:, :H * D], y[:, H * D:(H + Hkv) * D], y[:, (H + Hkv) * D:]
    for _ in range(2):                                   # a second time on the cache of the first: the same row again
        check(lib.q40_attn_tree_step(q.data_ptr(), W, k.data_ptr(), v.data_ptr(), W, pk.data_ptr(), pv.data_ptr(), maxP, plen_d.data_ptr(), pk.stride(0),
                                     pk.stride(1), *p(one), maxT, pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), n_pos, o1.data_ptr(), B, H, Hkv, D,
                                     ws.data_ptr(), ws.numel(), st))
        assert torch.equal(y, qkv) and torch.equal(o1, o2)
        for a, b in zip(one, two):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    appended = any(not torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(one, cache))
    assert appended == bool(((pos - plen >= 0) & (pos - plen < maxT)).any())


def test_refusals():
    from spec_mcts_b200._lib import lib
    p = 4096
    args = lambda **c: [c.get(k, d) for k, d in (("q", p), ("ldq", 256), ("k", p), ("v", p), ("ldk", 256), ("pk", p), ("pv", p), ("mp", 64), ("pl", p), ("ks", 256),
                        ("hs", 128), ("kq", p), ("kss", p), ("vq", p), ("vss", p), ("mt", 8), ("pos", p), ("cos", p), ("sin", p), ("np", 80), ("o", p), ("B", 1),
                        ("H", 2), ("Hkv", 2), ("D", 128), ("ws", p), ("wsb", 1 << 20), ("st", None))]
    assert lib.q40_attn_tree_step(*args(k=None)) == -1 and lib.q40_attn_tree_step(*args(sin=None)) == -1
    assert lib.q40_attn_tree_step(*args(np=0)) == -2 and lib.q40_attn_tree_step(*args(ldk=128)) == -2
    assert lib.q40_attn_tree_step(*args(cos=p + 8)) == -3 and lib.q40_attn_tree_step(*args(kss=p + 2)) == -3
    assert lib.q40_attn_tree_step(*args(D=64)) == -5 and lib.q40_attn_tree_step(*args(wsb=16)) < 0


@pytest.mark.parametrize("B,H,Hkv,own", [(3, 4, 4, 39), (3, 8, 2, 40), (5, 4, 1, 48), (40, 32, 8, 40)])
def test_positions_past_the_tables_behind_a_full_prompt(B, H, Hkv, own):
    """The appended row is then the cache's last, and within the length that the position as it is would give.  Such a position counts as the
    tables' last one: the bits of the two calls there, the same ones every time, the caches of every call alike."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import check, lib
    D, maxP, maxT = 128, 128, 40
    n_pos = maxP + maxT
    g = torch.Generator(device="cuda").manual_seed(own)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    W = (H + 2 * Hkv) * D
    qkv, pk, pv = normal(B, W), normal(maxP, Hkv, D), normal(maxP, Hkv, D)
    ang = torch.rand((n_pos, 64), generator=g, device="cuda") * 6.28
    cos, sin = ang.cos().half(), ang.sin().half()
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    plen, pos, last = i32(maxP), i32(*[maxP + own] * B), i32(*[n_pos - 1] * B)
    ws = torch.zeros(lib.q40_attn_shared_prefix_workspace_bytes(B, H, D, maxP), dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    cache = [torch.randint(-128, 128, (B, maxT, Hkv, 64), generator=g, device="cuda", dtype=torch.int8),
             (torch.rand((B, maxT, Hkv, 2), generator=g, device="cuda") * 0.3).half()]
    cache += [cache[0].flip(0).contiguous(), cache[1].flip(0).contiguous()]
    p = lambda c: [t.data_ptr() for t in c]
    two, x, want = [c.clone() for c in cache], qkv.clone(), torch.empty((B, H * D), dtype=torch.float16, device="cuda")
    q, k, v = x[:, :H * D], x[:, H * D:(H + Hkv) * D], x[:, (H + Hkv) * D:]
    check(lib.q40_rope_kv_append(q.data_ptr(), W, k.data_ptr(), W, v.data_ptr(), W, last.data_ptr(), plen.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                 n_pos, *p(two), B, H, Hkv, D, maxT, st))
    check(lib.q40_attn_tree_decode(q.data_ptr(), W, pk.data_ptr(), pv.data_ptr(), maxP, plen.data_ptr(), pk.stride(0), pk.stride(1), *p(two), maxT,
                                   last.data_ptr(), k.data_ptr(), v.data_ptr(), W, want.data_ptr(), B, H, Hkv, D, ws.data_ptr(), ws.numel(), st))
    q, k, v = qkv[:, :H * D], qkv[:, H * D:(H + Hkv) * D], qkv[:, (H + Hkv) * D:]
    for _ in range(20):
        one, got = [c.clone() for c in cache], torch.empty_like(want)
        check(lib.q40_attn_tree_step(q.data_ptr(), W, k.data_ptr(), v.data_ptr(), W, pk.data_ptr(), pv.data_ptr(), maxP, plen.data_ptr(), pk.stride(0),
                                     pk.stride(1), *p(one), maxT, pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), n_pos, got.data_ptr(), B, H, Hkv, D,
                                     ws.data_ptr(), ws.numel(), st))
        assert torch.equal(got, want)
        for a, b in zip(one, two):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
