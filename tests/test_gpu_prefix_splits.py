"""Shared-prefix attention where the number of prefix splits is decided by what a merge has in flight (few kv heads, long prefix: 16 splits of
several tiles, the last of them shorter) and by the branches' own keys (many of them: one split per SM)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hkv,prefix,suffix,page", [(4, 32, 8, 2048, 100, 16), (3, 16, 8, 1090, 20, 1), (6, 4, 1, 1025, 64, 16),
                                                        (2, 8, 8, 1024, 0, 16), (40, 8, 8, 512, 256, 16), (60, 4, 4, 449, 130, 1)])
def test_against_64_bits(B, H, Hkv, prefix, suffix, page):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(B + prefix)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    pages = max(1, -(-suffix // page))
    q, pk, pv = normal(B, H, 128), normal(prefix, Hkv, 128), normal(prefix, Hkv, 128)
    k, v = normal(Hkv, B * pages * page, 128), normal(Hkv, B * pages * page, 128)
    table = torch.randperm(B * pages, generator=g, device="cuda").to(torch.int32).view(B, pages)
    lens = torch.randint(0, suffix + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    lens[0] = 0
    got = K.shared_prefix_attn(q, pk, pv, prefix, table, lens, k, v, page_size=page, max_suffix=suffix).double()
    for b in range(B):
        at = torch.arange(int(lens[b]), device="cuda")
        slot = table[b].long()[at // page] * page + at % page
        kk, vv = (torch.cat((p.double().transpose(0, 1), s[:, slot].double()), 1).repeat_interleave(H // Hkv, 0) for p, s in ((pk, k), (pv, v)))
        w = torch.softmax((q[b].double()[:, None] @ kk.transpose(1, 2)) / 128 ** 0.5, -1)
        # weights of the prefix pass are fp16 operands (2^-11 of each product), sums fp32, the result fp16 (2^-11)
        bound = 2 ** -10 * (w @ vv.abs())[:, 0] + 2 ** -11 * (w @ vv).abs()[:, 0] + 1e-5
        assert ((got[b] - (w @ vv)[:, 0]).abs() <= bound).all()


@pytest.mark.parametrize("B,H,Hkv,prefix", [(1, 4, 1, 8192), (10, 8, 1, 16390), (34, 4, 1, 4097), (4, 32, 8, 32768 - 63)])
def test_long_prefixes(B, H, Hkv, prefix):
    """More splits than a merge has on their way at once, up to more than a warp has lanes; a last split that is shorter, or a single key."""
    test_against_64_bits(B, H, Hkv, prefix, 40, 16)


def test_two_threads_on_one_stream():
    """The partial results of a call are merged by that call, whatever another thread enqueues on the same stream."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import threading
    from spec_mcts_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(1)
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    calls = [(normal(10, 8, 128), normal(1024, 8, 128), normal(1024, 8, 128), 1024, None, None, None, None) for _ in range(2)]
    want, out = [K.shared_prefix_attn(*c) for c in calls], [[], []]

    def work(i):
        for _ in range(500):
            out[i].append(K.shared_prefix_attn(*calls[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(len(o) == 500 and all(torch.equal(y, w) for y in o) for o, w in zip(out, want))
