"""GPU tests of the kernels that work on single rows: widths at the edges of the normalisation's vectors, rotations of queries
and keys in one launch."""
import numpy as np
import pytest
import torch

from oracle import q40_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from spec_mcts_b200 import kernels
    return kernels


# on either side of one, two and four vectors of eight per thread (256 threads), and the kernel for any width
@pytest.mark.parametrize("dim", [8, 2040, 2048, 2056, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("in_place", [False, True])
def test_rmsnorm_widths(K, dim, in_place):
    rng = np.random.default_rng(dim)
    x, r = (rng.standard_normal((3, dim)).astype(np.float16) for _ in range(2))
    w = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float16)
    xd, rd, wd = (torch.from_numpy(v).cuda() for v in (x, r, w))
    if in_place:                                                  # the sum takes the place of the row, as in a pass
        from spec_mcts_b200._lib import check, lib
        y, h = torch.empty_like(xd), xd
        check(lib.q40_rmsnorm(xd.data_ptr(), rd.data_ptr(), wd.data_ptr(), y.data_ptr(), h.data_ptr(), 3, dim, 1e-5,
                              torch.cuda.current_stream().cuda_stream))
    else:
        y, h = K.rmsnorm(xd, wd, 1e-5, residual=rd)
    href = (x.astype(np.float32) + r.astype(np.float32)).astype(np.float16)
    assert (h.cpu().numpy().view(np.int16) == href.view(np.int16)).all()
    for got, want in ((y, O.rmsnorm(href, w, 1e-5)), (K.rmsnorm(h, wd, 1e-5), O.rmsnorm(href, w, 1e-5))):
        # fp32 sums in another order: a result on a rounding edge may fall to the other side, by one step of each rounding
        d = np.abs(got.cpu().numpy().view(np.int16).astype(np.int32) - want.view(np.int16).astype(np.int32))
        assert d.max() <= 2 and (d > 0).mean() < 0.01


# one launch; unequal heads; a tensor that only the one-pair kernel takes
@pytest.mark.parametrize("rows,Hq,Hk,D,pad_q,pad_k", [(1, 1, 1, 128, 0, 0), (77, 8, 2, 128, 0, 8), (33, 3, 5, 64, 16, 0), (5, 2, 2, 128, 0, 4),
                                                      (9, 2, 1, 20, 0, 0)])
def test_rope_of_queries_and_keys_has_the_bits_of_two_launches(K, rows, Hq, Hk, D, pad_q, pad_k):
    from spec_mcts_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(rows)
    q, k = (torch.randn((rows, h * D + p), generator=g, device="cuda").half() for h, p in ((Hq, pad_q), (Hk, pad_k)))
    cos, sin = (torch.randn((100, D // 2), generator=g, device="cuda").half() for _ in range(2))
    pos = torch.randint(0, 100, (rows,), generator=g, device="cuda", dtype=torch.int32)
    want = [x.clone() for x in (q, k)]
    for x, h in zip(want, (Hq, Hk)):
        K.rope_(x[:, :h * D].unflatten(1, (h, D)), pos, cos, sin)
    check(lib.q40_rope_qk(q.data_ptr(), Hq, q.stride(0), k.data_ptr(), Hk, k.stride(0), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                          rows, D, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(q, want[0]) and torch.equal(k, want[1])
