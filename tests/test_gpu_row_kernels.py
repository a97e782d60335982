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



# activations 16 and 8 bytes apart; rows at the edges of a tile of eight and of a launch; a k range that ends inside a piece
@pytest.mark.parametrize("M,Kd,N", [(1, 128, 192), (7, 1152, 192), (9, 4096, 192), (16, 2176, 192), (33, 1152, 192),
                                    (1, 2176, 11904), (9, 2176, 11904)])          # these: 768 k in a piece, 640 in the last
def test_linear_on_rows_of_any_alignment(K, M, Kd, N):
    from spec_mcts_b200._lib import check, lib
    rng = np.random.default_rng(M + Kd)
    q, s = O.quantize_q40((rng.standard_normal((N, Kd)) * 0.1).astype(np.float16), 64)
    x = rng.standard_normal((M, Kd)).astype(np.float16)
    want = O.linear_q40_nk(x, q, s, (N, Kd), 64).astype(np.float32)
    qd, sd = torch.from_numpy(q).cuda(), torch.from_numpy(s).cuda()
    ws = torch.zeros(lib.q40_gemm_workspace_bytes(M, N, Kd), dtype=torch.uint8, device="cuda")
    bits = []
    for first, pad in ((0, 0), (0, 4), (4, 8), (8, 8)):                  # halves before the first row and behind each
        buf = torch.zeros(first + M * (Kd + pad), dtype=torch.float16, device="cuda")
        view = buf[first:].view(M, Kd + pad)[:, :Kd]
        view.copy_(torch.from_numpy(x))
        y = torch.empty((M, N), dtype=torch.float16, device="cuda")
        check(lib.q40_gemm_nk(view.data_ptr(), Kd + pad, qd.data_ptr(), sd.data_ptr(), y.data_ptr(), N, M, N, Kd, 64, ws.data_ptr(),
                              ws.numel(), torch.cuda.current_stream().cuda_stream))
        # fp16 result of fp32 sums: half a step, and a step more where the sums' order moves one across an edge
        np.testing.assert_allclose(y.float().cpu().numpy(), want, rtol=2e-3, atol=2e-3)
        bits.append(y)
    assert all(torch.equal(b, bits[0]) for b in bits)
