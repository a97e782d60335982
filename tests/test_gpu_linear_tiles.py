"""linear_q40 at the edges of its one-CTA-per-SM kernel: rows of its three widths and beyond, single steps of k, odd numbers of steps (scales
off an 8-byte boundary), rows of W that do not fill a tile, tiles that do not fill a CTA, k split over a cluster."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(1, 128, 1), (10, 4096, 1), (40, 384, 1), (1, 128, 2), (8, 128, 17), (9, 256, 16), (16, 384, 33), (17, 640, 15), (32, 1152, 100), (33, 1152, 100), (64, 1280, 7000), (65, 1152, 7000), (97, 2048, 2050),
                                   (10, 4096, 11008), (1, 11008, 4099), (10, 11008, 4096), (16, 11008, 1000), (32, 8320, 80), (3, 896, 11841),
                                   (13, 2944, 2368), (5, 2048, 2369),
                                   # what the other kernel takes, and its neighbours: long chains of steps above eight rows, uneven CTAs up to four, a remainder of 32
                                   (16, 7040, 9825), (17, 6144, 6165), (33, 6144, 6165), (1, 4224, 4963), (4, 4224, 4963), (5, 4224, 4963), (36, 4224, 4963),
                                   (2, 1152, 2596), (1, 2048, 10711)])
def test_against_64_bits(M, K, N):
    """What is rounded: operands fp16(code * scale), by half a step (2^-11) of each product; sums in fp32 (1e-5 of the sum of magnitudes
    covers 2^-24 per addition over K); the result, by half an fp16 step (2^-11, subnormals 2^-25)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(M * 7 + K + N)
    q, s = KK.quantize_q40((torch.randn((N, K), generator=g, device="cuda") * 0.05).half())
    x = torch.randn((M, K), generator=g, device="cuda").half()
    y = KK.linear_q40(x, q, s, (N, K)).double()
    qq = q.reshape(-1, 64)
    w = torch.cat((qq >> 4, (qq << 4) >> 4), 1).view(-1, 64).double() * s.reshape(-1, 1).double()
    w, xd = w.view(N, K), x.double()
    want = xd @ w.t()
    bound = want.abs() * 2 ** -11 + 2 ** -25 + (xd.abs() @ w.abs().t()) * (1e-5 + 2 ** -11)
    assert ((y - want).abs() <= bound).all(), ((y - want).abs() / bound).max()


def test_infinities_and_nan_stay_in_their_row_and_column():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as KK
    N, K = 40, 256
    w = torch.ones((N, K), device="cuda").half()
    w[3] = -1
    q, s = KK.quantize_q40(w)
    x = torch.ones((10, K), device="cuda").half()
    x[1, 5], x[2, 77] = float("inf"), float("nan")
    s2 = s.clone().view(N, -1)
    s2[7, 1] = float("inf")
    y = KK.linear_q40(x, q, s2.view_as(s), (N, K))
    clean = [n for n in range(N) if n not in (3, 7)]
    assert torch.isnan(y[2]).all() and (y[1, clean] == float("inf")).all() and y[1, 3] == -float("inf")
    rows = [m for m in range(10) if m not in (1, 2)]
    assert (y[rows, 7] == float("inf")).all() and torch.isfinite(y[rows][:, clean]).all()
