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
                                   (2, 1152, 2596), (1, 2048, 10711),
                                   # pairs of CTAs: one block of k and one feature, ragged features on either CTA of a pair, odd rows of the result, k split over two to
                                   # four pairs, more tiles than pairs, rows on both sides of 128 and of 256
                                   (33, 128, 1), (40, 128, 129), (48, 256, 255), (100, 4096, 257), (33, 11008, 383), (64, 2048, 1000), (77, 384, 20001), (100, 4096, 11008),
                                   (128, 640, 511), (129, 640, 640), (256, 256, 20000), (300, 1152, 1003), (513, 128, 300), (12, 8704, 8754), (9, 7040, 7001)])
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
    assert KK.tc_error_flag() == 0


@pytest.mark.parametrize("M,K,N", [(40, 1024, 515), (100, 512, 20001), (64, 4096, 300)])
def test_what_lies_around_the_result_stays_and_weights_just_written_are_read(M, K, N):
    """Behind a launch that writes the weights, as a dependent launch of its own; the result is column ranges of wider rows."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as KK
    from spec_mcts_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(N)
    ws = torch.zeros(lib.q40_gemm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    x = torch.randn((M, K + 8), generator=g, device="cuda").half()[:, :K]
    st = torch.cuda.current_stream().cuda_stream
    q, s = torch.zeros((N * K // 128, 64), dtype=torch.int8, device="cuda"), torch.zeros(N * K // 64, dtype=torch.float16, device="cuda")
    for first in (8, 1, 2):
        w = (torch.randn((N, K), generator=g, device="cuda") * 0.05).half()
        y = torch.full((M + 1, N + 11), 7.0, dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        check(lib.q40_quantize(w.data_ptr(), q.data_ptr(), s.data_ptr(), N * K, 64, st))
        check(lib.q40_gemm_nk(x.data_ptr(), x.stride(0), q.data_ptr(), s.data_ptr(), y[:, first:].data_ptr(), y.stride(0), M, N, K, 64, ws.data_ptr(), ws.numel(), st))
        want = x.double() @ KK.dequantize_q40(q, s, 64, (N, K)).double().t()
        got = y[:M, first:first + N].double()
        # as above, without the operands' rounding: fp32 sums and the result's half step
        assert ((got - want).abs() <= want.abs() * 2 ** -11 + 2 ** -25 + 1e-5 * (x.double().abs() @ KK.dequantize_q40(q, s, 64, (N, K)).double().abs().t())).all()
        assert (y[M] == 7).all() and (y[:, :first] == 7).all() and (y[:, first + N:] == 7).all()
        assert not ws.any()                                   # no counter, no error word


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


@pytest.mark.parametrize("M,K,N", [(33, 256, 300), (100, 1152, 2050)])
def test_rows_off_16_bytes_have_the_same_bits_captured_too(M, K, N):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as KK
    from spec_mcts_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(M)
    q, s = KK.quantize_q40((torch.randn((N, K), generator=g, device="cuda") * 0.05).half())
    x = torch.randn((M, K), generator=g, device="cuda").half()
    off = torch.zeros(4 + M * (K + 4), dtype=torch.float16, device="cuda")[4:].view(M, K + 4)[:, :K].copy_(x)
    ws = torch.zeros(max(lib.q40_gemm_workspace_bytes(M, N, K), 4096 + 2 * M * K), dtype=torch.uint8, device="cuda")

    def call(x, y):
        check(lib.q40_gemm_nk(x.data_ptr(), x.stride(0), q.data_ptr(), s.data_ptr(), y.data_ptr(), N, M, N, K, 64, ws.data_ptr(), ws.numel(),
                              torch.cuda.current_stream().cuda_stream))
        return y
    y = [torch.zeros((M, N), dtype=torch.float16, device="cuda") for _ in range(3)]
    call(x, y[0])
    call(off, y[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(off, y[2])
    graph.replay()
    assert torch.equal(y[0], y[1]) and torch.equal(y[0], y[2])


# one block of k; more blocks than the ring has stages; k split over a cluster and not; rows that fill no pair of eight; several chunks of rows
@pytest.mark.parametrize("M,K,N", [(33, 128, 300), (40, 11008, 1000), (100, 4096, 20001), (20, 4096, 11008), (64, 11008, 128), (128, 2048, 515), (129, 640, 640), (300, 4096, 700), (513, 128, 300)])
def test_rows_8_bytes_off_have_the_same_bits_whatever_the_scratch(M, K, N, monkeypatch):
    """What a call computes, and how, does not depend on where its activations lie, nor on the calls before it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels as KK
    from spec_mcts_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    q, s = KK.quantize_q40((torch.randn((N, K), generator=g, device="cuda") * 0.05).half())
    x = torch.randn((M, K), generator=g, device="cuda").half()
    off = torch.zeros(4 + M * K, dtype=torch.float16, device="cuda")[4:].view(M, K).copy_(x)
    assert off.data_ptr() % 16 == 8
    want = KK.linear_q40(x, q, s, (N, K))
    monkeypatch.setattr(KK, "_workspaces", {})
    for _ in range(2):                                        # a first call, and one that the native way may take
        assert torch.equal(KK.linear_q40(off, q, s, (N, K)), want)
    with pytest.raises(KK.Q40Error):                          # nearer than 8 bytes: refused as ever
        KK.linear_q40(torch.zeros(1 + M * K, dtype=torch.float16, device="cuda")[1:].view(M, K), q, s, (N, K))
    assert KK.tc_error_flag() == 0
    # rows further apart, and a result that is column ranges of wider rows
    wide = torch.full((M, K + 12), 9.0, dtype=torch.float16, device="cuda")
    y = torch.full((M + 1, N + 3), 7.0, dtype=torch.float16, device="cuda")
    wide[:, 4:4 + K] = x
    ws = torch.zeros(lib.q40_gemm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    check(lib.q40_gemm_nk(wide[:, 4:].data_ptr(), K + 12, q.data_ptr(), s.data_ptr(), y[:, 1:].data_ptr(), N + 3, M, N, K, 64, ws.data_ptr(), ws.numel(),
                          torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y[:M, 1:1 + N], want) and (y[M] == 7).all() and (y[:, 0] == 7).all() and (y[:, 1 + N:] == 7).all()
    assert not ws.any()


def test_rows_8_bytes_off_from_two_threads_on_one_stream():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import threading
    from spec_mcts_b200 import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(1)
    M, K, N = 40, 2048, 1000
    q, s = KK.quantize_q40((torch.randn((N, K), generator=g, device="cuda") * 0.05).half())
    xs = [torch.zeros(4 + M * K, dtype=torch.float16, device="cuda")[4:].view(M, K).copy_(torch.randn((M, K), generator=g, device="cuda")) for _ in range(2)]
    want = [KK.linear_q40(x.clone(), q, s, (N, K)) for x in xs]
    out = [[], []]

    def work(i):
        for _ in range(300):
            out[i].append(KK.linear_q40(xs[i], q, s, (N, K)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert all(len(o) == 300 and all(torch.equal(y, w) for y in o) for o, w in zip(out, want))
