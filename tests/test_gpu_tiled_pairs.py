"""GPU tests of the tensor-core matmul by pairs of CTAs (q40_gemm_tiled_tc_ws): edges of its tiles, of its k blocks and of
the shares that pairs take of a tile, against the numpy oracle."""
import ctypes

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


def mats(K, rng, Kd, Ns):
    packed = [O.quantize_q40((rng.standard_normal((Kd, n)) * 0.1).astype(np.float16), 64) for n in Ns]
    tiled = [K.relayout_tiled(torch.from_numpy(q).cuda(), torch.from_numpy(s).cuda(), (Kd, n)) for (q, s), n in zip(packed, Ns)]
    return packed, tiled


def scratch(K, M):
    from spec_mcts_b200._lib import lib
    return torch.zeros(max(lib.q40_gemm_tiled_tc_ws_bytes(M), 16), dtype=torch.uint8, device="cuda")


def launch(a, tiled, outs, Ns, silu, ws, pdl=0):
    from spec_mcts_b200._lib import check, lib
    n = len(tiled)
    P = ctypes.c_void_p * n
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    check(lib.q40_gemm_tiled_tc_ws(n, a.data_ptr(), a.stride(0), P(*[t.data_ptr() for t in tiled]), P(*[o.data_ptr() for o in outs]),
                                   (ctypes.c_int64 * n)(*[o.stride(0) for o in outs]), (ctypes.c_int * n)(*Ns), a.shape[0],
                                   a.shape[1], silu, ws.data_ptr(), ws.numel(), err.data_ptr(), pdl,
                                   torch.cuda.current_stream().cuda_stream), "q40_gemm_tiled_tc_ws")
    assert int(err.item()) == 0


def close(got, want):
    # fp32 sums of fp16 operands in any order: rel 2^-11 for the rounded result and 2^-24 per addition, against the
    # oracle's own fp16 result; the floor is that of cancelled sums (a few fp16 steps of the mean magnitude)
    want = want.astype(np.float32)
    scale = float(np.abs(want).mean())
    np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=2e-3, atol=4e-3 * max(scale, 1e-6))


# rows at the edges of 16-row tiles, of the two ways of tensor memory (192, 256) and of the row chunks; k of one step, an odd
# number of steps, and whole blocks; one span, several, and more than there are pairs
@pytest.mark.parametrize("M,Kd,Ns", [(9, 64, (256,)), (16, 192, (256, 512)), (17, 128, (256,)), (100, 4160, (512,)), (128, 320, (256, 256, 256)),
                                     (129, 64, (512,)), (192, 320, (256,)), (193, 256, (512, 256)), (256, 192, (256,)), (257, 1024, (256,)),
                                     (10, 256, (9728, 9728)), (112, 448, (19200,)), (300, 192, (19200,))])
def test_products_at_the_edges(K, M, Kd, Ns):
    rng = np.random.default_rng(M * 100 + Kd)
    packed, tiled = mats(K, rng, Kd, Ns)
    a = rng.standard_normal((M, Kd)).astype(np.float16)
    a_d, ws = torch.from_numpy(a).cuda(), scratch(K, M)
    outs = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in Ns]
    launch(a_d, tiled, outs, Ns, 0, ws)
    for o, (q, s), n in zip(outs, packed, Ns):
        close(o, O.matmul_q40(a, q, s, (Kd, n)))
    # once more behind a dependent launch of the same scratch: the same bits, and the flags as they were found
    again = [torch.empty_like(o) for o in outs]
    launch(a_d, tiled, again, Ns, 0, ws, 1)
    assert all(torch.equal(x, y) for x, y in zip(outs, again))
    assert not ws[:8192].any()


def test_rows_and_strides_outside_stay(K):
    """Outputs that are column ranges of a wider buffer, at 16-byte and at 4-byte alignment, and activations with a row pitch:
    nothing around them is written."""
    rng = np.random.default_rng(5)
    M, Kd, n = 21, 192, 256
    packed, tiled = mats(K, rng, Kd, (n,))
    wide = torch.from_numpy(rng.standard_normal((M, Kd + 8)).astype(np.float16)).cuda()
    a = wide[:, :Kd]
    want = O.matmul_q40(np.ascontiguousarray(a.cpu().numpy()), *packed[0], (Kd, n))
    for first, pitch in ((8, 272), (2, 262)):
        buf = torch.full((M + 1, pitch), 7.0, dtype=torch.float16, device="cuda")
        launch(a, tiled, [buf[:M, first:first + n]], (n,), 0, scratch(K, M))
        close(buf[:M, first:first + n], want)
        assert (buf[:M, :first] == 7).all() and (buf[:M, first + n:] == 7).all() and (buf[M] == 7).all()


@pytest.mark.parametrize("M,Kd,n", [(9, 64, 256), (16, 192, 512), (77, 1088, 512), (128, 256, 256), (129, 320, 512), (300, 192, 1024),
                                    (20, 256, 9728)])
def test_silu_product_is_that_of_the_separate_launches(K, M, Kd, n):
    rng = np.random.default_rng(M + Kd)
    _, tiled = mats(K, rng, Kd, (n, n))
    a, ws = torch.from_numpy(rng.standard_normal((M, Kd)).astype(np.float16)).cuda(), scratch(K, M)
    outs = [torch.empty((M, n), dtype=torch.float16, device="cuda") for _ in range(2)]
    launch(a, tiled, outs, (n, n), 0, ws)
    g = torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda")
    launch(a, tiled, [g, g], (n, n), 1, ws, 1)
    want = K.silu_mul(*outs)
    # k may be cut at other places, which moves a sum by its last fp32 bits and a product by an fp16 step of either factor
    np.testing.assert_allclose(g.float().cpu().numpy(), want.float().cpu().numpy(), rtol=4e-3, atol=1e-4)
    assert (g == want).float().mean() > 0.97


def test_silu_of_every_fp16_value(K):
    """The product's SiLU rounds like the launch that divides: x and y are the activation itself, which takes every value."""
    Kd, n, M = 64, 256, 65536
    q, s = np.zeros((Kd * n // 128, 64), np.int8), np.zeros((Kd * n // 64,), np.float16)
    q[:n // 128], s[:n // 64] = 0x11, 1                          # the first row of the matrix: ones
    tiled = [K.relayout_tiled(torch.from_numpy(q).cuda(), torch.from_numpy(s).cuda(), (Kd, n))] * 2
    x = torch.arange(M, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.float16)
    a = torch.zeros((M, Kd), dtype=torch.float16, device="cuda")
    a[:, 0] = x
    g = torch.empty((M, n), dtype=torch.float16, device="cuda")
    launch(a, tiled, [g, g], (n, n), 1, scratch(K, M))
    want = K.silu_mul(x, x)
    assert torch.equal(g.view(torch.int16)[~want.isnan()], want.view(torch.int16)[~want.isnan()].view(-1, 1).expand(-1, n)) and g[want.isnan()].isnan().all()


@pytest.mark.parametrize("M,n", [(16, 256), (10, 9728), (129, 512)])
def test_silu_of_a_sum_that_rounds_to_minus_zero(K, M, n):
    """x is a negative sum below the smallest fp16, y is 1: the product is -0, as by the launch that divides."""
    Kd, rows = 64, n // 128
    mats = [(np.zeros((Kd * rows, 64), np.int8), np.zeros((Kd * n // 64,), np.float16)) for _ in range(2)]
    for k, (q, s) in enumerate(mats):                            # row k of matrix k: 2^-14 in the first, ones in the second
        q[k * rows:(k + 1) * rows], s[k * n // 64:(k + 1) * n // 64] = 0x11, 1 if k else 2 ** -14
    tiled = [K.relayout_tiled(torch.from_numpy(q).cuda(), torch.from_numpy(s).cuda(), (Kd, n)) for q, s in mats]
    a = torch.zeros((M, Kd), dtype=torch.float16, device="cuda")
    a[:, 0], a[:, 1] = -2.0 ** -24, 1
    g, ws = torch.empty((M, n), dtype=torch.float16, device="cuda"), scratch(K, M)
    launch(a, tiled, [g, g], (n, n), 1, ws)
    outs = [torch.empty((M, n), dtype=torch.float16, device="cuda") for _ in range(2)]
    launch(a, tiled, outs, (n, n), 0, ws)
    assert (outs[0].view(torch.int16) == -0x8000).all() and (outs[1] == 1).all()
    assert torch.equal(g.view(torch.int16), K.silu_mul(*outs).view(torch.int16)) and torch.signbit(g).all()


# the k range of a tile over two, three and four pairs of a cluster, each finishing some groups of four rows: one group and none for
# some ranks, the last one ragged, as many as divide and not
@pytest.mark.parametrize("M", [1, 4, 9, 13, 17, 36, 100, 128])
@pytest.mark.parametrize("Kd,n", [(1024, 1024), (4096, 4096), (11008, 256), (8256, 512)])
def test_k_split_over_a_cluster(K, M, Kd, n):
    rng = np.random.default_rng(M + Kd)
    packed, tiled = mats(K, rng, Kd, (n,))
    a = rng.standard_normal((M, Kd)).astype(np.float16)
    a_d, out = torch.from_numpy(a).cuda(), torch.full((M + 1, n + 8), 7.0, dtype=torch.float16, device="cuda")
    launch(a_d, tiled, [out[:M, :n]], (n,), 0, scratch(K, M))
    close(out[:M, :n], O.matmul_q40(a, *packed[0], (Kd, n)))
    assert (out[M] == 7).all() and (out[:, n:] == 7).all()
    again = torch.empty((M, n), dtype=torch.float16, device="cuda")
    for _ in range(3):
        launch(a_d, tiled, [again], (n,), 0, scratch(K, M), 1)
        assert torch.equal(again, out[:M, :n])


# as many tiles as take more than a wave of pairs, or less than one, with k ranges long enough to be worth sharing, whether 60 or
# 74 pairs run: a tile on two pairs or on three (40 tiles), blocks that do and do not divide among them, one and several
# 16-row chunks
@pytest.mark.parametrize("M,Kd,Ns,silu", [(10, 4096, (11008, 11008), 1), (16, 8320, (5120, 5120), 1), (16, 8064, (10240,), 0), (9, 4160, (19456,), 0),
                                          (33, 6144, (10240, 10240), 0)])
def test_tiles_shared_between_pairs(K, M, Kd, Ns, silu):
    rng = np.random.default_rng(M * 100 + Kd)
    packed, tiled = mats(K, rng, Kd, Ns)
    acts = [rng.standard_normal((M, Kd)).astype(np.float16) for _ in range(2)]
    acts_d, ws = [torch.from_numpy(a).cuda() for a in acts], scratch(K, M)

    def run(a, pdl=0):
        outs = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in (Ns[:1] if silu else Ns)]
        launch(a, tiled, outs * 2 if silu else outs, Ns, silu, ws, pdl)
        return outs

    first = [run(a) for a in acts_d]
    assert ws[8192:].any(), "no sums went through the scratch"
    for a, outs in zip(acts, first):
        want = [O.matmul_q40(a, q, s, (Kd, n)) for (q, s), n in zip(packed, Ns)]
        if not silu:
            for o, w in zip(outs, want):
                close(o, w)
            continue
        # the bounds of `close` for either factor f (df = 2e-3 |f| + 4e-3 mean|f|), and two more roundings to fp16
        x, y = (w.astype(np.float64) for w in want)
        dx, dy = (2e-3 * np.abs(f) + 4e-3 * np.abs(f).mean() for f in (x, y))
        g = x / (1 + np.exp(-x))
        bound = 1.1 * dx * np.abs(y) + np.abs(g) * dy + dx * dy + 2e-3 * np.abs(g * y) + 1e-4       # |silu'| < 1.1
        assert (np.abs(outs[0].double().cpu().numpy() - g * y) <= bound).all()
    # scratch and flags of one launch are the next one's, launched while it drains
    for i in (0, 1, 1, 0, 1):
        assert all(torch.equal(o, f) for o, f in zip(run(acts_d[i], 1), first[i]))
    assert not ws[:8192].any()


def test_a_share_that_never_comes_is_given_up_after_seconds(K):
    """Arrivals of the first pair start so low that the wait for its sums runs out: an error word instead of a result, not
    before the time that the kernel's other waits allow, and the next launch on zeroed scratch works.  The word may be host
    memory, as that of a model's steps is."""
    from spec_mcts_b200._lib import check, lib
    rng = np.random.default_rng(1)
    M, Kd, n = 16, 8064, 5120                       # 40 tiles: all are shared, on 60 to 74 pairs
    _, tiled = mats(K, rng, Kd, (n, n))
    a, ws = torch.from_numpy(rng.standard_normal((M, Kd)).astype(np.float16)).cuda(), scratch(K, M)
    want, g = (torch.empty((M, n), dtype=torch.float16, device="cuda") for _ in range(2))
    launch(a, tiled, [want, want], (n, n), 1, ws)
    assert ws[8192:].any()                          # sums went through the scratch
    ws[:8192].view(torch.int32)[:8] = -1000
    P, err = ctypes.c_void_p * 2, torch.zeros(1, dtype=torch.int32).pin_memory()
    t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    t0.record()
    check(lib.q40_gemm_tiled_tc_ws(2, a.data_ptr(), a.stride(0), P(*[t.data_ptr() for t in tiled]), P(*[g.data_ptr()] * 2),
                                   (ctypes.c_int64 * 2)(n, n), (ctypes.c_int * 2)(n, n), M, Kd, 1, ws.data_ptr(), ws.numel(),
                                   err.data_ptr(), 0, torch.cuda.current_stream().cuda_stream), "q40_gemm_tiled_tc_ws")
    t1.record()
    t1.synchronize()
    assert int(err.item()) == 1 and 1000 < t0.elapsed_time(t1) < 20000
    ws[:8192].zero_()
    launch(a, tiled, [g, g], (n, n), 1, ws, 1)
    assert torch.equal(g, want)


@pytest.mark.parametrize("M", [161, 171, 176, 177])     # tiles of 176 rows, and the smaller ones of the next more
def test_largest_tiles_with_sums_of_ranges(K, M):
    """k in ranges that are summed one after the other, in tiles whose ring has just the room it needs, against float64."""
    g = torch.Generator(device="cuda").manual_seed(M)
    Kd, Ns = 4096, (4096, 4096, 4096)
    packed = [K.quantize_q40((torch.randn((Kd, n), generator=g, device="cuda") * 0.05).half()) for n in Ns]
    tiled = [K.relayout_tiled(q, s, (Kd, n)) for (q, s), n in zip(packed, Ns)]
    a, ws = torch.randn((M, Kd), generator=g, device="cuda").half(), scratch(K, M)
    outs = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in Ns]
    launch(a, tiled, outs, Ns, 0, ws)
    for o, (q, s), n in zip(outs, packed, Ns):
        w = K.dequantize_q40(q, s, 64, (Kd, n)).double()         # the operand as it is multiplied
        want, size = a.double() @ w, a.double().abs() @ w.abs()
        # fp32 sums (2^-24 per addition, 1e-5 covers 4096 of them in any grouping) and the result's half step
        assert ((o.double() - want).abs() <= want.abs() * 2 ** -11 + 2 ** -25 + 1e-5 * size).all()
    again = [torch.empty_like(o) for o in outs]
    launch(a, tiled, again, Ns, 0, ws, 1)
    assert all(torch.equal(x, y) for x, y in zip(outs, again))


@pytest.mark.parametrize("M,n,silu", [(16, 5120, 1), (100, 4096, 0), (300, 4096, 0)])     # shared tiles; one tile a pair; ranges and chunks of rows
def test_a_launch_behind_one_that_waits_for_seconds(K, M, n, silu):
    """A dependent launch is there early.  It does not count the time that the launch in front takes (here one whose wait runs out) as its own."""
    from spec_mcts_b200._lib import check, lib
    rng = np.random.default_rng(M)
    m, Kd, n0 = 16, 8064, 5120
    _, front = mats(K, rng, Kd, (n0, n0))
    _, tiled = mats(K, rng, Kd, (n,) * (1 + silu))
    x, a = (torch.from_numpy(rng.standard_normal((r, Kd)).astype(np.float16)).cuda() for r in (m, M))
    ws0, ws = scratch(K, m), scratch(K, M)
    want, got = (torch.empty((M, n), dtype=torch.float16, device="cuda") for _ in range(2))
    launch(a, tiled, [want] * (1 + silu), (n,) * (1 + silu), silu, ws)
    g = torch.empty((m, n0), dtype=torch.float16, device="cuda")
    err = torch.zeros(2, dtype=torch.int32).pin_memory()
    ws0[:8192].view(torch.int32)[:8] = -1000
    torch.cuda.synchronize()

    def one(mats_, x_, out, N, s, w, e):
        k = len(mats_)
        P = ctypes.c_void_p * k
        check(lib.q40_gemm_tiled_tc_ws(k, x_.data_ptr(), x_.stride(0), P(*[t.data_ptr() for t in mats_]), P(*[out.data_ptr()] * k), (ctypes.c_int64 * k)(*[N] * k),
                                       (ctypes.c_int * k)(*[N] * k), x_.shape[0], Kd, s, w.data_ptr() if w.numel() else None, w.numel(), e.data_ptr(), 1,
                                       torch.cuda.current_stream().cuda_stream), "q40_gemm_tiled_tc_ws")

    one(front, x, g, n0, 1, ws0, err[:1])
    one(tiled, a, got, n, silu, ws, err[1:])
    torch.cuda.synchronize()
    assert err.tolist() == [1, 0] and torch.equal(got, want)
