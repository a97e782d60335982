"""CPU-only checks of the C-ABI library: it loads, exports every symbol the header declares,
and rejects bad arguments with the documented status codes before touching the GPU."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_functions():
    text = open(os.path.join(ROOT, "include", "q40b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(q40_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_something():
    fns = header_functions()
    assert "q40_gemm_kn" in fns and "q40_attn_shared_prefix" in fns and len(fns) >= 14


def test_library_exports_every_declared_symbol():
    from spec_mcts_b200 import _lib
    for name in header_functions():
        assert hasattr(_lib.lib, name), f"{name} declared in include/q40b200.h but not exported"
    # and the Python binding table covers the header exactly
    assert sorted(_lib.SIGNATURES) == header_functions()


def test_argument_errors_are_status_codes():
    from spec_mcts_b200._lib import lib
    assert lib.q40_abi_version() >= 1
    assert lib.q40_quantize(None, None, None, 128, 64, None) == -1          # NULL
    buf = ctypes.create_string_buffer(4096)
    p = ctypes.addressof(buf)
    p16 = (p + 15) // 16 * 16
    assert lib.q40_quantize(p16, p16, p16, 100, 64, None) == -2               # numel % 128
    assert lib.q40_quantize(p16, p16, p16, 128, 48, None) == -5               # group
    assert lib.q40_dequantize(p16 + 1, p16, p16, 128, 64, None) == -3         # alignment
    assert lib.q40_gemm_kn(p16, 64, p16, p16, p16, 100, 1, 100, 64, 64, None, 0, None) == -2   # N % 128
    assert lib.q40_gemm_nk(p16, 64, p16, p16, p16, 128, 1, 128, 64, 64, None, 0, None) == -2   # K % 128
    assert lib.q40_attn_decode(p16, p16, p16, p16, 1, 8, 4, 4, 64, None) == -5                  # D != 128
    assert lib.q40_attn_decode(p16, p16, p16, p16, 1, 8, 6, 4, 128, None) == -2                 # H % Hkv
    assert b"NULL" in lib.q40_strerror(-1)
    assert lib.q40_gemm_workspace_bytes(1, 4096, 4096) > 4096
    assert lib.q40_gemm_workspace_bytes(0, 4096, 4096) == 0


def test_workspace_of_a_single_output():
    """linear_q40 asks for the scratch of a layer with one output."""
    from spec_mcts_b200._lib import lib
    for M in (1, 8, 16, 100):
        for Kd in (128, 4096):
            assert lib.q40_gemm_workspace_bytes(M, 1, Kd) >= lib.q40_gemm_workspace_bytes(M, 2, Kd) > 4096


def test_abi_version_covers_the_tiled_layout():
    """Low nibbles of a tiled copy hold code + 8 since version 2."""
    from spec_mcts_b200._lib import lib
    assert lib.q40_abi_version() == 2


def test_extension_is_built_for_this_torch(monkeypatch):
    import torch
    from spec_mcts_b200 import build
    build.build_host()
    assert not build.host_needs_build() and not build.needs_build()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.host_needs_build() and not build.needs_build()


def test_without_extension(monkeypatch):
    """No compiler, or another torch's extension: a warning that names it, and the general way."""
    from spec_mcts_b200 import build
    from spec_mcts_b200 import kernels as K

    def fails(force=False):
        raise RuntimeError("no headers here")

    monkeypatch.setattr(build, "build_host", fails)
    with pytest.warns(UserWarning, match="_host_calls.*no headers here"):
        assert K._load_host_calls() is None
    monkeypatch.undo()
    assert K._load_host_calls() is not None


def prefix_splits(B, H, Hkv, prefix, Lmax):
    """Splits of q40_attn_shared_prefix: the scratch that it asks for is theirs.  The scratch handed over is off its boundary, so nothing is launched."""
    from spec_mcts_b200._lib import lib
    buf = ctypes.create_string_buffer(4096)
    p16 = (ctypes.addressof(buf) + 15) // 16 * 16
    status = lambda n: lib.q40_attn_shared_prefix(p16, p16, p16, prefix, Hkv * 128, 128, p16, 4, 1 << 20, p16, p16, p16, p16, 1 << 20, B, Lmax, H, Hkv, 128,
                                                  16, p16 + 4, n * B * H * 130 * 4, None)
    n = next(n for n in range(1, 400) if status(n) != -4)
    assert status(n) == -3
    assert n * B * H * 130 * 4 <= lib.q40_attn_shared_prefix_workspace_bytes(B, H, 128, prefix)
    return n


def test_prefix_splits():
    # a merge has 16 splits on their way at once: no more for up to 2048 keys ...
    assert [prefix_splits(B, 8 * Hkv, Hkv, 2048, 64) for B in (1, 4, 16) for Hkv in (1, 2)] == [16] * 6
    # ... but a longer prefix goes to as many SMs as its time is worth
    assert prefix_splits(16, 8, 1, 32768, 64) >= 64 and prefix_splits(1, 8, 1, 8192, 64) >= 32 and prefix_splits(4, 32, 8, 32768, 64) >= 32
    # one an SM behind many own keys; a table with room for many more says nothing about them
    assert prefix_splits(64, 32, 32, 1024, 256) == 4 and prefix_splits(64, 32, 32, 1024, 100) == 8
    assert prefix_splits(64, 32, 32, 8192, 4096) == prefix_splits(64, 32, 32, 8192, 64) >= 8
    for prefix in (1, 64, 65, 1024, 1025, 2049, 9999, 32768, 100000):
        for B, Hkv, rep in ((1, 1, 1), (3, 1, 8), (100, 1, 8), (1, 32, 1), (100, 32, 1), (7, 5, 3), (500, 8, 4)):
            assert 1 <= prefix_splits(B, Hkv * rep, Hkv, prefix, 64) <= min(296, -(-prefix // 64))


def test_python_api_refuses_cpu_tensors():
    import torch
    from spec_mcts_b200 import kernels as K
    with pytest.raises(K.Q40Error):
        K.quantize_q40(torch.zeros(128, dtype=torch.float16), 64)
    with pytest.raises(K.Q40Error):
        K.matmul_q40(torch.zeros((1, 128), dtype=torch.float16), torch.zeros((128, 64), dtype=torch.int8),
                     torch.zeros((256, 1), dtype=torch.float16), (128, 128))


def test_new_entry_points_check_their_arguments():
    """Host-side checks of the entries added for the wide matmul, the prompt pass and tensor parallelism: every
    refusal comes back as a status code before anything is enqueued."""
    from spec_mcts_b200._lib import lib
    buf = ctypes.create_string_buffer(8192)
    p16 = (ctypes.addressof(buf) + 255) // 256 * 256
    P1 = ctypes.c_void_p * 1
    one64, one32 = (ctypes.c_int64 * 1)(512), (ctypes.c_int * 1)(512)
    # tiled tensor-core matmul: K % 64, N % 256, NULL error word
    assert lib.q40_gemm_tiled_tc_multi(1, p16, 100, P1(p16), P1(p16), one64, one32, 20, 100, p16, 0, None) == -2
    bad_n = (ctypes.c_int * 1)(384)
    assert lib.q40_gemm_tiled_tc_multi(1, p16, 128, P1(p16), P1(p16), one64, bad_n, 20, 128, p16, 0, None) == -2
    assert lib.q40_gemm_tiled_tc_multi(1, p16, 128, P1(p16), P1(p16), one64, one32, 20, 128, None, 0, None) == -1
    assert lib.q40_gemm_tiled_tc_multi(4, p16, 128, P1(p16), P1(p16), one64, one32, 20, 128, p16, 0, None) == -5
    # one projection on its tiled copy: no rows, K % 16 and cluster size (up to 16 rows), K % 64, N % 256, NULL error
    # word, output pitch (above)
    mm = lambda M, N, Kd, ldc=512, cluster=16, err=p16: lib.q40_matmul_tiled(p16, p16, ldc, p16, 128, M, N, Kd, cluster, err, 0, None)
    assert mm(0, 512, 128) == -2 and mm(16, 512, 120) == -2 and mm(16, 384, 128) == -2
    assert mm(16, 512, 128, cluster=4) == -5
    assert mm(17, 512, 80) == -2 and mm(17, 384, 128) == -2 and mm(17, 512, 128, ldc=256) == -2
    assert mm(17, 512, 128, err=None) == -1
    assert lib.q40_matmul_tiled(None, p16, 512, p16, 128, 17, 512, 128, 16, p16, 0, None) == -1
    assert lib.q40_matmul_tiled(p16, p16, 512, p16 + 2, 128, 4, 512, 128, 16, None, 0, None) == -3
    # causal attention: head dim, H % Hkv, row strides
    assert lib.q40_attn_causal(p16, 256, p16, 256, p16, 256, p16, 256, 4, 2, 2, 64, None) == -5
    assert lib.q40_attn_causal(p16, 384, p16, 256, p16, 256, p16, 384, 4, 3, 2, 128, None) == -2
    assert lib.q40_attn_causal(p16, 128, p16, 256, p16, 256, p16, 256, 4, 2, 2, 128, None) == -2
    assert lib.q40_attn_causal(p16, 256, p16, 256, p16, 256, p16, 256, 0, 2, 2, 128, None) == 0      # nothing to do
    # tensor-parallel buffers: layout is pure host arithmetic
    out = (ctypes.c_size_t * 2)()
    assert lib.q40_tp_layout(8, 64, 8192, out) == 0
    assert out[0] == 256 and out[1] == 256 + 2 * 8 * 64 * 8192 * 4
    assert lib.q40_tp_layout(0, 64, 8192, out) == -2
    arr = (ctypes.c_void_p * 2)(p16, p16)
    assert lib.q40_tp_allreduce_norm(p16, 512, p16, p16, p16, 9, 512, 1e-5, 0, 2, arr, 8, 0, None) == -2     # rows > max
    assert lib.q40_tp_allreduce_norm(p16, 512, p16, p16, None, 4, 512, 1e-5, 0, 2, arr, 8, 0, None) == -1    # norm without xn
    assert lib.q40_tp_allreduce_norm(p16, 512, p16, p16, p16, 4, 512, 1e-5, 2, 2, arr, 8, 0, None) == -2     # rank >= world
    arr3 = (ctypes.c_void_p * 3)(p16, p16, p16)
    assert lib.q40_tp_allreduce_norm(p16, 520, p16, p16, p16, 4, 520, 1e-5, 0, 3, arr3, 8, 0, None) == -2    # slices of whole chunks


def test_concatenated_projection_rule():
    """Transformer._concat_tileable: widths of whole 128-column blocks that add up to whole 256-column spans, same
    K, outputs that are consecutive column ranges of one buffer."""
    import torch
    from spec_mcts_b200.model import LinearQ4_0, Transformer

    def lin(n, k=8192):
        l = LinearQ4_0(k, n, 64)
        l.shape = (n, k)
        return l

    buf = torch.zeros((4, 1280), dtype=torch.float16)
    q, k, v = buf[:, :1024], buf[:, 1024:1152], buf[:, 1152:]
    assert Transformer._concat_tileable([lin(1024), lin(128), lin(128)], [q, k, v])
    assert not Transformer._concat_tileable([lin(1024), lin(128)], [q, k])                       # 1152 is not whole spans
    assert not Transformer._concat_tileable([lin(1024), lin(128), lin(128)], [q, v, k])          # not consecutive
    assert not Transformer._concat_tileable([lin(1024), lin(128), lin(128, 4096)], [q, k, v])    # K differs
    sep = [torch.zeros((4, 1024), dtype=torch.float16), torch.zeros((4, 128), dtype=torch.float16),
           torch.zeros((4, 128), dtype=torch.float16)]
    assert not Transformer._concat_tileable([lin(1024), lin(128), lin(128)], sep)                # separate buffers


@pytest.fixture
def launches(monkeypatch):
    """kernels.py with its device calls faked: a list of (rows, whether the matmul was launched with programmatic
    dependent launch) of the matmul_q40 calls made, on CPU tensors."""
    import torch
    from types import SimpleNamespace
    from spec_mcts_b200 import kernels as K
    calls = []

    def matmul_tiled(bw, c, ldc, a, lda, M, N, Kd, cluster, err, pdl, stream):
        calls.append((M, bool(pdl)))
        return 0

    monkeypatch.setattr(K, "lib", SimpleNamespace(q40_matmul_tiled=matmul_tiled, q40_tiled_bytes=lambda N, Kd: 128))
    monkeypatch.setattr(K, "_need_cuda", lambda *t: torch.device("cpu"))
    monkeypatch.setattr(K, "_stream", lambda dev: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(K, "_recorded_event", lambda dev, st: None, raising=False)
    monkeypatch.setattr(K, "relayout_tiled", lambda w, s, shape: torch.zeros(128, dtype=torch.uint8))
    monkeypatch.setattr(K, "_workspaces", {})
    monkeypatch.setattr(K, "_relayout_cache", {})
    monkeypatch.setattr(K, "_relayout_bytes", [0])
    monkeypatch.setattr(K, "_cluster_sizes", {})
    return K, calls


@pytest.mark.parametrize("rows", [1, 16, 17, 129])
def test_a_matmul_right_behind_its_copy_is_no_dependent_launch(launches, rows):
    """A dependent launch reads weights before it waits for the launch in front of it: not behind the one that writes
    the copy, neither the first time nor when it is made again for weights written in place, or when another weight's
    entry goes away meanwhile."""
    import torch
    K, calls = launches
    Kd, N = 64, 256
    w, s = torch.zeros((Kd * N // 128, 64), dtype=torch.int8), torch.zeros(Kd * N // 64, dtype=torch.float16)
    a = torch.zeros((rows, Kd), dtype=torch.float16)
    run = lambda w=w: K.matmul_q40(a, w, s, (Kd, N))
    run(), run()
    w.add_(1)
    run(), run()
    s.add_(1)
    run(), run()
    other = w.clone()
    run(other)
    relayout = K.relayout_tiled

    def drop_other(*args):
        nonlocal other
        other = None                       # its entry is dropped while this weight's new copy is made
        return relayout(*args)

    K.relayout_tiled = drop_other
    w.add_(1)
    run(), run()
    assert [p for _, p in calls] == [False, True, False, True, False, True, False, False, True]


def test_a_matmul_on_another_stream_waits_for_the_copy(launches, monkeypatch):
    """The copy is written on the stream that first used the weight: another stream waits for it once, by a plain
    launch, and the copy's memory is not given back under it.  A capturing stream cannot wait, and need not: its launches
    stay dependent ones."""
    import torch
    K, calls = launches
    Kd, N = 64, 256
    w, s = torch.zeros((Kd * N // 128, 64), dtype=torch.int8), torch.zeros(Kd * N // 64, dtype=torch.float16)
    a = torch.zeros((20, Kd), dtype=torch.float16)
    stream, capturing, log = [1], [False], []

    class Stream:
        def wait_event(self, e):
            log.append((stream[0], "waits", e))

    class Copy(torch.Tensor):
        def record_stream(self, _):
            log.append((stream[0], "holds"))

    monkeypatch.setattr(K, "_stream", lambda dev: stream[0])
    monkeypatch.setattr(K, "_recorded_event", lambda dev, st: "copied")
    monkeypatch.setattr(K, "relayout_tiled", lambda *args: torch.zeros(128, dtype=torch.uint8).as_subclass(Copy))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: Stream())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    for st, capture in ((1, False), (1, False), (2, False), (2, False), (3, True), (3, True), (3, False), (3, False), (1, False)):
        stream[0], capturing[0] = st, capture
        K.matmul_q40(a, w, s, (Kd, N))
    assert [p for _, p in calls] == [False, True, False, True, True, True, False, True, True]
    assert log == [(2, "waits", "copied"), (2, "holds"), (3, "waits", "copied"), (3, "holds")]


def test_rows_that_need_no_cluster_do_not_choose_its_size(launches, monkeypatch):
    """On a device that schedules clusters of 8 and not of 16: 9 to 16 rows run on a kernel without them, and what they are
    given must not be taken for what the device can do."""
    import torch
    K, _ = launches
    ran = []

    def matmul_tiled(bw, c, ldc, a, lda, M, N, Kd, cluster, err, pdl, stream):
        if M <= 8 and cluster == 16:
            return -5
        ran.append((M, cluster))
        return 0

    monkeypatch.setattr(K.lib, "q40_matmul_tiled", matmul_tiled)
    Kd, N = 64, 256
    w, s = torch.zeros((Kd * N // 128, 64), dtype=torch.int8), torch.zeros(Kd * N // 64, dtype=torch.float16)
    for rows in (10, 1, 16, 8):
        K.matmul_q40(torch.zeros((rows, Kd), dtype=torch.float16), w, s, (Kd, N))
    assert [M for M, _ in ran] == [10, 1, 16, 8] and ran[1][1] == ran[3][1] == 8


@pytest.mark.parametrize("dev", ["cuda", "cuda:1"])
def test_scratch_of_an_expired_wait_is_reset_on_an_idle_device(monkeypatch, dev):
    """Of every stream of that device, named with an index or without one, and only while nothing uses it."""
    import torch
    from spec_mcts_b200 import kernels as K
    here, there = (torch.ones(64, dtype=torch.uint8) for _ in range(2))
    monkeypatch.setattr(K, "_workspaces", {("tiled_tc", 1, 7): here, ("tiled_tc", 0, 7): there})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    waits = []
    monkeypatch.setattr(torch.cuda, "synchronize", lambda d=None: waits.append((torch.device(d).index, bool(here.any()))))
    K._reset_tiled_tc_workspaces(torch.device(dev))
    assert not here.any() and there.all() and waits == [(1, True), (1, False)]


def test_scratch_made_in_a_capture_is_not_kept(launches, monkeypatch):
    """It holds nothing until that graph runs: launches of one capture share it, and neither another capture on the stream
    nor a call after the capture finds it.  Scratch that was there before serves captures too."""
    import torch
    K, _ = launches
    capture = [0]

    def capture_id(st, out):
        out._obj.value = capture[0]
        return 0

    monkeypatch.setattr(K.lib, "q40_capture_id", capture_id, raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capture[0] != 0)
    monkeypatch.setattr(K, "_capture_workspaces", {}, raising=False)
    cpu, stream = torch.device("cpu"), [1]
    monkeypatch.setattr(K, "_stream", lambda dev: stream[0])
    get = lambda n=4096: K._workspace("gemm", cpu, n, zero=True)
    # a matmul of 9 to 16 rows (or more) passes an error word of that scratch
    Kd, N = 64, 256
    w, s = torch.zeros((Kd * N // 128, 64), dtype=torch.int8), torch.zeros(Kd * N // 64, dtype=torch.float16)
    for rows in (10, 20):
        K.matmul_q40(torch.zeros((rows, Kd), dtype=torch.float16), w, s, (Kd, N))
    kept = get()
    stream[0], capture[0] = 2, 7
    for rows in (10, 20):
        K.matmul_q40(torch.zeros((rows, Kd), dtype=torch.float16), w, s, (Kd, N))
    first, large = get(), get(3 << 20)
    assert get() is large and large is not first
    capture[0] = 8
    second = get()
    assert second is not large and second is not first and not second.any()
    capture[0] = 0
    after = get()
    assert all(after is not b for b in (first, large, second)) and get() is after
    capture[0] = 9
    assert get() is after
    stream[0] = 1
    assert get() is kept


def test_outgrown_scratch_is_not_given_back(launches, monkeypatch):
    """A graph may have its address.  Sizes at least double, so that what is held stays below the last one's size."""
    import torch
    import weakref
    K, _ = launches
    monkeypatch.setattr(K, "_outgrown", [], raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    get = lambda n: K._workspace("gemm", torch.device("cpu"), n, zero=True)
    seen = []
    for n in (4096, 2 << 20, (2 << 20) + 1, 3 << 20, 40 << 20, (40 << 20) + 1):
        buf = get(n)
        assert buf.numel() >= n and get(n) is buf and not buf.any()
        if not seen or seen[-1]() is not buf:
            seen.append(weakref.ref(buf))
        del buf
    sizes = [r().numel() for r in seen]
    assert sum(sizes[:-1]) <= sizes[-1] and len(sizes) == 5
    # beyond what is always held: given back, unless a capture has used it
    capturing = [False]
    monkeypatch.setattr(K, "_SMALL_WORKSPACE", 1 << 20)
    monkeypatch.setattr(K, "_large_in_graphs", set())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    for used, n in ((False, 81 << 20), (True, 82 << 20), (False, 83 << 20)):
        old = seen[-1]
        capturing[0] = used
        get(4096)
        capturing[0] = False
        seen.append(weakref.ref(get(n)))
        assert (old() is not None) == used and seen[-1]().numel() == n


@pytest.mark.parametrize("dev", [None, "cuda", "cuda:1"])
def test_status_calls_take_a_device_without_an_index(monkeypatch, dev):
    """torch.device("cuda") is the current device."""
    import torch
    from spec_mcts_b200 import kernels as K

    def raw_stream(index):
        if not isinstance(index, int):
            raise TypeError("an index is required")
        return 7

    words = torch.zeros(4096, dtype=torch.uint8)
    words.view(torch.int32)[-1], words.view(torch.int32)[0] = 3, 5
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", raw_stream, raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    monkeypatch.setattr(K, "_workspaces", {("gemm", 1, 7): words, ("stream", 1, 7): words})
    dev = None if dev is None else torch.device(dev)
    assert K.tc_error_flag(dev) == 3 and K.stream_status(dev) == 5
