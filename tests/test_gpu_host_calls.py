"""The native call of a repeated matmul_q40 or linear_q40: what it takes gives the bits of the general way, what is not the plain repeated
call goes that way, with its results and errors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import kernels
    return kernels


def data(K, M=3, Kd=256, N=512, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, s = K.quantize_q40((torch.randn((Kd, N), generator=g, device="cuda") * 0.05).half())
    return torch.randn((M, Kd), generator=g, device="cuda").half(), q, s, (Kd, N)


def count(monkeypatch, K):
    """How many of the calls the native way took."""
    import types
    taken = []
    real = K._host_calls

    def through(name):
        def call(*a):
            r = getattr(real, name)(*a)
            taken.append(r is not None)
            return r
        return call

    monkeypatch.setattr(K, "_host_calls", types.SimpleNamespace(matmul=through("matmul"), linear=through("linear")))
    return taken


@pytest.mark.parametrize("M", [1, 8, 9, 40, 130])
def test_matmul(K, monkeypatch, M):
    a, q, s, shape = data(K, M)
    first = K.matmul_q40(a, q, s, shape)
    K.matmul_q40(a[:1].contiguous(), q, s, shape)          # the cluster size is known from a call of few rows
    out = torch.empty_like(first)
    want = K.matmul_q40(a, q, s, shape, out=out).clone()   # the general way
    taken = count(monkeypatch, K)
    got = K.matmul_q40(a, q, s, shape)
    assert taken == [True] and torch.equal(got, want) and torch.equal(first, want)
    # a parameter, and inference tensors, are tensors; another stream waits for the copy once; written weights are copied again
    with torch.inference_mode():
        assert torch.equal(K.matmul_q40(torch.nn.Parameter(a, requires_grad=False), q, s, shape), want) and taken == [True, True]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        outs = [K.matmul_q40(a, q, s, shape) for _ in range(3)]
    side.synchronize()
    assert taken[2:3] == [False] and taken[-1] and all(torch.equal(o, want) for o in outs)
    del taken[:]
    s.mul_(2)
    again = K.matmul_q40(a, q, s, shape)
    assert taken == [False] and torch.allclose(again.float(), 2 * want.float(), rtol=2e-3, atol=1e-3)
    assert torch.equal(K.matmul_q40(a, q, s, shape), again) and taken[-1]


def test_what_matmul_hands_back(K, monkeypatch):
    a, q, s, shape = data(K)
    want = K.matmul_q40(a, q, s, shape)
    taken = count(monkeypatch, K)
    assert torch.equal(K.matmul_q40(a, q, s, torch.tensor(shape)), want)          # a shape that is no tuple
    wide = torch.zeros((3, 512), device="cuda", dtype=torch.float16)
    wide[:, 1:257] = a
    with pytest.raises(K.Q40Error):                                               # rows off a 16-byte boundary
        K.matmul_q40(wide.view(-1)[1:769].view(3, 256), q, s, shape)
    with pytest.raises(AssertionError):
        K.matmul_q40(wide[:, 1:257], q, s, shape)
    with pytest.raises(AssertionError):
        K.matmul_q40(a[:, :128].contiguous(), q, s, shape)
    with pytest.raises(K.Q40Error):
        K.matmul_q40(a.float(), q, s, shape)
    with pytest.raises(K.Q40Error):
        K.matmul_q40(a.cpu(), q, s, shape)
    assert K.matmul_q40(a[:0], q, s, shape).shape == (0, 512)
    assert not any(taken)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        c = K.matmul_q40(a, q, s, shape)
    g.replay()
    assert torch.equal(c, want)


@pytest.mark.parametrize("M,group", [(1, 64), (10, 64), (33, 64), (10, 32)])
def test_linear(K, monkeypatch, M, group):
    g = torch.Generator(device="cuda").manual_seed(M)
    q, s = K.quantize_q40((torch.randn((300, 512), generator=g, device="cuda") * 0.05).half(), group)
    x = torch.randn((M, 512), generator=g, device="cuda").half()
    want = K.linear_q40(x.view(1, M, 512), q, s, (300, 512), group_size=group)       # three dimensions: the general way
    taken = count(monkeypatch, K)
    assert torch.equal(K.linear_q40(x, q, s, (300, 512), group_size=group), want[0]) and taken == [True]
    strided = torch.zeros((M, 600), device="cuda", dtype=torch.float16)[:, :512].copy_(x)
    assert torch.equal(K.linear_q40(strided, q, s, (300, 512), group_size=group), want[0]) and taken == [True, M == 1]    # one row is contiguous
    with pytest.raises(K.Q40Error):
        K.linear_q40(x.float(), q, s, (300, 512), group_size=group)
    with pytest.raises(K.Q40Error):
        K.linear_q40(x, q, s, (300, 512), group_size=48)
    assert K.linear_q40(x[:0], q, s, (300, 512), group_size=group).shape == (0, 300)


def test_interpreter_is_free_meanwhile(K, monkeypatch):
    """In the place of the library's functions, one that returns 0 if the thread does not hold the interpreter's lock."""
    import ctypes
    a, q, s, shape = data(K)
    K.matmul_q40(a, q, s, shape)
    y = K.linear_q40(a, q, s, (512, 256))
    taken = count(monkeypatch, K)
    from spec_mcts_b200 import _host_calls
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value
    try:
        _host_calls.init(*[address(ctypes.pythonapi.PyGILState_Check)] * 2)
        K.matmul_q40(a, q, s, shape)
        K.linear_q40(a, q, s, (512, 256))
    finally:
        _host_calls.init(address(K.lib.q40_matmul_tiled), address(K.lib.q40_gemm_nk))
    assert taken == [True, True]
    assert torch.equal(K.linear_q40(a, q, s, (512, 256)), y)


def test_without_the_extension(K, monkeypatch):
    a, q, s, shape = data(K, 9)
    K.matmul_q40(a[:1].contiguous(), q, s, shape)
    K.matmul_q40(a, q, s, shape)
    c, y = K.matmul_q40(a, q, s, shape), K.linear_q40(a, q, s, (512, 256))
    monkeypatch.setattr(K, "_host_calls", None)
    assert torch.equal(K.matmul_q40(a, q, s, shape), c) and torch.equal(K.linear_q40(a, q, s, (512, 256)), y)


@pytest.mark.parametrize("op,M", [("matmul_q40", 1), ("matmul_q40", 9), ("matmul_q40", 40), ("matmul_q40", 130), ("linear_q40", 1), ("linear_q40", 40), ("linear_q40", 300)])
def test_the_first_call_of_a_thread_is_like_any_other(K, op, M):
    """A thread that has made no call of the CUDA runtime gets the bits, and so the route, of the others."""
    import threading
    a, q, s, shape = data(K, M, 4096, 4096)
    for _ in range(2):                                        # the copy is made, the output's memory is there
        want = getattr(K, op)(a, q, s, shape)
    got = []
    t = threading.Thread(target=lambda: got.append(getattr(K, op)(a, q, s, shape)))
    t.start()
    t.join()
    assert got and torch.equal(got[0], want)
