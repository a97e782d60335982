"""A prompt pass whose layers are enqueued by one native call, against the same launches made one by one: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,S", [(8, None, 17), (8, 4, 65), (4, 2, 128), (8, 8, 129), (6, None, 40)])
def test_same_bits_as_the_launches_one_by_one(heads, kv, S, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200 import model as M
    m = M.Transformer(M.ModelArgs(dim=heads * 128, n_layers=3, n_heads=heads, n_kv_heads=kv, vocab_size=1000, multiple_of=256, max_batch_size=2,
                                  max_seq_len=16, max_prompt_seq_len=136))
    M.random_init_(m, seed=5, std=0.03)
    toks = [torch.randint(0, 1000, (1, s), generator=torch.Generator().manual_seed(s)).cuda() for s in (S, S + 1)]
    calls = []
    real = M.lib.q40_prompt_layers

    class Lib:
        def __getattr__(self, name):
            return (lambda *a: calls.append(1) or real(*a)) if name == "q40_prompt_layers" else getattr(lib, name)

    lib = M.lib
    monkeypatch.setattr(M, "lib", Lib())
    state = lambda: [m._caches[c][:, :S].clone() for c in ("pk", "pv")]
    native = [(m(t, 0).clone(), *state()) for t in toks]
    assert len(calls) == 2                                           # more than 16 tokens, copies of all projections
    lengths = [l.attention.cache_prompt_len for l in m.layers]
    assert lengths == [S + 1] * 3 and int(m._prefix_len_dev) == S + 1 and m.prompt_status() == 0
    monkeypatch.setattr(m, "_prompt_table", lambda plan: None)
    one_by_one = [(m(t, 0).clone(), *state()) for t in toks]
    assert len(calls) == 2
    for x, y in zip(native, one_by_one):
        assert all(torch.equal(a, b) for a, b in zip(x, y))
    # an assigned weight is multiplied by the next pass
    monkeypatch.undo()
    ff = m.layers[1].feed_forward
    ff.w1.w = ff.w1.w.flip(0).contiguous()
    new = m(toks[0], 0).clone()
    monkeypatch.setattr(m, "_prompt_table", lambda plan: None)
    assert torch.equal(new, m(toks[0], 0)) and not torch.equal(new, native[0][0])


def test_refusals():
    from spec_mcts_b200._lib import lib
    p = 4096
    args = lambda **c: [c.get(k, d) for k, d in (("layers", p), ("n", 0), ("S", 20), ("dim", 256), ("hid", 512), ("H", 2), ("Hkv", 2), ("eps", 1e-5), ("h", p), ("xn", p),
                        ("q", p), ("ao", p), ("o", p), ("g", p), ("f", p), ("pos", p), ("cos", p), ("sin", p), ("ws", p), ("wsb", 1 << 20), ("err", p), ("pdl", 1), ("st", None))]
    assert lib.q40_prompt_layers(*args()) == 0                       # no layer: nothing is read
    for k in ("layers", "h", "xn", "q", "ao", "o", "g", "f", "pos", "cos", "sin", "err"):
        assert lib.q40_prompt_layers(*args(**{k: None})) == -1
    assert lib.q40_prompt_layers(*args(S=0)) == -2 and lib.q40_prompt_layers(*args(n=-1)) == -2 and lib.q40_prompt_layers(*args(Hkv=3)) == -2
