"""Decode steps of 5 to 8 branches of a model with wide layers: tensor-core matmuls on the tiled copies, then the library's own lm_head."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def model(dim=2048, layers=2, max_b=9):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200.model import ModelArgs, Transformer, random_init_
    m = Transformer(ModelArgs(dim=dim, n_layers=layers, n_heads=dim // 128, n_kv_heads=4 if dim % 512 == 0 else None, vocab_size=1000, multiple_of=256, max_batch_size=max_b,
                              max_seq_len=32, max_prompt_seq_len=64))
    random_init_(m, seed=11, std=0.03)
    m(tokens(1, 1, 21), 0)
    return m


def tokens(seed, *shape):
    return torch.randint(0, 1000, shape, generator=torch.Generator().manual_seed(seed)).cuda()


class Counted:
    """The library, with the names of the calls made through it."""
    def __init__(self, lib):
        self._lib, self.names = lib, []

    def __getattr__(self, name):
        self.names.append(name)
        return getattr(self._lib, name)


@pytest.mark.parametrize("B", [5, 8])
@pytest.mark.parametrize("feedback", [False, True])
def test_against_checkpoint_layout(B, feedback, monkeypatch):
    """The same steps by the narrow matmuls on the checkpoint layout.  Operands there are fp16(code * scale) too; sums, and the norms' sums of squares,
    are in another order: activations differ by an fp16 step here and there (the model tests' tolerance)."""
    from spec_mcts_b200 import model as M
    m = model()
    m.use_cuda_graph = False
    m.greedy_feedback = feedback
    runs = {}
    for tiled in (True, False):
        m.use_tiled = tiled
        counted = Counted(m_lib := M.lib)
        monkeypatch.setattr(M, "lib", counted)
        toks, outs = tokens(2, B, 1), []
        for step in range(3):
            outs.append(m(toks, 21 + step).float().view(B, -1).clone())
            if feedback:
                assert torch.equal(m._tok_dev[:B], outs[-1].argmax(-1)) and (m._pos_dev[:B] == 22 + step).all()
            toks = tokens(3 + step, B, 1)                # not what was generated: one logit's last bit would decide what follows
        monkeypatch.setattr(M, "lib", m_lib)
        assert counted.names.count("q40_lm_head") == 3
        assert ("q40_gemm_tiled_tc_multi" in counted.names) == tiled
        launches = [n for n in counted.names if n not in ("q40_lm_head_scratch_bytes", "q40_gemm_tiled_tc_ws_bytes", "q40_decode_chain_ws_bytes",
                                                          "q40_gemv_fused_ss_count", "q40_attn_shared_prefix_workspace_bytes", "q40_gemm_workspace_bytes")]
        assert not tiled or len(launches) + launches.count("q40_attn_tree_step") == 3 * m.launches_per_step      # that call is two launches
        runs[tiled] = outs
    for a, b in zip(runs[True], runs[False]):
        torch.testing.assert_close(a, b, rtol=2e-2, atol=0.05)
        assert ((a - b).norm() / b.norm()).item() < 1e-2
    assert m.decode_status() == 0


@pytest.mark.parametrize("graph", [False, True])
def test_ties_and_tail_switch(graph):
    """Of equal logits the smaller index is the next token; without the fused tail, torch's product of the same rows gives the same logits to an fp16 step."""
    m = model()
    m.use_cuda_graph = graph
    with torch.no_grad():
        m.output.weight[500:1000] = m.output.weight[:500]
    m.greedy_feedback = True
    toks = tokens(5, 8, 1)
    a = m(toks, 21).float().view(8, -1).clone()
    assert torch.equal(a[:, :500], a[:, 500:]) and torch.equal(m._tok_dev[:8], a[:, :500].argmax(-1))
    m.use_fused_tail = False
    b = m(toks, 21).float().view(8, -1)
    assert ((a - b).norm() / b.norm()).item() < 1e-3


def test_switches_choose_among_captured_steps():
    """A graph is replayed for the switches that it was captured with, and the launches that are reported are its own."""
    m = model(dim=2304, layers=2, max_b=6)              # 18 heads: one launch for all layers at widths 1 and 2
    toks = tokens(7, 1, 1)
    seen = {}
    for chain in (True, False, True, False):
        m.use_chain = chain
        out = m(toks, 21).clone()
        assert m._chained[1] == chain
        assert seen.setdefault(chain, m.launches_per_step) == m.launches_per_step and torch.equal(seen.setdefault(("out", chain), out), out)
    assert seen[True] == 2 < seen[False]
    m.use_chain = True
    m(toks, 21)
    m.use_fused = False                                 # the launch-per-operation body, at a width that has just been one launch
    m(toks, 21)
    assert m.launches_per_step > 2 and not m._chained[1]
    m.use_fused = True
    toks, counts = tokens(8, 5, 1), {}
    for most in (4, 8, 4):
        m.narrow_max = most
        m(toks, 21)
        assert counts.setdefault(most, m.launches_per_step) == m.launches_per_step
    assert counts[4] == 2 * 8 + 3 and counts[8] == 2 * 6 + 2
