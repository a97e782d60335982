"""All layers of a narrow step as one launch (q40_decode_chain) against the numpy model oracle and against the same step as a chain
of launches."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def model(dim=4096, layers=1, heads=32, kv_heads=None, vocab=512, max_b=2, max_t=256, max_p=512, seed=5, multiple_of=256):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200.model import ModelArgs, Transformer, random_init_
    m = Transformer(ModelArgs(dim=dim, n_layers=layers, n_heads=heads, n_kv_heads=kv_heads, vocab_size=vocab, multiple_of=multiple_of,
                              max_batch_size=max_b, max_seq_len=max_t, max_prompt_seq_len=max_p))
    random_init_(m, seed=seed, std=0.03)
    return m


def tokens(seed, *shape):
    return torch.randint(0, 512, shape, generator=torch.Generator().manual_seed(seed)).cuda()


def fill_suffix(m, B, t):
    """Random rows in the first t positions of every branch."""
    from spec_mcts_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(9)
    for layer in m.layers if t else ():
        att = layer.attention
        for codes, scales in ((att.cache_k, att.cache_k_s), (att.cache_v, att.cache_v_s)):
            q, s = K.quantize_q40(torch.randn((B * t, codes.shape[2] * 128), generator=g, device="cuda").half())
            codes[:B, :t] = q.view(B, t, *codes.shape[2:])
            scales[:B, :t] = s.view(B, t, *scales.shape[2:])


@pytest.mark.parametrize("B,kv_heads", [(1, 18), (1, 2), (2, 18), (2, 2)])
def test_against_model_oracle(B, kv_heads):
    """Several steps at a width whose groups do not divide evenly over clusters (36 of wo and w2), the oracle's suffix replaced by
    the rows that the step wrote: logits within the model tests' tolerance."""
    from oracle import model_oracle as MO
    from oracle import q40_oracle as O
    m = model(dim=2304, layers=2, heads=18, kv_heads=kv_heads, max_t=16, max_p=32)
    hid = m.layers[0].feed_forward.hidden_dim
    orc = MO.ModelOracle(2304, 2, 18, kv_heads, 512, hid, 1e-5, 1e6, 2, 16, 32)
    n = lambda t: t.detach().cpu().numpy()
    orc.emb, orc.out, orc.norm["norm"] = n(m.tok_embeddings.weight), n(m.output.weight), n(m.norm.weight)
    for i, layer in enumerate(m.layers):
        orc.norm[f"layers.{i}.attention_norm"], orc.norm[f"layers.{i}.ffn_norm"] = n(layer.attention_norm.weight), n(layer.ffn_norm.weight)
        for name in ("attention.wq", "attention.wk", "attention.wv", "attention.wo", "feed_forward.w1", "feed_forward.w2", "feed_forward.w3"):
            lin = layer.get_submodule(name)
            orc.w[f"layers.{i}.{name}"] = (n(lin.w), n(lin.s), lin.kn())
    prompt = tokens(1, 1, 9)
    m(prompt, 0)
    orc.forward(n(prompt), 0)
    for l in range(2):              # the same prompt rows on both sides
        orc.pk[l], orc.pv[l] = n(m._caches["pk"][l, :9]), n(m._caches["pv"][l, :9])
    toks, C = n(tokens(2, B, 1)), m._caches
    for step in range(3):
        got = n(m(torch.from_numpy(toks).cuda(), 9 + step)[:, -1].float())
        assert m._chained[B] and m.launches_per_step == 2
        np.testing.assert_allclose(got, orc.forward(toks, 9 + step)[:, 0].astype(np.float32), rtol=2e-2, atol=0.15)
        for l in range(2):
            for b in range(B):
                for cache, k in ((orc.sk, "k"), (orc.sv, "v")):
                    cache[l][b][step] = O.dequantize_q40(n(C[k + "q"][l, b, step]), n(C[k + "s"][l, b, step]).reshape(-1, 1), 64, (kv_heads, 128))
        toks = got.argmax(-1).reshape(B, 1)
    assert m.decode_status() == 0


# keys at the ends of a half warp's batch (512 prompt keys and 128 suffix rows of a cluster), none of one kind, the last slot
@pytest.mark.parametrize("B,prompt,suffix,kv_heads", [(1, 1, 0, 32), (1, 512, 64, 32), (1, 513, 127, 32), (1, 31, 128, 8), (1, 511, 255, 32),
                                                      (2, 512, 1, 32), (2, 77, 130, 8), (2, 640, 255, 32)])
def test_against_launches(B, prompt, suffix, kv_heads):
    """One layer of the 7B shapes.  Both paths round activations at the same points; matmul operands differ by 2^-12 at most (the
    launches round scale * x to fp16), so do sums, and a code of the appended row may be its neighbour."""
    m = model(kv_heads=kv_heads, max_p=640)
    m(tokens(3, 1, prompt), 0)
    fill_suffix(m, B, suffix)
    toks, out = tokens(4, B, 1), {}
    for chain in (False, True):
        m.use_chain = chain
        logits = m(toks, prompt + suffix).float().clone()
        assert m._chained[B] == chain
        out[chain] = [logits] + [m._caches[k][0, :B, suffix].clone() for k in ("kq", "vq", "ks", "vs")]
    (l0, kq0, vq0, ks0, vs0), (l1, kq1, vq1, ks1, vs1) = out[False], out[True]
    assert ((l0 - l1).norm() / l0.norm()).item() < 5e-3
    for a, b in ((kq0, kq1), (vq0, vq1)):
        nib = lambda x: torch.stack(((x >> 4), ((x << 4) >> 4))).int()
        assert (nib(a) - nib(b)).abs().max() <= 1 and (a != b).float().mean() < 0.03
    for a, b in ((ks0, ks1), (vs0, vs1)):
        torch.testing.assert_close(a, b, rtol=4e-3, atol=0)
    assert all(torch.equal(m(toks, prompt + suffix).float(), l1) for _ in range(3))        # the same bits every time
    assert m.decode_status() == 0


def test_rows_that_are_not_finite():
    """An infinity in a branch's residual stream makes its logits NaN, as in the chain of launches, and leaves the other's alone."""
    m = model()
    m(tokens(3, 1, 20), 0)
    toks = torch.tensor([[7], [11]], device="cuda")
    clean = m(toks, 20).clone()
    m.tok_embeddings.weight.data[7, 100] = float("inf")
    for chain in (True, False):
        m.use_chain = chain
        out = m(toks, 20)
        assert torch.isnan(out[0]).all()
        if chain:
            assert torch.equal(out[1], clean[1])


def test_two_streams():
    """Steps of two models on two streams: the bits that each gives alone."""
    ms = [model(layers=3, seed=s) for s in (5, 6)]
    want, streams = [], [torch.cuda.Stream() for _ in ms]
    for m in ms:
        m(tokens(3, 1, 40), 0)
        want.append(m(tokens(4, 1, 1), 40).clone())
    torch.cuda.synchronize()
    for _ in range(20):
        for m, s in zip(ms, streams):
            with torch.cuda.stream(s):
                m.decode_replay(1)
    torch.cuda.synchronize()
    for m, w in zip(ms, want):
        assert torch.equal(m._bufs[1]["logits"].view(-1), w.view(-1)) and m.decode_status() == 0


def test_sizes_that_it_does_not_take():
    """Too few column groups, too wide, an odd kv width: the chain of launches, and no scratch is offered."""
    from spec_mcts_b200._lib import lib
    m = model(dim=512, heads=4, max_p=32)
    m(tokens(3, 1, 20), 0)
    assert torch.isfinite(m(tokens(4, 1, 1), 20)).all() and not m._chained[1] and m.launches_per_step > 2
    for B, dim, hid, H, Hkv in [(1, 8192, 28672, 64, 8), (3, 4096, 11008, 32, 32), (1, 4096, 11008, 32, 1), (1, 4096, 11000, 32, 32)]:
        assert lib.q40_decode_chain_ws_bytes(B, 32, dim, hid, H, Hkv) == 0
    assert lib.q40_decode_chain_ws_bytes(1, 32, 4096, 11008, 32, 32) > 0


def test_sizes_that_leave_warps_without_work():
    """Fewer 32-row pairs of a matmul in a cluster than it has warps: wo with one 64-column group of 6 to 14 pairs.  Not taken: sums over
    warps would read slabs that nobody wrote.  One with 16 pairs or more is."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spec_mcts_b200._lib import lib
    for H, Hkv in [(14, 14), (14, 2), (6, 6), (12, 12)]:
        assert lib.q40_decode_chain_ws_bytes(1, 2, 2304, 6144, H, Hkv) == 0
    assert lib.q40_decode_chain_ws_bytes(1, 2, 2304, 6144, 16, 16) > 0


def test_table_outlives_released_graphs():
    """A graph that the caller captured reads the table of the layers' addresses: it goes with the tiled copies, not with the model's own graphs."""
    m = model(layers=2)
    m.use_cuda_graph = False
    m(tokens(3, 1, 40), 0)
    toks = tokens(4, 1, 1)
    want = m(toks, 40).clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.decode_replay(1)
    assert m._chained[1]
    (table,) = m._chain_tables.values()
    m.release_graphs()
    assert next(iter(m._chain_tables.values())) is table
    with torch.inference_mode():
        m._bufs[1]["logits"].zero_()
    g.replay()
    assert torch.equal(m._bufs[1]["logits"].view(-1), want.view(-1))
    del g
    m.drop_tiled_copies()
    assert not m._chain_tables
    assert torch.equal(m(toks, 40), want)


def test_prompt_caches_with_strides():
    """Prompt caches that are views of something wider, head by head: the launches take their strides, the one launch leaves them to those."""
    m = model(layers=2, kv_heads=8)
    m(tokens(3, 1, 40), 0)
    toks = tokens(4, 2, 1)
    want = m(toks, 40).float()
    assert m._chained[2]
    for layer in m.layers:
        att = layer.attention
        for name in ("cache_prompt_k", "cache_prompt_v"):
            old = getattr(att, name)
            wide = torch.full((old.shape[1], old.shape[0] + 3, 128), float("nan"), dtype=old.dtype, device="cuda")
            wide[:, :old.shape[0]] = old.transpose(0, 1)
            setattr(att, name, wide[:, :old.shape[0]].transpose(0, 1))
    m.release_graphs()
    got = m(toks, 40).float()
    assert not m._chained[2] and ((got - want).norm() / want.norm()).item() < 5e-3


def layer64(m, tok, pos):
    """One layer's step of one branch without own keys, sums and weights in 64 bits, activations rounded where the reference rounds them."""
    from spec_mcts_b200 import kernels as K
    layer, S = m.layers[0], int(m._prefix_len_dev)
    att, ff, H = layer.attention, layer.feed_forward, m._H

    def lin(x, l):
        q = l.w.reshape(-1, 64)
        w = torch.cat((q >> 4, (q << 4) >> 4), 1).view(-1, 64).double() * l.s.reshape(-1, 1).double()
        return (x.double() @ w.view(l.kn())).half()

    def norm(h, w):
        return (h.double() * (h.double().square().mean() + m.params.norm_eps).rsqrt()).half() * w

    h = m.tok_embeddings.weight[tok]
    x, p = norm(h, layer.attention_norm.weight), torch.tensor([pos], device="cuda")
    q, k = (K.rope_(lin(x, l).view(1, H, 128), p, m._cos, m._sin)[0] for l in (att.wq, att.wk))
    keys, values = (torch.cat((c[:S], new[None])).double() for c, new in ((att.cache_prompt_k, k), (att.cache_prompt_v, lin(x, att.wv).view(H, 128))))
    w = torch.softmax(torch.einsum("hd,khd->hk", q.double(), keys) / 128 ** 0.5, -1)
    h = h + lin(torch.einsum("hk,khd->hd", w, values).reshape(-1).half(), att.wo)
    x = norm(h, layer.ffn_norm.weight)
    a = lin(x, ff.w1)
    return h + lin((a.double() * torch.sigmoid(a.double())).half() * lin(x, ff.w3), ff.w2)


@pytest.mark.parametrize("ratio", [1, 1000, 10000])
def test_one_activation_far_above_the_rest(ratio):
    """128 activations share an exponent: with one of them `ratio` times the rest, the layer's result in all other columns is no further from 64 bits
    than that of the launches, which round each scale * x to fp16."""
    m = model()
    m(tokens(3, 1, 20), 0)
    with torch.no_grad():
        m.tok_embeddings.weight[7, 100] = 0.03 * ratio
    want = layer64(m, 7, 20).double()
    rest = torch.arange(4096, device="cuda") != 100
    change, errors = (want - m.tok_embeddings.weight[7].double())[rest].norm(), {}
    for chain in (False, True):
        m.use_chain = chain
        m(torch.tensor([[7]], device="cuda"), 20)
        assert m._chained[1] == chain
        errors[chain] = ((m._bufs[1]["h"][0].double() - want)[rest].norm() / change).item()
    assert errors[True] < 1.05 * errors[False] < 5e-3
