"""The workloads this package's speed is judged by, each one pass through its public entry points.

Sizes are those of the 7B architecture the package is written for (dim 4096, 32 layers, 32 heads of 128,
FFN 11008, vocabulary 32016), of the batch widths it is used at (1, 10 and 100 tree branches) and of the
512-token prompts its benchmark takes; `draw` spreads the same kinds of call over the ranges in between.

  decode       one step of `Transformer.forward` for all live branches of a tree: what a search spends its
               time in.  Width 1 is the start of every search and plain greedy decoding, 10 and 100 are a
               narrow and a full tree.
  prompt       the prompt pass of the same model, once per question: a full prompt and a short ragged one.
  matmul       `matmul_q40`, the call a host that keeps its own model code makes for every projection
               (checkpoint layout, groups along the outputs).
  linear       `linear_q40`, the same for weights quantised in memory (groups along the inputs).
  tree_attn    `shared_prefix_attn`: branches that share a long prompt and own paged suffixes.
  branch_attn  `page_flash_attn` / `flash_attn`: branches that share nothing, paged or contiguous.
  pack         `quantize_q40` followed by `dequantize_q40`: converting one projection of a checkpoint and
               expanding it again.

The token tree search itself (`tree.mcts.search`) is not listed: its result is a chain of random draws, in
which one logit's last bit decides all later tokens.  A search is the decode steps above plus a sampling
launch per step.
"""
from __future__ import annotations

import math

import torch

from spec_mcts_b200 import kernels as K
from spec_mcts_b200.model import ModelArgs, Transformer, random_init_

DEV = "cuda"
DIM, LAYERS, HEADS, HEAD_DIM, FFN, VOCAB = 4096, 32, 32, 128, 11008, 32016
MAX_PROMPT, MAX_SUFFIX = 512, 256


def listed():
    return [
        # greedy decoding, or the first steps of a search: weights are streamed for a single row
        {"name": "decode_width1", "kind": "decode", "width": 1, "prompt": 512, "suffix": 64},
        # a narrow tree; an even step further into the answer
        {"name": "decode_width10", "kind": "decode", "width": 10, "prompt": 512, "suffix": 64},
        # a full tree: the largest decode step
        {"name": "decode_width100", "kind": "decode", "width": 100, "prompt": 512, "suffix": 64},
        # the longest prompt of the benchmark's configuration
        {"name": "prompt_512", "kind": "prompt", "prompt": 512},
        # a short question, no multiple of anything
        {"name": "prompt_77", "kind": "prompt", "prompt": 77},
        # the smallest call: one attention projection of one row, where latency and host time count
        {"name": "matmul_attn_m1", "kind": "matmul", "rows": 1, "k": 4096, "n": 4096},
        # the FFN's second projection for a narrow tree: long sums
        {"name": "matmul_w2_m10", "kind": "matmul", "rows": 10, "k": 11008, "n": 4096},
        # the FFN's first projection for a full tree
        {"name": "matmul_w1_m100", "kind": "matmul", "rows": 100, "k": 4096, "n": 11008},
        # in-memory quantised layer (groups along the inputs) for a narrow tree
        {"name": "linear_w1_m10", "kind": "linear", "rows": 10, "k": 4096, "n": 11008, "group": 64},
        # 64 branches over one 2048-token prompt, ragged private suffixes in 16-token pages
        {"name": "tree_attn_64", "kind": "tree_attn", "width": 64, "prompt": 2048, "suffix": 256, "heads": 32,
         "kv_heads": 32, "page": 16},
        # ten independent branches of one pool, token-granular page table
        {"name": "paged_attn_10", "kind": "branch_attn", "width": 10, "keys": 512, "heads": 32, "kv_heads": 32,
         "paged": True},
        # one FFN projection of a checkpoint through the packer and back
        {"name": "pack_w1", "kind": "pack", "rows": 4096, "cols": 11008, "group": 64},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, round(v / step) * step))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "matmul", "matmul", "linear", "tree_attn", "branch_attn", "pack"])
    if kind == "decode":
        return {"kind": kind, "width": _log(rng, 1, 100), "prompt": rng.randint(16, MAX_PROMPT),
                "suffix": rng.randint(1, MAX_SUFFIX - 1)}
    if kind == "prompt":
        return {"kind": kind, "prompt": _log(rng, 16, MAX_PROMPT)}
    if kind == "matmul":
        return {"kind": kind, "rows": _log(rng, 1, 512), "k": _log(rng, 1024, 11008, 64), "n": _log(rng, 1024, 32128, 128)}
    if kind == "linear":
        return {"kind": kind, "rows": _log(rng, 1, 128), "k": _log(rng, 1024, 11008, 128), "n": rng.randint(1000, 11008),
                "group": rng.choice([64, 64, 32])}
    if kind == "tree_attn":
        kv = rng.choice([32, 8])
        return {"kind": kind, "width": _log(rng, 2, 100), "prompt": _log(rng, 64, 2048), "suffix": rng.randint(16, 256),
                "heads": 32, "kv_heads": kv, "page": rng.choice([1, 16])}
    if kind == "branch_attn":
        return {"kind": kind, "width": _log(rng, 1, 100), "keys": _log(rng, 16, 768), "heads": 32,
                "kv_heads": rng.choice([32, 8]), "paged": rng.random() < 0.5}
    return {"kind": kind, "rows": _log(rng, 64, 4096), "cols": _log(rng, 256, 11008, 128), "group": rng.choice([64, 64, 32])}


def _model(gen, width):
    """The 7B architecture with random weights, drawn on the device and packed by the library's packer."""
    m = Transformer(ModelArgs(max_batch_size=width, max_seq_len=MAX_SUFFIX, max_prompt_seq_len=MAX_PROMPT))
    random_init_(m, seed=int(torch.randint(0, 1 << 30, (1,), generator=gen, device=DEV)))
    return m


def _normal(gen, *shape, std=1.0):
    return (torch.randn(shape, generator=gen, device=DEV) * std).to(torch.float16)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    kind = case["kind"]
    if kind == "decode":
        # a model some way into its answer: the prompt has been read, `suffix` tokens of every branch are
        # in the packed cache (random keys and values of about the size that projections give)
        w, t = case["width"], case["suffix"]
        m = _model(gen, w)
        m(torch.randint(0, VOCAB, (1, case["prompt"]), generator=gen, device=DEV), 0)
        for layer in m.layers:
            att = layer.attention
            for codes, scales in ((att.cache_k, att.cache_k_s), (att.cache_v, att.cache_v_s)):
                q, s = K.quantize_q40(_normal(gen, w * t, DIM))
                codes[:w, :t] = q.view(w, t, HEADS, 64)
                scales[:w, :t] = s.view(w, t, HEADS, 2)
        tokens = torch.randint(0, VOCAB, (w, 1), generator=gen, device=DEV)
        return {"kind": kind, "model": m, "tokens": tokens, "pos": case["prompt"] + t}
    if kind == "prompt":
        m = _model(gen, 1)
        return {"kind": kind, "model": m, "tokens": torch.randint(0, VOCAB, (1, case["prompt"]), generator=gen, device=DEV)}
    if kind == "matmul":
        q, s = K.quantize_q40(_normal(gen, case["k"], case["n"], std=0.02))
        return {"kind": kind, "x": _normal(gen, case["rows"], case["k"]), "w": q, "s": s, "shape": (case["k"], case["n"])}
    if kind == "linear":
        q, s = K.quantize_q40(_normal(gen, case["n"], case["k"], std=0.02), case["group"])
        return {"kind": kind, "x": _normal(gen, case["rows"], case["k"]), "w": q, "s": s,
                "shape": (case["n"], case["k"]), "group": case["group"]}
    if kind == "tree_attn":
        b, p, h, hkv, page = case["width"], case["prompt"], case["heads"], case["kv_heads"], case["page"]
        pages = -(-case["suffix"] // page)
        table = torch.randperm(b * pages, generator=gen, device=DEV).to(torch.int32).view(b, pages)
        return {"kind": kind, "q": _normal(gen, b, h, HEAD_DIM), "pk": _normal(gen, p, hkv, HEAD_DIM),
                "pv": _normal(gen, p, hkv, HEAD_DIM), "prompt": p, "table": table, "page": page, "suffix": case["suffix"],
                "lens": torch.randint(0, case["suffix"] + 1, (b,), generator=gen, device=DEV, dtype=torch.int32),
                "k": _normal(gen, hkv, b * pages * page, HEAD_DIM), "v": _normal(gen, hkv, b * pages * page, HEAD_DIM)}
    if kind == "branch_attn":
        b, n, h, hkv = case["width"], case["keys"], case["heads"], case["kv_heads"]
        st = {"kind": kind, "q": _normal(gen, b, h, HEAD_DIM), "dims": (b, n, h, HEAD_DIM), "paged": case["paged"]}
        if case["paged"]:
            # branches that grew from a common root hold runs of the same slots: a pool of half the rows
            slots = min(32767, max(n, b * n // 2))
            st["table"] = torch.randint(0, slots, (b, n), generator=gen, device=DEV, dtype=torch.int16)
            st["slots"] = slots
            st["k"], st["v"] = _normal(gen, hkv, slots, HEAD_DIM), _normal(gen, hkv, slots, HEAD_DIM)
        else:
            st["k"], st["v"] = _normal(gen, b, hkv, n, HEAD_DIM), _normal(gen, b, hkv, n, HEAD_DIM)
        return st
    return {"kind": kind, "w": _normal(gen, case["rows"], case["cols"], std=0.02), "group": case["group"]}


def run(state):
    kind = state["kind"]
    if kind == "decode":
        m = state["model"]
        logits = m(state["tokens"], state["pos"])
        c = m._caches          # the step appended one packed row per branch, layer and head
        return {"logits": logits, "k": c["kq"], "k_scale": c["ks"], "v": c["vq"], "v_scale": c["vs"]}
    if kind == "prompt":
        m = state["model"]
        logits = m(state["tokens"], 0)
        return {"logits": logits, "k": m._caches["pk"], "v": m._caches["pv"]}
    if kind == "matmul":
        return K.matmul_q40(state["x"], state["w"], state["s"], state["shape"])
    if kind == "linear":
        return K.linear_q40(state["x"], state["w"], state["s"], state["shape"], group_size=state["group"])
    if kind == "tree_attn":
        return K.shared_prefix_attn(state["q"], state["pk"], state["pv"], state["prompt"], state["table"], state["lens"],
                                    state["k"], state["v"], page_size=state["page"], max_suffix=state["suffix"])
    if kind == "branch_attn":
        b, n, h, d = state["dims"]
        if state["paged"]:
            return K.page_flash_attn(state["table"], state["q"], state["k"], state["v"], state["slots"], b, n, h, d)
        return K.flash_attn(state["q"], state["k"], state["v"], b, n, h, d)
    q, s = K.quantize_q40(state["w"], state["group"])
    return {"codes": q, "scales": s, "back": K.dequantize_q40(q, s, state["group"], state["w"].shape)}


def _q40_bytes(n, group=64):
    return n // 2 + 2 * (n // group)


PROJECTIONS = 4 * DIM * DIM + 3 * DIM * FFN       # weights of one layer's seven projections
KV_ROW = HEADS * HEAD_DIM                         # values of one position's keys (or values)


def work(case):
    kind = case["kind"]
    if kind == "decode":
        w, p, t = case["width"], case["prompt"], case["suffix"]
        per_layer = (_q40_bytes(PROJECTIONS) + 2 * DIM * 2 + 2 * p * KV_ROW * 2      # weights, norms, prompt cache
                     + 2 * w * (t + 1) * _q40_bytes(KV_ROW))                         # suffix read, new row written
        flops = 2 * w * PROJECTIONS + 4 * w * KV_ROW * (p + t + 1)
        return {"bytes": LAYERS * per_layer + (VOCAB * DIM + DIM) * 2 + w * (2 * DIM + 2 * VOCAB + 8),
                "flops": LAYERS * flops + 2 * w * VOCAB * DIM}
    if kind == "prompt":
        s = case["prompt"]
        per_layer = _q40_bytes(PROJECTIONS) + 2 * DIM * 2 + 2 * s * KV_ROW * 2
        flops = 2 * s * PROJECTIONS + 4 * KV_ROW * s * (s + 1) // 2
        return {"bytes": LAYERS * per_layer + (VOCAB * DIM + DIM) * 2 + s * (2 * DIM + 2 * VOCAB + 8),
                "flops": LAYERS * flops + 2 * s * VOCAB * DIM}
    if kind in ("matmul", "linear"):
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": _q40_bytes(n * k, case.get("group", 64)) + 2 * m * (k + n), "flops": 2 * m * n * k}
    if kind == "tree_attn":
        b, h, hkv = case["width"], case["heads"], case["kv_heads"]
        suffix = b * case["suffix"] / 2                                              # lengths are uniform from 0
        return {"bytes": 4 * (case["prompt"] + suffix) * hkv * HEAD_DIM + 4 * b * h * HEAD_DIM,
                "flops": 4 * h * HEAD_DIM * (b * case["prompt"] + suffix)}
    if kind == "branch_attn":
        b, n, h, hkv = case["width"], case["keys"], case["heads"], case["kv_heads"]
        rows = b * n
        if case["paged"]:
            slots = min(32767, max(n, b * n // 2))
            rows = slots * (1 - math.exp(-b * n / slots))                            # different slots of the table
        return {"bytes": 4 * rows * hkv * HEAD_DIM + 4 * b * h * HEAD_DIM + (2 * b * n if case["paged"] else 0),
                "flops": 4 * b * h * n * HEAD_DIM}
    n = case["rows"] * case["cols"]
    return {"bytes": 2 * n + _q40_bytes(n, case["group"]) + 2 * n, "flops": 4 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "pack":
        return "exact"
    if kind in ("decode", "prompt"):
        # fp16 activations rounded some dozen times a layer, 32 layers deep; codes of the appended row
        # flip where a value sits at the middle between two codes (one row of the cache's 256).  Two operand
        # roundings, fp16(code * scale) and fp16(scale * x), put the logits 0.9 % apart
        return {"rel": 1.5e-2, "max": 0.2, "differ": 1e-3}
    # fp16 operands and result, fp32 sums: half an fp16 step per operand and on the way out
    return {"rel": 1.5e-3, "max": 2e-2}


def _expand(q, s, group, shape):
    """The packed matrix in 64 bits: a byte row holds two groups, the even one in the high nibbles."""
    q = q.reshape(-1, group)
    codes = torch.cat(((q >> 4).double(), ((q << 4) >> 4).double()), dim=1).view(-1, group)
    return (codes * s.reshape(-1, 1).double()).view(shape)


def _attend(q, k, v, mask=None):
    """softmax(q k^T / sqrt(d)) v over [..., rows, d] operands in 64 bits; `mask` is true where a key counts."""
    sc = q @ k.transpose(-1, -2) / math.sqrt(HEAD_DIM)
    if mask is not None:
        sc = sc.masked_fill(~mask, -math.inf)
    return torch.softmax(sc, dim=-1) @ v


def _exact_model(case, seed):
    """Logits of the prompt pass, or of the decode step after it, layer by layer in 64 bits."""
    state = prepare(case, seed)
    m, eps = state["model"], 1e-5
    lin = lambda x, l: x @ _expand(l.w, l.s, 64, (int(l.shape[1]), int(l.shape[0])))
    norm = lambda x, w: x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * w.double()
    freq = m.params.rope_theta ** (-torch.arange(0, HEAD_DIM, 2, device=DEV).double() / HEAD_DIM)

    def rope(x, pos):                                  # value i turns with value i + 64, [rows, heads, 128]
        ang = (pos.double()[:, None] * freq)[:, None]
        lo, hi = x.chunk(2, dim=-1)
        return torch.cat((lo * ang.cos() - hi * ang.sin(), hi * ang.cos() + lo * ang.sin()), dim=-1)

    split = lambda x: x.view(x.shape[0], HEADS, HEAD_DIM)
    decode = case["kind"] == "decode"
    if decode:
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        torch.randint(0, 1 << 30, (1,), generator=gen, device=DEV)
        prompt = torch.randint(0, VOCAB, (1, case["prompt"]), generator=gen, device=DEV).view(-1)
    else:
        prompt = state["tokens"].view(-1)
    S = prompt.numel()
    at = torch.arange(S, device=DEV)
    causal = at[:, None] >= at[None, :]
    h = m.tok_embeddings.weight[prompt].double()
    if decode:
        w, t = case["width"], case["suffix"]
        d = m.tok_embeddings.weight[state["tokens"].view(-1)].double()
        here = torch.full((w,), state["pos"], device=DEV)
    heads = lambda x: x.transpose(0, 1)
    for layer in m.layers:
        att, ff = layer.attention, layer.feed_forward
        feed = lambda x: lin(torch.nn.functional.silu(lin(x, ff.w1)) * lin(x, ff.w3), ff.w2)
        x = norm(h, layer.attention_norm.weight)
        k, v = rope(split(lin(x, att.wk)), at), split(lin(x, att.wv))
        o = _attend(heads(rope(split(lin(x, att.wq)), at)), heads(k), heads(v), causal)
        h = h + lin(heads(o).reshape(S, -1), att.wo)
        h = h + feed(norm(h, layer.ffn_norm.weight))
        if decode:
            x = norm(d, layer.attention_norm.weight)
            dq, dk, dv = rope(split(lin(x, att.wq)), here), rope(split(lin(x, att.wk)), here), split(lin(x, att.wv))
            out = []
            for b in range(w):
                own = [torch.cat((p, _expand(c[b, :t], s[b, :t], 64, (t, HEADS, HEAD_DIM)), n[b:b + 1])) for p, c, s, n in
                       ((k, att.cache_k, att.cache_k_s, dk), (v, att.cache_v, att.cache_v_s, dv))]
                out.append(_attend(dq[b][:, None], heads(own[0]), heads(own[1])).reshape(1, -1))
            d = d + lin(torch.cat(out), att.wo)
            d = d + feed(norm(d, layer.ffn_norm.weight))
    r = norm(d if decode else h, m.norm.weight) @ m.output.weight.double().t()
    return r.view(w, 1, -1) if decode else r.view(1, S, -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pack":
        return None                    # codes, and one rounding each way: compared bit for bit
    if kind in ("decode", "prompt"):
        logits = _exact_model(case, seed)
        if kind == "prompt":
            return {"logits": logits, "k": None, "v": None}
        return {"logits": logits, "k": None, "k_scale": None, "v": None, "v_scale": None}
    st = prepare(case, seed)
    if kind == "matmul":
        return st["x"].double() @ _expand(st["w"], st["s"], 64, st["shape"])
    if kind == "linear":
        return st["x"].double() @ _expand(st["w"], st["s"], st["group"], st["shape"]).t()
    h, hkv = case["heads"], case["kv_heads"]
    rep = h // hkv
    out = []
    for b in range(case["width"]):
        if kind == "tree_attn":
            n, page = int(st["lens"][b]), st["page"]
            at = torch.arange(n, device=DEV)
            slot = st["table"][b].long()[at // page] * page + at % page
            k, v = (torch.cat((p.double().transpose(0, 1), s[:, slot].double()), dim=1)
                    for p, s in ((st["pk"], st["k"]), (st["pv"], st["v"])))
        elif st["paged"]:
            k, v = (st[x][:, st["table"][b].long()].double() for x in ("k", "v"))
        else:
            k, v = st["k"][b].double(), st["v"][b].double()
        q = st["q"][b].double()[:, None]
        out.append(_attend(q, k.repeat_interleave(rep, 0), v.repeat_interleave(rep, 0)).view(h, HEAD_DIM))
    return torch.stack(out)
