"""Llama-architecture decoder with Q4_0 linears, a shared fp16 prompt KV cache and a Q4_0
per-branch suffix cache: the host-side mirror of the reference's
hf_model_q40_kv_shared.Transformer (same class and attribute names, same
forward(tokens, start_pos) / fork / resetSeq calls, same checkpoint tensors
`.w`/`.s`/`.shape` per linear), running on the q40b200 kernels.

What differs from the reference is how a decode step executes, not what it computes:
  * the whole step is one CUDA graph per batch width (positions and lengths live in device
    memory, so the graph is replayed for every token);
  * attention reads the shared prompt cache once for all branches and the packed Q4_0
    suffix rows directly, instead of dequantising the whole suffix, concatenating it with a
    per-branch expansion of the prompt and calling SDPA (hf_model_q40_kv_shared.py:346-405);
  * the rounding points of the reference are kept: RMSNorm (fp32 inside, fp16 out, fp16
    weight), fp16(code*scale) weights with fp32 accumulation, fp16 rotary embedding, the
    token being decoded attends to its own un-quantised K/V while later steps see its Q4_0
    round trip, fp16 residual adds, fp16 SiLU-mul.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn.functional as F
from torch import nn

from . import kernels as K
from ._lib import check, lib

DTYPE = torch.float16
GROUP_SIZE = 64


@dataclass
class ModelArgs:
    """Same fields and defaults as the reference's ModelArgs (hf_model_q40_kv_shared.py:58-72)."""
    dim: int = 4096
    n_layers: int = 32
    n_heads: int = 32
    n_kv_heads: Optional[int] = None
    vocab_size: int = 32016
    multiple_of: int = 256
    ffn_dim_multiplier: Optional[float] = None
    norm_eps: float = 1e-5
    rope_theta: float = 1000000.0

    max_batch_size: int = 80
    max_seq_len: int = 256
    max_prompt_seq_len: int = 256


def precompute_freqs_cis(dim: int, end: int, theta: float = 10000.0):
    """fp32 angles exactly as the reference (hf_model_q40_kv_shared.py:137-142)."""
    freqs = 1.0 / (theta ** (torch.arange(0, dim, 2)[: (dim // 2)].float() / dim))
    t = torch.arange(end, device=freqs.device, dtype=torch.float32)
    freqs = torch.outer(t, freqs)
    return torch.polar(torch.ones_like(freqs), freqs)


class HostWord:
    """An int32 in host memory that kernels can write; copies of its owner have one of their own."""
    __slots__ = ("host", "ptr", "_pinned")

    def __init__(self):
        self._pinned = torch.zeros(1, dtype=torch.int32).pin_memory()
        self.host, self.ptr = self._pinned.numpy(), self._pinned.data_ptr()

    def __reduce__(self):
        return HostWord, ()


class RMSNorm(nn.Module):
    def __init__(self, dim: int, eps: float = 1e-6):
        super().__init__()
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(dim), requires_grad=False)

    def forward(self, x):
        return K.rmsnorm(x, self.weight.to(DTYPE), self.eps)


class LinearQ4_0(nn.Module):
    """Holder of one packed weight, as in the reference (hf_model_q40_kv_shared.py:217-236):
    `w` int8 [in*out/128, 64], `s` fp16 [in*out/64], `shape` = (in_features, out_features)
    until a loader overwrites it with the checkpoint's (out, in) — either way the call below
    passes (shape[1], shape[0]) like the reference does."""

    def __init__(self, in_features, out_features, group_size):
        super().__init__()
        self.group_size = group_size
        # placeholders; a loader assigns the checkpoint tensors (already on the device)
        self.w = torch.empty((in_features * out_features // group_size // 2, group_size), dtype=torch.int8,
                             device="meta")
        self.s = torch.empty(in_features * out_features // group_size, dtype=DTYPE, device="meta")
        self.shape = (in_features, out_features)
        self._tiled = self._tiled_cat = None       # rearranged copies (kernels.TiledCopy), made on first use

    def kn(self):
        """(K, N) of the stored [K, N] matrix."""
        return int(self.shape[1]), int(self.shape[0])

    def forward(self, x):
        shape = x.shape
        x2 = x.reshape(shape[0] * shape[1], -1)
        y = K.matmul_q40(x2.contiguous(), self.w, self.s, self.kn(), group_size=self.group_size)
        return y.view(shape[0], shape[1], -1)


class Attention(nn.Module):
    def __init__(self, args: ModelArgs, layer_id: int, caches, tp_world: int = 1):
        super().__init__()
        self.args = args
        self.n_kv_heads = args.n_heads if args.n_kv_heads is None else args.n_kv_heads
        assert args.n_heads % self.n_kv_heads == 0
        # tensor parallel: query heads and kv heads are split across ranks (the reference fixes
        # model_parallel_size = 1, hf_model_q40_kv_shared.py:258-260)
        assert args.n_heads % tp_world == 0 and self.n_kv_heads % tp_world == 0
        self.n_local_heads = args.n_heads // tp_world
        self.n_local_kv_heads = self.n_kv_heads // tp_world
        self.n_rep = self.n_local_heads // self.n_local_kv_heads
        self.head_dim = args.dim // args.n_heads
        self.wq = LinearQ4_0(args.dim, self.n_local_heads * self.head_dim, GROUP_SIZE)
        self.wk = LinearQ4_0(args.dim, self.n_local_kv_heads * self.head_dim, GROUP_SIZE)
        self.wv = LinearQ4_0(args.dim, self.n_local_kv_heads * self.head_dim, GROUP_SIZE)
        self.wo = LinearQ4_0(self.n_local_heads * self.head_dim, args.dim, GROUP_SIZE)
        # views into the model-wide cache tensors (same names as the reference's attributes)
        self.cache_prompt_k = caches["pk"][layer_id]     # [maxP, Hkv, D] fp16
        self.cache_prompt_v = caches["pv"][layer_id]
        self.cache_k = caches["kq"][layer_id]            # [maxB, maxT, Hkv, 64] int8
        self.cache_k_s = caches["ks"][layer_id]          # [maxB, maxT, Hkv, 2] fp16
        self.cache_v = caches["vq"][layer_id]
        self.cache_v_s = caches["vs"][layer_id]
        self.cache_prompt_len = 0


class FeedForward(nn.Module):
    def __init__(self, dim: int, hidden_dim: int, multiple_of: int, ffn_dim_multiplier: Optional[float],
                 tp_world: int = 1):
        super().__init__()
        hidden_dim = int(2 * hidden_dim / 3)
        if ffn_dim_multiplier is not None:
            hidden_dim = int(ffn_dim_multiplier * hidden_dim)
        hidden_dim = multiple_of * ((hidden_dim + multiple_of - 1) // multiple_of)
        self.full_hidden_dim = hidden_dim
        assert hidden_dim % (128 * tp_world) == 0, "the FFN width must split into 128-column blocks per rank"
        hidden_dim //= tp_world          # this rank's columns of w1/w3 and rows of w2
        self.hidden_dim = hidden_dim
        self.w1 = LinearQ4_0(dim, hidden_dim, GROUP_SIZE)
        self.w2 = LinearQ4_0(hidden_dim, dim, GROUP_SIZE)
        self.w3 = LinearQ4_0(dim, hidden_dim, GROUP_SIZE)

    def forward(self, x):
        return self.w2(K.silu_mul(self.w1(x), self.w3(x)))


class TransformerBlock(nn.Module):
    def __init__(self, layer_id: int, args: ModelArgs, caches, tp_world: int = 1):
        super().__init__()
        self.n_heads = args.n_heads
        self.dim = args.dim
        self.head_dim = args.dim // args.n_heads
        self.attention = Attention(args, layer_id, caches, tp_world)
        self.feed_forward = FeedForward(dim=args.dim, hidden_dim=4 * args.dim, multiple_of=args.multiple_of,
                                        ffn_dim_multiplier=args.ffn_dim_multiplier, tp_world=tp_world)
        self.layer_id = layer_id
        self.attention_norm = RMSNorm(args.dim, eps=args.norm_eps)
        self.ffn_norm = RMSNorm(args.dim, eps=args.norm_eps)


def _projections(layer: TransformerBlock):
    att, ff = layer.attention, layer.feed_forward
    return [att.wq, att.wk, att.wv, att.wo, ff.w1, ff.w3, ff.w2]


class Transformer(nn.Module):
    """forward(tokens, start_pos): start_pos == 0 is the prompt (batch 1; fills the shared
    prompt cache), start_pos > 0 with one token per branch is a decode step
    (hf_model_q40_kv_shared.py:492-510)."""

    def __init__(self, params: ModelArgs, device: Optional[torch.device] = None, tp_rank: int = 0,
                 tp_world: int = 1, process_group=None):
        """tp_world > 1: Megatron-style tensor parallelism over one process per GPU — wq/wk/wv/w1/w3
        hold this rank's output columns, wo/w2 its input rows, and the partial outputs of wo and w2
        are summed with an all-reduce over `process_group` (NCCL)."""
        super().__init__()
        self.tp_rank, self.tp_world, self.tp_group = tp_rank, tp_world, process_group
        if not torch.cuda.is_available():
            raise RuntimeError("spec_mcts_b200.model needs a CUDA device (no CPU path)")
        self.device = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        self.params = params
        self.vocab_size = params.vocab_size
        self.n_layers = params.n_layers
        p = params
        Hkv = (p.n_heads if p.n_kv_heads is None else p.n_kv_heads) // tp_world    # local kv heads
        D = p.dim // p.n_heads
        assert D == 128, "the attention kernels are written for head_dim 128"
        self._H = p.n_heads // tp_world                                            # local query heads
        L, dev = p.n_layers, self.device
        self._caches = {
            "pk": torch.zeros((L, p.max_prompt_seq_len, Hkv, D), dtype=DTYPE, device=dev),
            "pv": torch.zeros((L, p.max_prompt_seq_len, Hkv, D), dtype=DTYPE, device=dev),
            "kq": torch.zeros((L, p.max_batch_size, p.max_seq_len, Hkv, 64), dtype=torch.int8, device=dev),
            "ks": torch.zeros((L, p.max_batch_size, p.max_seq_len, Hkv, 2), dtype=DTYPE, device=dev),
            "vq": torch.zeros((L, p.max_batch_size, p.max_seq_len, Hkv, 64), dtype=torch.int8, device=dev),
            "vs": torch.zeros((L, p.max_batch_size, p.max_seq_len, Hkv, 2), dtype=DTYPE, device=dev),
        }
        self.tok_embeddings = nn.Embedding(p.vocab_size, p.dim, device="meta")
        self.layers = nn.ModuleList(TransformerBlock(i, p, self._caches, tp_world) for i in range(p.n_layers))
        self.norm = RMSNorm(p.dim, eps=p.norm_eps)
        self.output = nn.Linear(p.dim, p.vocab_size, bias=False, device="meta")
        self.freqs_cis = precompute_freqs_cis(D, p.max_seq_len + p.max_prompt_seq_len, p.rope_theta)
        self._n_pos = p.max_seq_len + p.max_prompt_seq_len
        self._cos = self.freqs_cis.real.to(DTYPE).contiguous().to(dev)   # [n_pos, 64]
        self._sin = self.freqs_cis.imag.to(DTYPE).contiguous().to(dev)
        self._Hkv, self._D = Hkv, D
        self._prefix_len_dev = torch.zeros(1, dtype=torch.int32, device=dev)
        self._pos_dev = torch.zeros(p.max_batch_size, dtype=torch.int32, device=dev)
        self._tok_dev = torch.zeros(p.max_batch_size, dtype=torch.int64, device=dev)
        self._graphs = {}
        self._bufs = {}
        self._tc_ws = None          # see _step_tc_ws
        self.use_cuda_graph = True
        # when set, a decode step also writes argmax(logits) back as the next input token and
        # advances the positions on the device, so steps can be replayed without the host
        self.greedy_feedback = False
        # kernels of this library enqueued by one decode step (set by it)
        self.launches_per_step = params.n_layers * 8 + 1
        # B <= narrow_max uses the fused, cluster-reduced, dependent-launch-chained matmuls; up to 16 what `_fused_body` says
        self.use_fused = True
        self.use_pdl = True
        self.max_cluster = 16
        # the fused matmuls read a rearranged ("tiled") copy of each weight, made on first use
        self.use_tiled = True
        # above, and the prompt pass: the tensor-core matmul that reads the same tiled copies (A operand
        # written to tensor memory); False: B <= 16 as B <= narrow_max, above the tensor-core matmul on the checkpoint layout
        self.use_tiled_tc = True
        # steps of more branches than this take it: where a layer's launches, three more of them, have enough to do.  Us a step of 8
        # layers (prompt 512, 64 own keys), the narrow matmuls and it: dim 4096, 4 branches 528 and 549, 5 560 and 548, 8 605 and 560;
        # dim 2048, 5 branches 403 and 344; dim 1024, 5 260 and 276, 8 298 and 280; dim 512, 5 213 and 256, 8 222 and 257
        self.narrow_max = 4 if tp_world == 1 and params.dim >= 2048 else 8
        # tensor parallel: all-reduce + residual add + RMSNorm as one launch over peer-mapped buffers (plain
        # stores into the peers' memory); False: torch.distributed all_reduce + the norm kernel
        self.use_tp_fused_allreduce = True
        self.tp_wait_cycles = 0     # limit of the wait for a peer's rows in SM cycles (0: 2^31, about a second)
        self._tp_peer = None
        # the prompt pass above 16 rows reads the tiled copies too (the decode step needs them anyway); True: it reads
        # the checkpoint layout and makes no copies
        self.prefill_checkpoint_layout = False
        # the copies are also made of weights whose writes torch does not count (made under inference_mode), and the
        # call waits for the device and raises itself if a wait in it ran out
        self.prefill_tiled_tc = False
        # True: the prompt pass returns logits of the last position only, [1, 1, vocab] (all a caller that
        # samples the next token needs); False: of every position like the reference
        self.prefill_last_only = False
        # device word that the last prompt pass's tensor-core launches set on a wait expiry (the one of
        # kernels.tc_error_flag), its copy of the last finished pass, and whether nothing has waited for it yet
        self._tc_err = None
        self._tc_err_own = torch.zeros(1, dtype=torch.int32, device=dev)      # ... in place of a captured pass's own word
        self._tc_err_host = torch.zeros(1, dtype=torch.int32).pin_memory()
        self._prompt_unchecked = False
        # the error word of the steps' tensor-core matmuls: host memory that they can write, so that nothing has to be copied
        # (a copy behind each step: 11 us of one of 10 branches)
        self._step_err = HostWord()
        # ... True: through the byte-balanced stream-K launch (one CTA per SM, bulk-copy ring, no clusters);
        # False: the cluster-reduced launch on the same tiled copies (faster on B200, the default)
        self.use_stream = False
        self.stream_smem_budget = 0      # 0 = the library's default (two launches' CTAs share an SM)
        # single-launch attention (rotary + append + attention) up to this width; wider steps read the
        # shared prompt once for all branches (see `_attn_step`)
        # width <= 8: final RMSNorm, fp16 lm_head, arg-max and position bump as one launch (above, the
        # library GEMM is faster than the streaming kernel).  Us of a step of 8 layers behind the
        # tensor-core matmuls, with torch's product and arg-max and with it: dim 4096, 5 branches 545 and 549, with feedback
        # 559 and 553, 8 branches 555 and 561, 571 and 565; its sums are fp32 and a tie goes to the smaller index
        self.use_fused_tail = True
        self.use_fused_attn = True
        self.fused_attn_max_width = 1
        # ... and while prompt + suffix fit in two register batches of its clusters (640 keys each);
        # longer contexts go through the tensor-core prefix pass
        self.fused_attn_max_keys = 1280
        # ... and all layers of a step of up to two branches as one launch, while the same limit holds
        self.use_chain = True
        self._chain_tables = {}     # its layers' addresses, as the kernel reads them
        self._chained = {}          # by width: whether the last step was such a launch
        self._lm_head_q4 = None     # set by quantize_lm_head()

    # ------------------------------------------------------------------ reference API
    @torch.inference_mode()
    def forward(self, tokens: torch.Tensor, start_pos: int):
        bsz, seqlen = tokens.shape
        if start_pos == 0:
            return self._prefill(tokens)
        assert seqlen == 1, "decode steps take one token per branch"
        return self._decode(tokens, start_pos)

    def fork(self, origin: int, curr_batch: int, forks: int):
        """Copy branch `origin`'s suffix cache to `forks` new branches starting at index
        curr_batch, in every layer (hf_model_q40_kv_shared.py:282-297, 512-516)."""
        if forks <= 0:
            return
        for name in ("kq", "ks", "vq", "vs"):
            c = self._caches[name]
            c[:, curr_batch:curr_batch + forks] = c[:, origin:origin + 1]

    def resetSeq(self):
        for layer in self.layers:
            layer.attention.cache_prompt_len = 0
        self._prefix_len_dev.zero_()

    def release_graphs(self):
        """Destroy the captured decode graphs (they are rebuilt on the next step).  With tensor parallelism
        the graphs contain NCCL collectives, and a communicator cannot be torn down while a graph that
        captured its work is alive: call this before torch.distributed.destroy_process_group()."""
        torch.cuda.synchronize(self.device)
        self._graphs.clear()

    def _forget_copies(self):
        """... before tiled copies go away, and with them the tables that hold their addresses.  (Tables stay where graphs alone are released: a
        graph that the caller has captured may read them.)"""
        self.release_graphs()
        self._chain_tables.clear()

    # ------------------------------------------------------------------ prompt
    def _prefill(self, tokens):
        p = self.params
        bsz, S = tokens.shape
        assert bsz == 1, "the prompt is processed once and shared by all branches"
        assert S <= p.max_prompt_seq_len
        if self._prompt_unchecked and int(self._tc_err_host) != 0:      # without waiting for the pass before this one
            self._prompt_failed()
        dev = self.device
        H, Hkv, D = self._H, self._Hkv, self._D
        hid = self.layers[0].feed_forward.hidden_dim
        # K and the widths of the four matmuls of a layer, and whether their shapes are multiplied through tiled copies
        sites = ((p.dim, (H * D, Hkv * D, Hkv * D)), (H * D, (p.dim,)), (p.dim, (hid, hid)), (hid, (p.dim,)))
        copies_read = S > 16 and self.use_tiled and self.use_tiled_tc and not self.prefill_checkpoint_layout
        tiled = [copies_read and Kd % 64 == 0 and all(n % 256 == 0 for n in Ns) for Kd, Ns in sites]
        # copies are made ahead of the pass: a dependent launch reads its weights before it waits for the launch in
        # front of it, which must not be the one that writes them
        plan, capturing = [], torch.cuda.is_current_stream_capturing()
        for layer in self.layers:
            att, ff = layer.attention, layer.feed_forward
            lins = ((att.wq, att.wk, att.wv), (att.wo,), (ff.w1, ff.w3), (ff.w2,))
            plan.append((att, layer.attention_norm.weight, layer.ffn_norm.weight,
                         [(ls, self._prefill_copies(ls, *site, ok, capturing)) for ls, site, ok in zip(lins, sites, tiled)]))
        # the norm launches take bare addresses: not loaded yet, or another device's
        K._need_cuda(self.norm.weight, *[w for _, *ws, _ in plan for w in ws])
        h = self.tok_embeddings(tokens.to(dev)).to(DTYPE).view(S, p.dim)
        pos = torch.arange(S, dtype=torch.int32, device=dev)
        st = torch.cuda.current_stream(dev).cuda_stream
        err = K._tc_error_word(h.device)
        e = lambda n: torch.empty((S, n), dtype=DTYPE, device=dev)
        xn, q, ao, o, a1, a3, g, f = (e(n) for n in (p.dim, H * D, H * D, p.dim, hid, hid, hid, p.dim))
        args = [self._mm_args(Ns) for _, Ns in sites]
        # of all layers' launches with the SiLU product
        scratch = K._tiled_tc_workspace(h.device, S) if any(mm[2][1] is not None for *_, mm in plan) else None
        silu_ws = self._tc_ws_args(scratch)
        pending = None     # output of the previous sub-block, added to h by the next norm kernel
        table = self._prompt_table(plan) if self.tp_world == 1 else None
        if table is not None:
            check(lib.q40_prompt_layers(table, len(plan), S, p.dim, hid, H, Hkv, float(p.norm_eps), h.data_ptr(), xn.data_ptr(), q.data_ptr(),
                                        ao.data_ptr(), o.data_ptr(), g.data_ptr(), f.data_ptr(), pos.data_ptr(), self._cos.data_ptr(),
                                        self._sin.data_ptr(), *silu_ws, err.data_ptr(), 1 if self.use_pdl else 0, st), "q40_prompt_layers")
            for att, *_ in plan:
                att.cache_prompt_len = S
            plan, pending = (), f
        for att, attn_norm, ffn_norm, (qkv, wo, w13, w2) in plan:
            # keys and values go straight to their place in the prompt cache
            ck, cv = att.cache_prompt_k[:S], att.cache_prompt_v[:S]
            self._norm(h, pending, attn_norm, xn, st)
            self._mm(xn, qkv, [q, ck.view(S, Hkv * D), cv.view(S, Hkv * D)], args[0], err, st)
            check(lib.q40_rope_qk(q.data_ptr(), H, H * D, ck.data_ptr(), Hkv, Hkv * D, pos.data_ptr(), self._cos.data_ptr(),
                                  self._sin.data_ptr(), S, D, st), "q40_rope_qk")
            att.cache_prompt_len = S
            # causal attention over the prompt (grouped-query heads read their kv head directly)
            K.causal_attn(q.view(S, H, D), ck, cv, out=ao.view(S, H, D))
            self._mm(ao, wo, [o], args[1], err, st)
            self._all_reduce(o)
            self._norm(h, o, ffn_norm, xn, st)
            if w13[1] is not None:
                self._mm_silu(xn, w13[1], g, args[2], silu_ws, err, st)
            else:
                self._mm(xn, w13, [a1, a3], args[2], err, st)
                check(lib.q40_silu_mul(a1.data_ptr(), a3.data_ptr(), g.data_ptr(), g.numel(), st), "q40_silu_mul")
            self._mm(g, w2, [f], args[3], err, st)
            self._all_reduce(f)
            pending = f
        self._prefix_len_dev.fill_(S)
        self._tc_err = K._tc_error_word(h.device)
        if self._tc_err.data_ptr() != err.data_ptr():     # a larger workspace took the first one's place meanwhile
            self._tc_err |= err
        if capturing and not K._tc_error_word_lasts(h.device):
            # the word is the capture's, and holds nothing until the graph runs
            self._tc_err_own |= self._tc_err
            self._tc_err = self._tc_err_own
        self._tc_err_host.copy_(self._tc_err, non_blocking=True)
        self._prompt_unchecked = S > 16        # narrower passes run no kernel that waits
        if self.prefill_last_only:
            # the tree search reads the last position only (mcts.py:105); the reference computes all S rows
            h, xn, pending = h[S - 1:], xn[S - 1:], pending[S - 1:]
        self._norm(h, pending, self.norm.weight, xn, st)
        logits = F.linear(xn, self.output.weight).to(DTYPE).view(1, h.shape[0], -1)
        if self.prefill_tiled_tc:
            self._check_prompt()
        return logits

    def _prompt_table(self, plan):
        """The addresses that q40_prompt_layers reads, or None where a layer is not multiplied through tiled copies alone or its buffers are
        not laid out for it."""
        rows = []
        rest = (self._Hkv * self._D, self._D, 1)
        for att, attn_norm, ffn_norm, sites in plan:
            ck, cv = att.cache_prompt_k, att.cache_prompt_v
            if (any(tiled is None for _, tiled in sites) or ck.stride() != rest or cv.stride() != rest or
                    not (attn_norm.is_contiguous() and ffn_norm.is_contiguous())):
                return None
            for _, tiled in sites:
                rows += tiled
            rows += (attn_norm, ffn_norm, ck, cv)
        return (ctypes.c_void_p * len(rows))(*[t.data_ptr() for t in rows]) if rows else None

    def _check_prompt(self):
        """Raise if a bounded wait inside a tensor-core matmul of the last prompt pass expired: waits for the pass, so
        that nothing is built on an undefined prompt cache.  Once per pass, by what uses it first."""
        if self._prompt_unchecked and not torch.cuda.is_current_stream_capturing():
            if int(self._tc_err.item()) != 0:
                self._prompt_failed()
            self._prompt_unchecked = False

    @torch.inference_mode()
    def _prompt_failed(self):
        K._reset_tiled_tc_workspaces(self.device)
        self._tc_err.zero_()
        self._tc_err_own.zero_()
        torch.cuda.synchronize(self.device)      # copies of passes in flight have landed
        self._tc_err_host.zero_()
        self._prompt_unchecked = False
        raise K.Q40Error("prompt pass: a bounded wait inside a tensor-core matmul expired")

    def prompt_status(self) -> int:
        """Non-zero if a bounded wait inside a tensor-core matmul of a prompt pass expired, which makes its logits and
        prompt cache undefined (synchronises).  For hosts that take no decode step: the first step after such a pass
        raises, and so does a later prompt pass once the word has reached the host."""
        return 0 if self._tc_err is None else int(self._tc_err.item())

    def _prefill_copies(self, lins, Kd, Ns, tiled, capturing):
        """The tiled copies that a prompt pass multiplies these projections through, or None where it reads the
        checkpoint layout: `tiled` is false, or a copy could be old (a write into an inference tensor is not counted),
        or would have to be made inside a capture (it would hold nothing until the graph runs)."""
        for l, n in zip(lins, Ns):
            if l.kn() != (Kd, n):
                raise K.Q40Error(f"prompt pass: a projection of shape {l.kn()} where {(Kd, n)} is expected")
            if tiled and (l.group_size != 64 or not (self.prefill_tiled_tc or K.writes_counted(l.w, l.s)) or
                          (capturing and self._tiled_copy(l) is None)):
                tiled = False
        if tiled:
            return self._tiled_of(lins)[0]
        if not capturing:
            self._drop_stale(lins)
        return None

    @staticmethod
    def _mm_args(Ns):
        """What the launches of one matmul of every layer share: array types and the output widths."""
        n = len(Ns)
        return n, ctypes.c_void_p * n, (ctypes.c_int64 * n)(*Ns), (ctypes.c_int * n)(*Ns)

    def _mm(self, x, weights, outs, args, err, st):
        """outs[i] = x @ deq(W_i) for projections that share the activations x [M, K] (prompt pass): one tensor-core
        launch when they have tiled copies, matmul_q40 per projection otherwise.  All operands are contiguous."""
        lins, tiled = weights
        if tiled is not None:
            n, P, widths64, widths = args
            check(lib.q40_gemm_tiled_tc_multi(n, x.data_ptr(), x.shape[1], P(*[t.data_ptr() for t in tiled]),
                                              P(*[o.data_ptr() for o in outs]), widths64, widths, x.shape[0], x.shape[1],
                                              err.data_ptr(), 1 if self.use_pdl else 0, st),
                  "q40_gemm_tiled_tc_multi")
            return
        # relayout=False: the checkpoint-layout kernels
        for l, o in zip(lins, outs):
            K.matmul_q40(x, l.w, l.s, l.kn(), group_size=l.group_size, relayout=False, out=o)

    @staticmethod
    def _tc_ws_args(ws):
        return (ws.data_ptr(), ws.numel()) if ws is not None else (None, 0)

    def _mm_silu(self, x, tiled, g, args, ws, err, st):
        """g = silu(x @ deq(W_1)) * (x @ deq(W_3)) for the tiled copies of the two: one launch (prompt pass).  `ws`: address
        and size of its scratch."""
        _, P, widths64, widths = args
        check(lib.q40_gemm_tiled_tc_ws(2, x.data_ptr(), x.stride(0), P(*[t.data_ptr() for t in tiled]), P(*[g.data_ptr()] * 2),
                                       widths64, widths, x.shape[0], x.shape[1], 1, *ws, err.data_ptr(),
                                       1 if self.use_pdl else 0, st), "q40_gemm_tiled_tc_ws")

    # ------------------------------------------------------------------ decode
    def _step_buffers(self, B):
        b = self._bufs.get(B)
        if b is None:
            p, dev = self.params, self.device
            H, Hkv, D = self._H, self._Hkv, self._D
            hid = self.layers[0].feed_forward.hidden_dim
            e = lambda *s: torch.empty(s, dtype=DTYPE, device=dev)
            nb_attn = lib.q40_attn_shared_prefix_workspace_bytes(B, H, D, p.max_prompt_seq_len)
            nb_gemm = max(lib.q40_gemm_workspace_bytes(B, n, k) for (n, k) in
                          [(H * D, p.dim), (hid, p.dim), (p.dim, hid), (p.dim, H * D)])
            b = dict(h=e(B, p.dim), xn=e(B, p.dim), q=e(B, H * D), k=e(B, Hkv * D), v=e(B, Hkv * D),
                     ao=e(B, H * D), o=e(B, p.dim), a1=e(B, hid), a3=e(B, hid), g=e(B, hid), f=e(B, p.dim),
                     attn_ws=torch.empty(nb_attn, dtype=torch.uint8, device=dev),
                     gemm_ws=torch.zeros(nb_gemm, dtype=torch.uint8, device=dev),
                     tc_ws=self._step_tc_ws(B) if B > self.narrow_max else None,
                     logits=e(B, p.vocab_size), qkv=e(B, (H + 2 * Hkv) * D),
                     ss_attn=torch.zeros((B, 1024), dtype=torch.float32, device=dev),
                     ss_ffn=torch.zeros((B, 1024), dtype=torch.float32, device=dev))
            self._bufs[B] = b
        return b

    def _check_steps(self):
        """Raise if a bounded wait inside a matmul of an earlier step expired, as far as the host has heard: without waiting
        for steps in flight."""
        if self._step_err.host[0] and not torch.cuda.is_current_stream_capturing():
            self._steps_failed()

    @torch.inference_mode()
    def _steps_failed(self):
        torch.cuda.synchronize(self.device)
        for bufs in self._bufs.values():
            bufs["gemm_ws"].zero_()
            if "chain_ws" in bufs:
                bufs["chain_ws"].zero_()
        if self._tc_ws is not None:
            self._tc_ws[:K._TILED_TC_FLAGS].zero_()
        torch.cuda.synchronize(self.device)
        self._step_err.host[0] = 0
        raise K.Q40Error("decode step: a bounded wait inside a tensor-core matmul expired")

    def decode_status(self) -> int:
        """Non-zero if a bounded wait inside a tensor-core matmul of a decode step expired, which makes its logits and cache
        rows undefined (synchronises).  The first step that finds the word set raises."""
        torch.cuda.synchronize(self.device)
        return int(self._step_err.host[0])

    def _step_tc_ws(self, B):
        """Scratch of q40_gemm_tiled_tc_ws for a step of B branches, or None where it uses none: one for all widths, whose
        steps run one after the other."""
        if lib.q40_gemm_tiled_tc_ws_bytes(B) == 0:
            return None
        if self._tc_ws is None:
            if torch.cuda.is_current_stream_capturing():
                return None                       # not ready outside of that graph
            nbytes = lib.q40_gemm_tiled_tc_ws_bytes(min(self.params.max_batch_size, 128))
            self._tc_ws = torch.empty(nbytes, dtype=torch.uint8, device=self.device)
            self._tc_ws[:K._TILED_TC_FLAGS].zero_()
        return self._tc_ws

    def _gemm(self, bufs, x, lin: LinearQ4_0, out, st):
        Kd, N = lin.kn()
        ws = bufs["gemm_ws"]
        check(lib.q40_gemm_kn(x.data_ptr(), x.stride(0), lin.w.data_ptr(), lin.s.data_ptr(), out.data_ptr(),
                              out.stride(0), x.shape[0], N, Kd, lin.group_size, ws.data_ptr(), ws.numel(), st),
              "q40_gemm_kn")

    def _step_site(self, x, lins, outs):
        """What the launches of one tensor-core matmul on tiled copies share in all layers of a step, or None where `lins`,
        the first layer's projections, are not multiplied that way.  Laid out once a step: with the rules of _gemm_multi
        asked, and its arrays made, in every layer, the first step at a width took 16.0 ms for 10 branches and 19.4 for 100
        (now 12.3 and 15.9)."""
        kns = [l.kn() for l in lins]
        if not (x.shape[0] > self.narrow_max and self.use_tiled and self.use_tiled_tc and x.stride(0) % 8 == 0 and
                all(l.group_size == 64 and self._tileable(l) and kn[0] == x.shape[1] and kn[0] % 64 == 0 and
                    o.stride(0) % 2 == 0 for l, kn, o in zip(lins, kns, outs))):
            return None
        n = len(lins)
        P = ctypes.c_void_p * n
        return (kns, n, x.data_ptr(), x.stride(0), P, P(*[o.data_ptr() for o in outs]),
                (ctypes.c_int64 * n)(*[o.stride(0) for o in outs]), (ctypes.c_int * n)(*[kn[1] for kn in kns]), *x.shape)

    def _step_mm(self, site, lins, st, silu_ws=None):
        """One layer's launch of a prepared matmul (`silu_ws`: of silu(x @ W_1) * (x @ W_3), with that scratch); False if its
        projections are not like the first layer's."""
        if site is None:
            return False
        kns, n, x, ldx, P, outs, ldc, widths, M, Kd = site
        for l, kn in zip(lins, kns):
            if l.kn() != kn or l.group_size != 64:
                return False
        tiled, pdl = self._tiled_of(lins)
        tiled, err = P(*[t.data_ptr() for t in tiled]), self._step_err.ptr
        if silu_ws is not None:
            check(lib.q40_gemm_tiled_tc_ws(n, x, ldx, tiled, outs, ldc, widths, M, Kd, 1, *silu_ws, err,
                                           1 if pdl else 0, st), "q40_gemm_tiled_tc_ws")
        else:
            check(lib.q40_gemm_tiled_tc_multi(n, x, ldx, tiled, outs, ldc, widths, M, Kd, err, 1 if pdl else 0, st),
                  "q40_gemm_tiled_tc_multi")
        return True

    def _gemm_multi(self, bufs, x, lins, outs, st):
        """Several projections of the same activations: one tensor-core launch above `narrow_max` rows when the
        shapes allow it, one launch per matrix otherwise."""
        M, n = x.shape[0], len(lins)
        if M > self.narrow_max and self.use_tiled and self.use_tiled_tc and x.stride(0) % 8 == 0:
            # matrices that have a tiled copy (N % 256 == 0) go through the tensor-core kernel that reads it;
            # the others (e.g. one kv head per rank under 8-way tensor parallelism) keep the checkpoint layout
            t_idx = [i for i, (l, o) in enumerate(zip(lins, outs))
                     if l.group_size == 64 and self._tileable(l) and l.kn()[0] % 64 == 0 and o.stride(0) % 2 == 0]
            if len(t_idx) < n and self._concat_tileable(lins, outs):
                # widths that cannot be tiled one by one (a kv head per rank: 128 columns) but whose outputs are
                # adjacent column ranges of one buffer: one tiled copy of the concatenated matrix, one launch
                cat, pdl = self._tiled_concat(lins)
                err = self._step_err.ptr
                P1 = ctypes.c_void_p * 1
                check(lib.q40_gemm_tiled_tc_multi(1, x.data_ptr(), x.stride(0), P1(cat.data_ptr()),
                                                  P1(outs[0].data_ptr()), (ctypes.c_int64 * 1)(outs[0].stride(0)),
                                                  (ctypes.c_int * 1)(sum(l.kn()[1] for l in lins)), M,
                                                  lins[0].kn()[0], err, 1 if pdl else 0, st),
                      "q40_gemm_tiled_tc_multi")
                return
            if t_idx and len(t_idx) < n:
                rest = [i for i in range(n) if i not in t_idx]
                self._gemm_multi(bufs, x, [lins[i] for i in t_idx], [outs[i] for i in t_idx], st)
                self.use_tiled_tc = False
                try:
                    self._gemm_multi(bufs, x, [lins[i] for i in rest], [outs[i] for i in rest], st)
                finally:
                    self.use_tiled_tc = True
                return
            if t_idx and n <= 3 and all(l.kn()[0] == lins[0].kn()[0] for l in lins):
                P = ctypes.c_void_p * n
                err = self._step_err.ptr
                tiled, pdl = self._tiled_of(lins)
                check(lib.q40_gemm_tiled_tc_multi(n, x.data_ptr(), x.stride(0), P(*[t.data_ptr() for t in tiled]),
                                                  P(*[o.data_ptr() for o in outs]),
                                                  (ctypes.c_int64 * n)(*[o.stride(0) for o in outs]),
                                                  (ctypes.c_int * n)(*[l.kn()[1] for l in lins]), M, lins[0].kn()[0],
                                                  err, 1 if pdl else 0, st), "q40_gemm_tiled_tc_multi")
                return
        ok = M > 16 and n <= 3 and all(l.group_size == 64 and l.kn()[1] % 128 == 0 and l.kn()[0] % 64 == 0 and
                                       l.kn()[0] == lins[0].kn()[0] and o.stride(0) % 2 == 0
                                       for l, o in zip(lins, outs)) and x.stride(0) % 8 == 0
        if not ok:
            for l, o in zip(lins, outs):
                self._gemm(bufs, x, l, o, st)
            return
        P = ctypes.c_void_p * n
        err = self._step_err.ptr
        check(lib.q40_gemm_kn_tc_multi(n, x.data_ptr(), x.stride(0), P(*[l.w.data_ptr() for l in lins]),
                                       P(*[l.s.data_ptr() for l in lins]), P(*[o.data_ptr() for o in outs]),
                                       (ctypes.c_int64 * n)(*[o.stride(0) for o in outs]),
                                       (ctypes.c_int * n)(*[l.kn()[1] for l in lins]), M, lins[0].kn()[0], err,
                                       1 if self.use_pdl else 0, st),
              "q40_gemm_kn_tc_multi")

    def _narrow(self, B):
        return self.use_fused and B <= 16 and self.tp_world == 1

    def _fused_body(self, B):
        """Whether a step of B branches takes the narrow matmuls with their fused neighbours.  Beyond `narrow_max` the
        tensor-core matmuls make up for two norm launches a layer (10 branches: 2.75 ms a step with the narrow ones), where the
        shapes and switches allow them."""
        if not self._narrow(B):
            return False
        if B <= self.narrow_max or self.use_stream or self._lm_head_q4 is not None or not (self.use_tiled and self.use_tiled_tc):
            return True
        layer = self.layers[0]
        return not all(l.group_size == 64 and self._tileable(l) and l.kn()[0] % 64 == 0 for l in _projections(layer))

    def _silu_pair(self, B, ff):
        """Whether w1 and w3 of a step of B branches are one launch with the SiLU product."""
        lins = (ff.w1, ff.w3)
        return (B > self.narrow_max and self.use_tiled and self.use_tiled_tc and lins[0].kn() == lins[1].kn() and
                all(l.group_size == 64 and self._tileable(l) and l.kn()[0] % 64 == 0 for l in lins))

    def _decode_body(self, B):
        """Enqueue one decode step for B branches on the current stream (captured into a graph)."""
        self._chained[B] = False
        if self._fused_body(B):
            return self._decode_body_fused(B)
        return self._decode_body_unfused(B)

    @staticmethod
    def _tileable(lin):
        return lin.kn()[1] % 256 == 0 and lin.kn()[0] % 16 == 0

    def _tiled_of(self, lins):
        """The rearranged copies of these layers' weights: made on first use, and again after `w` or `s` was assigned
        or written in place; and whether a launch may read them before it waits for the one in front of it (not if
        that one writes a copy)."""
        out, pdl = [], self.use_pdl
        for l in lins:
            c = self._tiled_copy(l)
            if c is None:
                if l._tiled is not None:
                    self._forget_copies()         # captured steps hold the address of the copy that goes away
                c = l._tiled = K.TiledCopy(K.relayout_tiled(l.w, l.s, l.kn()), l.kn(), l.w, l.s)
                pdl = False
            out.append(c.data)
        return out, pdl

    @staticmethod
    def _tiled_copy(l):
        """The copy of a layer's weight that is there and up to date, or None."""
        c = l._tiled
        return c if c is not None and c.is_of(l.kn(), l.w, l.s) else None

    def drop_tiled_copies(self):
        """Forget the rearranged weight copies (made again on the next step): for weights written in a way torch
        does not count, through `.data`, a raw pointer or under inference_mode."""
        self._forget_copies()
        for layer in self.layers:
            for l in _projections(layer):
                l._tiled = l._tiled_cat = None
        if self._lm_head_q4 is not None:
            self._lm_head_q4._tiled = None

    def _drop_stale(self, lins):
        """Drop these layers' copies, and the captured steps that read them, if their weights have changed."""
        for l in lins:
            cat = l._tiled_cat
            if l._tiled is not None and self._tiled_copy(l) is None:
                self._forget_copies()
                l._tiled = None
            if cat is not None and not cat.is_of(*self._concat_source(lins)):
                self.release_graphs()
                l._tiled_cat = None

    @staticmethod
    def _concat_source(lins):
        return (tuple(l.kn() for l in lins), *[t for l in lins for t in (l.w, l.s)])

    @staticmethod
    def _concat_tileable(lins, outs):
        """The matrices share K and the group size, their widths are whole 128-column packed blocks that add
        up to whole 256-column spans, and their outputs are consecutive column ranges of one row-major buffer."""
        Kd = lins[0].kn()[0]
        if Kd % 64 != 0 or any(l.group_size != 64 or l.kn()[0] != Kd or l.kn()[1] % 128 != 0 for l in lins):
            return False
        if sum(l.kn()[1] for l in lins) % 256 != 0 or outs[0].stride(0) % 2 != 0:
            return False
        ptr = outs[0].data_ptr()
        for l, o in zip(lins, outs):
            if o.data_ptr() != ptr or o.stride(0) != outs[0].stride(0) or o.stride(1) != 1:
                return False
            ptr += l.kn()[1] * o.element_size()
        return True

    def _tiled_concat(self, lins):
        """Tiled copy of [W_0 | W_1 | ...] (columns concatenated): packed rows and scale rows of the checkpoint
        layout concatenate block by block, so no code or scale changes.  Cached on the first matrix.  Returns the copy
        and the second value of _tiled_of."""
        pdl = self.use_pdl
        first, src = lins[0], self._concat_source(lins)
        c = first._tiled_cat
        if c is None or not c.is_of(*src):
            if c is not None:
                self.release_graphs()
            Kd = first.kn()[0]
            w = torch.cat([l.w.reshape(Kd, l.kn()[1] // 2) for l in lins], dim=1).contiguous()
            sc = torch.cat([l.s.reshape(Kd, l.kn()[1] // 64) for l in lins], dim=1).contiguous()
            data = K.relayout_tiled(w, sc, (Kd, sum(l.kn()[1] for l in lins)))
            c = first._tiled_cat = K.TiledCopy(data, *src)
            pdl = False
        return c.data, pdl

    def _streamable(self, lins, M):
        return self.use_tiled and self.use_stream and M <= 16 and all(self._tileable(l) for l in lins)

    def _stream_ws(self, bufs, M):
        """Workspace of the stream-K launches of one step (they run one after the other on one stream)."""
        ws = bufs.get("stream_ws")
        if ws is None:
            p, hid = self.params, self.layers[0].feed_forward.hidden_dim
            H, Hkv, D = self._H, self._Hkv, self._D
            vp = (p.vocab_size + 255) // 256 * 256
            shapes = [((H + 2 * Hkv) * D, p.dim), (p.dim, H * D), (2 * hid, p.dim), (p.dim, hid), (vp, p.dim)]
            nb = max(lib.q40_gemv_stream_workspace_bytes(M, n, k) for n, k in shapes if n % 256 == 0 and k % 16 == 0)
            ws = bufs["stream_ws"] = torch.zeros(max(nb, 4096), dtype=torch.uint8, device=self.device)
        return ws

    def _ss_count(self, N, Kd, M, lins):
        """Sum-of-squares partials per row written by the mode-2 launch that produces N columns."""
        if self._streamable(lins, M):
            return lib.q40_gemv_stream_ss_count(N)
        return lib.q40_gemv_fused_ss_count(N, Kd, self.max_cluster)

    def _fused(self, mode, lins, outs, ldc, a, lda, M, norm_w=None, ss_in=None, ss_in_count=0, h_in=None,
               ldh=0, ss_out=None, ss_out_count=0, st=None, bufs=None):
        n = len(lins)
        P = ctypes.c_void_p * n
        tiled = self.use_tiled and M <= 16 and all(self._tileable(l) for l in lins)
        pdl = self.use_pdl
        if tiled:
            copies, pdl = self._tiled_of(lins)
            bw = P(*[t.data_ptr() for t in copies])
        else:
            bw = P(*[l.w.data_ptr() for l in lins])
        op = P(*[o.data_ptr() for o in outs])
        nc = (ctypes.c_int * n)(*[l.kn()[1] for l in lins])
        Kd = lins[0].kn()[0]
        nw = norm_w.data_ptr() if norm_w is not None else None
        si = ss_in.data_ptr() if ss_in is not None else None
        hi = h_in.data_ptr() if h_in is not None else None
        so = ss_out.data_ptr() if ss_out is not None else None
        if tiled and self.use_stream and bufs is not None:
            ws = self._stream_ws(bufs, M)
            check(lib.q40_gemv_stream(mode, n, bw, op, nc, ldc, a.data_ptr(), lda, M, Kd, nw, si, ss_in_count,
                                      float(self.params.norm_eps), hi, ldh, so, ss_out_count, ws.data_ptr(),
                                      ws.numel(), self.stream_smem_budget, 1 if pdl else 0, st),
                  "q40_gemv_stream")
            return
        bs = P(*[l.s.data_ptr() for l in lins])
        fn = lib.q40_gemv_tiled if tiled else lib.q40_gemv_fused
        check(fn(mode, n, bw, bs, op, nc, ldc, a.data_ptr(), lda, M, Kd, nw, si, ss_in_count,
                 float(self.params.norm_eps), hi, ldh, so, ss_out_count,
                 self.max_cluster, 1 if pdl else 0, st), "q40_gemv_fused")

    def stream_status(self, B) -> int:
        """Non-zero if a bounded wait inside a stream-K launch of the last steps expired (synchronises)."""
        b = self._bufs.get(B)
        if b is None or "stream_ws" not in b:
            return 0
        return int(b["stream_ws"][:4].view(torch.int32).item())

    def _fused_attn_for(self, B):
        p = self.params
        return (self.use_fused_attn and B <= self.fused_attn_max_width and
                p.max_prompt_seq_len + p.max_seq_len <= self.fused_attn_max_keys)

    def _chain_ws_bytes(self, B):
        """Bytes of scratch of the launch that does all layers of a step of B branches, or 0 where a step is a chain of launches."""
        p = self.params
        if not (self.use_chain and self.use_tiled and not self.use_stream and self.use_fused_attn and B <= 2 and
                self.tp_world == 1 and p.max_prompt_seq_len + p.max_seq_len <= self.fused_attn_max_keys):
            return 0
        return lib.q40_decode_chain_ws_bytes(B, p.n_layers, p.dim, self.layers[0].feed_forward.hidden_dim, self._H, self._Hkv)

    def _chain(self, B, bufs, st):
        """Enqueue all layers of a step as one launch: bufs["h"] and the sums of squares in bufs["ss_ffn"], one per row, as the
        last layer leaves them.  False, and nothing is enqueued, where that cannot be."""
        nbytes = self._chain_ws_bytes(B)
        if nbytes == 0:
            return False
        p, hid = self.params, self.layers[0].feed_forward.hidden_dim
        H, Hkv = self._H, self._Hkv
        shapes = [(p.dim, H * 128), (p.dim, Hkv * 128), (p.dim, Hkv * 128), (H * 128, p.dim), (p.dim, hid), (p.dim, hid), (hid, p.dim)]
        for layer in self.layers:
            att, norms = layer.attention, (layer.attention_norm.weight, layer.ffn_norm.weight)
            if (any(l.group_size != 64 or l.kn() != kn for l, kn in zip(_projections(layer), shapes)) or
                    any(w.dtype != DTYPE or not w.is_contiguous() or w.data_ptr() % 8 for w in norms) or
                    any(c.stride() != (Hkv * 128, 128, 1) or c.data_ptr() % 16 for c in (att.cache_prompt_k, att.cache_prompt_v))):
                return False
        rows = []
        for layer in self.layers:
            att = layer.attention
            tensors = (*self._tiled_of(_projections(layer))[0], layer.attention_norm.weight, layer.ffn_norm.weight, att.cache_prompt_k,
                       att.cache_prompt_v, att.cache_k, att.cache_k_s, att.cache_v, att.cache_v_s)
            rows.append([t.data_ptr() for t in tensors] + [0])
        key = tuple(a for r in rows for a in r)
        table, ws = self._chain_tables.get(key), bufs.get("chain_ws")
        if table is None or ws is None:
            if torch.cuda.is_current_stream_capturing():
                return False                      # neither may be made inside a graph
            table = self._chain_tables[key] = torch.tensor(rows, dtype=torch.int64).to(self.device)
            if ws is None:
                ws = bufs["chain_ws"] = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)
        rc = lib.q40_decode_chain(table.data_ptr(), p.n_layers, B, p.dim, hid, H, Hkv, self._tok_dev.data_ptr(),
                                  self.tok_embeddings.weight.data_ptr(), p.vocab_size, self._pos_dev.data_ptr(),
                                  self._prefix_len_dev.data_ptr(), self._cos.data_ptr(), self._sin.data_ptr(), self._n_pos,
                                  p.max_seq_len, p.max_prompt_seq_len, float(p.norm_eps), bufs["h"].data_ptr(),
                                  bufs["ss_ffn"].data_ptr(), ws.data_ptr(), ws.numel(), self._step_err.ptr, st)
        if rc == -5:                              # Q40_E_UNSUPPORTED: the device does not give it all SMs
            self.use_chain = False
            return False
        check(rc, "q40_decode_chain")
        return True

    def _attn_step(self, att, q, k, v, ld, ao, B, ws, st):
        """Rotary embedding, cache append and attention of a step's new tokens (rows of `ld` values), as two launches, prompt and branches.
        With a launch of its own for rotation and append (q40_rope_kv_append) a step is slower at all widths: us for 8 layers with 32 heads,
        prompt 512, 64 and 200 own keys, 6 branches 528 and 545 / 548 and 563, 44 branches 612 and 622 / 685 and 693, 100 branches
        761 and 765 / 892 and 909."""
        p, pk, pv = self.params, att.cache_prompt_k, att.cache_prompt_v
        check(lib.q40_attn_tree_step(q.data_ptr(), ld, k.data_ptr(), v.data_ptr(), ld, pk.data_ptr(), pv.data_ptr(), p.max_prompt_seq_len,
                                     self._prefix_len_dev.data_ptr(), pk.stride(0), pk.stride(1), att.cache_k.data_ptr(),
                                     att.cache_k_s.data_ptr(), att.cache_v.data_ptr(), att.cache_v_s.data_ptr(), p.max_seq_len,
                                     self._pos_dev.data_ptr(), self._cos.data_ptr(), self._sin.data_ptr(), self._n_pos, ao.data_ptr(), B,
                                     self._H, self._Hkv, self._D, ws.data_ptr(), ws.numel(), st), "q40_attn_tree_step")

    def _decode_body_fused(self, B):
        """Decode step for few branches (see `_fused_body`): one launch for all layers (see `_chain`), or 6 per layer (qkv with RMSNorm prologue,
        2 of attention with rotary embedding and append, wo with residual epilogue, w1/w3 with RMSNorm prologue and
        SiLU-mul epilogue, w2 with residual epilogue), chained with programmatic dependent launch."""
        p, bufs = self.params, self._step_buffers(B)
        H, Hkv, D = self._H, self._Hkv, self._D
        self._check_loaded()
        st = torch.cuda.current_stream(self.device).cuda_stream
        hid = self.layers[0].feed_forward.hidden_dim
        l0 = self.layers[0]
        c_attn = self._ss_count(p.dim, H * D, B, [l0.attention.wo])             # written by wo
        c_ffn = self._ss_count(p.dim, hid, B, [l0.feed_forward.w2])             # written by w2
        h, qkv, ao, gbuf = bufs["h"], bufs["qkv"], bufs["ao"], bufs["g"]
        ss_attn, ss_ffn = bufs["ss_attn"], bufs["ss_ffn"]
        W = (H + 2 * Hkv) * D
        q, k, v = qkv[:, :H * D], qkv[:, H * D:(H + Hkv) * D], qkv[:, (H + Hkv) * D:]
        pos, plen, aws = self._pos_dev, self._prefix_len_dev, bufs["attn_ws"]
        chained = self._chained[B] = self._chain(B, bufs, st)
        if chained:
            c_ffn = 1
        else:
            check(lib.q40_embed_rows(self.tok_embeddings.weight.data_ptr(), self._tok_dev.data_ptr(), h.data_ptr(),
                                     ss_ffn.data_ptr(), c_ffn, B, p.dim, p.vocab_size, st), "q40_embed_rows")
        for layer in () if chained else self.layers:
            att, ff = layer.attention, layer.feed_forward
            self._fused(1, [att.wq, att.wk, att.wv], [q, k, v], W, h, p.dim, B,
                        norm_w=layer.attention_norm.weight, ss_in=ss_ffn, ss_in_count=c_ffn, st=st, bufs=bufs)
            if self._fused_attn_for(B):
                pk, pv = att.cache_prompt_k, att.cache_prompt_v
                check(lib.q40_attn_tree_fused(qkv.data_ptr(), W, pk.data_ptr(), pv.data_ptr(), att.cache_k.data_ptr(),
                                              att.cache_k_s.data_ptr(), att.cache_v.data_ptr(),
                                              att.cache_v_s.data_ptr(), pos.data_ptr(), plen.data_ptr(),
                                              self._cos.data_ptr(), self._sin.data_ptr(), self._n_pos, ao.data_ptr(),
                                              B, H, Hkv, D, p.max_seq_len, p.max_prompt_seq_len,
                                              1 if self.use_pdl else 0, st),
                      "q40_attn_tree_fused")
            else:
                self._attn_step(att, q, k, v, W, ao, B, aws, st)
            self._fused(2, [att.wo], [h], p.dim, ao, H * D, B, h_in=h, ldh=p.dim, ss_out=ss_attn,
                        ss_out_count=c_attn, st=st, bufs=bufs)
            self._fused(3, [ff.w1, ff.w3], [gbuf, gbuf], hid, h, p.dim, B, norm_w=layer.ffn_norm.weight,
                        ss_in=ss_attn, ss_in_count=c_attn, st=st, bufs=bufs)
            self._fused(2, [ff.w2], [h], p.dim, gbuf, hid, B, h_in=h, ldh=p.dim, ss_out=ss_ffn,
                        ss_out_count=c_ffn, st=st, bufs=bufs)
        if self._lm_head_q4 is not None:
            # final RMSNorm as the prologue of the Q4_0 lm_head launch; the padded columns are cut off
            lin = self._lm_head_q4
            vp = lin.kn()[1]
            if "logits_pad" not in bufs:
                bufs["logits_pad"] = torch.empty((B, vp), dtype=DTYPE, device=self.device)
            self._fused(1, [lin], [bufs["logits_pad"]], vp, h, p.dim, B, norm_w=self.norm.weight, ss_in=ss_ffn,
                        ss_in_count=c_ffn, st=st, bufs=bufs)
            logits = bufs["logits_pad"][:, :p.vocab_size]
        elif self._fused_tail(B):
            return self._lm_head(B, bufs, ss_ffn, c_ffn, st)
        else:
            self._norm(h, None, self.norm.weight, bufs["xn"], st)
            logits = bufs["logits"]
            torch.matmul(bufs["xn"], self.output.weight.t(), out=logits)
        if self.greedy_feedback:
            self._tok_dev[:B].copy_(logits.argmax(dim=-1))
            self._pos_dev[:B] += 1
        return logits

    def _fused_tail(self, B):
        return self.use_fused_tail and self._narrow(B) and B <= 8 and self.params.dim % 128 == 0

    def _lm_head(self, B, bufs, ss, ss_count, st):
        """Final RMSNorm of bufs["h"], fp16 lm_head and (greedy feedback) arg-max and position bump: one launch.  `ss`: partial
        sums of squares of the rows, or None."""
        p, h, logits, fb = self.params, bufs["h"], bufs["logits"], self.greedy_feedback
        if "lm_scratch" not in bufs:
            bufs["lm_scratch"] = torch.zeros(lib.q40_lm_head_scratch_bytes(), dtype=torch.uint8, device=self.device)
        check(lib.q40_lm_head(h.data_ptr(), p.dim, ss.data_ptr() if ss is not None else None, ss_count, self.norm.weight.data_ptr(),
                              float(p.norm_eps), self.output.weight.data_ptr(), p.vocab_size, p.dim,
                              logits.data_ptr(), logits.stride(0), B,
                              self._tok_dev.data_ptr() if fb else None, self._pos_dev.data_ptr() if fb else None,
                              bufs["lm_scratch"].data_ptr(), 1 if self.use_pdl else 0, st), "q40_lm_head")
        return logits

    def quantize_lm_head(self):
        """Optional, and NOT the reference's model (its lm_head stays fp16, so logits change by the
        quantisation error): pack `output.weight` as Q4_0 (vocabulary padded to a multiple of 256 with
        zero rows) and let decode steps of up to 16 branches compute final RMSNorm + lm_head in one
        tiled matmul launch.  Wider steps and the prompt pass keep the fp16 weight."""
        W = self.output.weight
        V, dim = W.shape
        vp = (V + 255) // 256 * 256
        wp = torch.zeros((vp, dim), dtype=DTYPE, device=W.device)
        wp[:V] = W.to(DTYPE)
        lin = LinearQ4_0(dim, vp, GROUP_SIZE)
        lin.w, lin.s = K.quantize_q40(wp.t().contiguous(), GROUP_SIZE)
        lin.shape = (vp, dim)
        self._lm_head_q4 = lin
        self._graphs.clear()

    def _decode_body_unfused(self, B):
        """One launch per operation; serves any batch width."""
        p, bufs = self.params, self._step_buffers(B)
        H, Hkv, D = self._H, self._Hkv, self._D
        self._check_loaded()
        st = torch.cuda.current_stream(self.device).cuda_stream
        h, xn = bufs["h"], bufs["xn"]
        if self._narrow(B):
            # one launch, which clamps token ids, as in the other body (the sums of squares are not used)
            check(lib.q40_embed_rows(self.tok_embeddings.weight.data_ptr(), self._tok_dev.data_ptr(), h.data_ptr(),
                                     bufs["ss_ffn"].data_ptr(), 1, B, p.dim, p.vocab_size, st), "q40_embed_rows")
        else:
            h.copy_(self.tok_embeddings(self._tok_dev[:B]).to(DTYPE))
        aws = bufs["attn_ws"]
        pending = None     # output of the previous sub-block, added to h by the next norm kernel
        peer = self._tp_peer_buffers() if self.tp_world > 1 and self.use_tp_fused_allreduce else None
        normed = False     # xn already holds the attention norm of h (written by the fused all-reduce)
        qkv, ao, g = bufs["qkv"], bufs["ao"], bufs["g"]
        Wq = (H + 2 * Hkv) * D
        bq, bk, bv = qkv[:, :H * D], qkv[:, H * D:(H + Hkv) * D], qkv[:, (H + Hkv) * D:]
        att, ff = self.layers[0].attention, self.layers[0].feed_forward
        q_site = self._step_site(xn, (att.wq, att.wk, att.wv), (bq, bk, bv))
        o_site = self._step_site(ao, (att.wo,), (bufs["o"],))
        f_site = self._step_site(g, (ff.w2,), (bufs["f"],))
        silu_site = self._step_site(xn, (ff.w1, ff.w3), (g, g)) if self._silu_pair(B, ff) else None
        scratch = bufs["tc_ws"]
        if scratch is None and silu_site is not None:
            scratch = K._tiled_tc_workspace(h.device, B)
        silu_ws = self._tc_ws_args(scratch)
        for li, layer in enumerate(self.layers):
            att, ff = layer.attention, layer.feed_forward
            if not normed:
                self._norm(h, pending, layer.attention_norm.weight, xn, st)
            if not self._step_mm(q_site, (att.wq, att.wk, att.wv), st):
                self._gemm_multi(bufs, xn, [att.wq, att.wk, att.wv], [bq, bk, bv], st)
            self._attn_step(att, bq, bk, bv, Wq, ao, B, aws, st)
            if not self._step_mm(o_site, (att.wo,), st):
                self._gemm_multi(bufs, ao, [att.wo], [bufs["o"]], st)
            if peer is not None:
                # all-reduce of the partial wo outputs + residual add + ffn norm: one launch
                peer.allreduce_norm(bufs["o"], h, layer.ffn_norm.weight, xn, p.norm_eps, st, self.tp_wait_cycles)
            else:
                self._all_reduce(bufs["o"])
                self._norm(h, bufs["o"], layer.ffn_norm.weight, xn, st)
            if not self._step_mm(silu_site, (ff.w1, ff.w3), st, silu_ws):
                self._gemm_multi(bufs, xn, [ff.w1, ff.w3], [bufs["a1"], bufs["a3"]], st)
                check(lib.q40_silu_mul(bufs["a1"].data_ptr(), bufs["a3"].data_ptr(), g.data_ptr(), g.numel(), st),
                      "q40_silu_mul")
            if not self._step_mm(f_site, (ff.w2,), st):
                self._gemm_multi(bufs, g, [ff.w2], [bufs["f"]], st)
            if peer is not None:
                # ... of the partial w2 outputs + residual add + the next layer's attention norm (or the final norm)
                nxt = self.layers[li + 1].attention_norm.weight if li + 1 < len(self.layers) else self.norm.weight
                peer.allreduce_norm(bufs["f"], h, nxt, xn, p.norm_eps, st, self.tp_wait_cycles)
                normed = True
            else:
                self._all_reduce(bufs["f"])
                pending = bufs["f"]
        if not normed:
            self._norm(h, pending, self.norm.weight, xn, st)
        if self._fused_tail(B):
            # the launch in front has added the last sub-block to h
            return self._lm_head(B, bufs, None, 0, st)
        torch.matmul(xn, self.output.weight.t(), out=bufs["logits"])
        if self.greedy_feedback:
            self._tok_dev[:B].copy_(bufs["logits"].argmax(dim=-1))
            self._pos_dev[:B] += 1
        return bufs["logits"]

    def _tp_peer_buffers(self):
        """Peer-mapped buffers of the fused all-reduce launch (made on first use: a collective call)."""
        if self._tp_peer is None:
            from .tp_comm import PeerBuffers
            self._tp_peer = PeerBuffers(self.tp_rank, self.tp_world, self.params.max_batch_size, self.params.dim,
                                        self.device, group=self.tp_group)
        return self._tp_peer

    def tp_status(self) -> int:
        """Non-zero if a bounded wait of a fused all-reduce launch expired (1 + the missing rank; synchronises)."""
        return self._tp_peer.status() if self._tp_peer is not None else 0

    def release_tp_buffers(self):
        """Unmap and free the peer-mapped buffers (collective; after release_graphs, before the process group
        is destroyed)."""
        if self._tp_peer is not None:
            self._tp_peer.close()
            self._tp_peer = None

    def _all_reduce(self, t):
        """Sum the partial outputs of a row-parallel matmul over the tensor-parallel ranks."""
        if self.tp_world > 1:
            import torch.distributed as dist
            dist.all_reduce(t, op=dist.ReduceOp.SUM, group=self.tp_group)
        return t

    def _check_loaded(self):
        for t in (self.norm.weight, self.layers[0].attention_norm.weight, self.output.weight,
                  self.tok_embeddings.weight, self.layers[0].attention.wq.w):
            if not t.is_cuda or (t.is_floating_point() and t.dtype != DTYPE):
                raise RuntimeError("model weights must be loaded and moved with model.to(device, float16) "
                                   "before the first step (found a %s %s tensor)" % (t.device, t.dtype))

    def _norm(self, h, residual, weight, out, st):
        """out = RMSNorm(h + residual) with h updated in place (residual may be None)."""
        p = self.params
        check(lib.q40_rmsnorm(h.data_ptr(), residual.data_ptr() if residual is not None else None,
                              weight.contiguous().data_ptr(), out.data_ptr(), h.data_ptr() if residual is not None else None,
                              h.shape[0], p.dim, float(p.norm_eps), st), "q40_rmsnorm")

    def _decode(self, tokens, start_pos):
        B = tokens.shape[0]
        assert B <= self.params.max_batch_size
        self._tok_dev[:B].copy_(tokens.reshape(B), non_blocking=True)
        self._pos_dev[:B].fill_(start_pos)
        logits = self.decode_replay(B)
        return logits.view(B, 1, -1)

    def decode_replay(self, B):
        """Run one decode step for B branches with the tokens/positions already in the device
        buffers (`_tok_dev`, `_pos_dev`); returns the static logits buffer [B, vocab]."""
        self._check_prompt()
        self._check_steps()
        fused = self._fused_body(B)
        if not self.use_cuda_graph:
            logits = self._decode_body(B)
            self._count_launches(B, fused)
            return logits
        key = self._graph_key(B)
        if key not in self._graphs:
            # torch requires capture on a side stream after a warm-up run; with greedy feedback that run
            # overwrites the input token and advances the position, so both are put back afterwards
            tok_saved = self._tok_dev[:B].clone() if self.greedy_feedback else None
            s = torch.cuda.Stream(self.device)
            s.wait_stream(torch.cuda.current_stream(self.device))
            with torch.cuda.stream(s):
                try:
                    self._decode_body(B)
                except K.Q40Error:
                    if not (fused and self.max_cluster == 16):
                        raise
                    # this device cannot schedule 16-CTA clusters: use the portable size
                    self.max_cluster = 8
                    self._decode_body(B)
            key = self._graph_key(B)              # with what the warm-up run has found out about the device
            torch.cuda.current_stream(self.device).wait_stream(s)
            torch.cuda.synchronize(self.device)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                self._decode_body(B)
            self._graphs[key] = g, self._chained.get(B)
            if self.greedy_feedback:
                # capture itself executes nothing
                self._pos_dev[:B] -= 1
                self._tok_dev[:B].copy_(tok_saved)
        g, self._chained[B] = self._graphs[key]
        g.replay()
        self._count_launches(B, fused)
        if self._lm_head_q4 is not None and fused:      # only narrow steps compute with it
            return self._bufs[B]["logits_pad"][:, :self.params.vocab_size]
        return self._bufs[B]["logits"]

    def _graph_key(self, B):
        """What decides the launches of a step of B branches."""
        return (B, self.greedy_feedback, self.use_fused, self.use_pdl, self.max_cluster, self.use_stream,
                self.use_tiled, self.use_fused_attn, self.fused_attn_max_width, self.stream_smem_budget,
                self.use_fused_tail, self.use_tiled_tc, self.use_tp_fused_allreduce, self.use_chain, self.narrow_max)

    def _count_launches(self, B, fused):
        """launches_per_step of the step just enqueued."""
        if fused and self._chained.get(B):
            self.launches_per_step = 2
            return
        per_layer = (5 if self._fused_attn_for(B) else 6) if fused else (8 if self._silu_pair(B, self.layers[0].feed_forward) else 9)
        self.launches_per_step = self.params.n_layers * per_layer + (2 if self._narrow(B) else 1) + (not fused and self._fused_tail(B))


def random_init_(model: Transformer, seed: int = 0, std: float = 0.02) -> None:
    """Fill a model with N(0, std^2) weights quantised on the device by the library's own
    packer (norm weights = 1): the synthetic stand-in for a CodeLlama checkpoint converted
    by the reference's fp16_to_int4.py (which stores quantize_q40(W.t()) per linear)."""
    dev = model.device
    g = torch.Generator(device=dev).manual_seed(seed)
    p = model.params

    def fill(lin: LinearQ4_0, in_f, out_f):
        wt = (torch.randn((in_f, out_f), generator=g, device=dev, dtype=torch.float32) * std).to(DTYPE)
        q, s = K.quantize_q40(wt, GROUP_SIZE)       # [K, N] row-major: groups along N
        lin.w, lin.s, lin.shape = q, s.view(-1), (out_f, in_f)

    for layer in model.layers:
        att, ff = layer.attention, layer.feed_forward
        H, Hkv, D = model._H, model._Hkv, model._D
        fill(att.wq, p.dim, H * D)
        fill(att.wk, p.dim, Hkv * D)
        fill(att.wv, p.dim, Hkv * D)
        fill(att.wo, H * D, p.dim)
        fill(ff.w1, p.dim, ff.hidden_dim)
        fill(ff.w3, p.dim, ff.hidden_dim)
        fill(ff.w2, ff.hidden_dim, p.dim)
        for n in (layer.attention_norm, layer.ffn_norm):
            n.weight = nn.Parameter(torch.ones(p.dim, dtype=DTYPE, device=dev), requires_grad=False)
    model.norm.weight = nn.Parameter(torch.ones(p.dim, dtype=DTYPE, device=dev), requires_grad=False)
    emb = (torch.randn((p.vocab_size, p.dim), generator=g, device=dev) * std).to(DTYPE)
    out = (torch.randn((p.vocab_size, p.dim), generator=g, device=dev) * std).to(DTYPE)
    model.tok_embeddings = nn.Embedding.from_pretrained(emb, freeze=True)
    model.output = nn.Linear(p.dim, p.vocab_size, bias=False, device=dev, dtype=DTYPE)
    model.output.weight = nn.Parameter(out, requires_grad=False)
