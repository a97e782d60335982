// Shared-prefix stage of tree/speculative decode attention.
//
// All B branches attend to the same prompt K/V.  Instead of letting every (branch, head)
// CTA re-read the prefix, the queries of all branches (times the GQA group) of one kv head
// are stacked as the M dimension of a tensor-core product: a CTA loads a 64-key tile of the
// prefix once (cp.async, double buffered, 16 KB of K + 16 KB of V) and applies it to up to
// 128 query rows with mma.m16n8k16 (S = Q K^T, online softmax in fp32 in the log2 domain,
// O += P V).  The prefix is split across CTAs flash-decoding style; each CTA writes its
// un-normalised partial (m, l, O) per row to a scratch buffer, and the per-branch kernel
// (attn_branch.cu) folds those partials into the result after walking the branch's private
// suffix pages.  This is the computation the reference's chunk_attn was aiming for
// (triton_kernels.py:1150-1231) and what its model does by materialising
// cat(prompt.expand(B), suffix) for SDPA (hf_model_q40_kv_shared.py:375-376, 405).
//
// Algorithmic traffic: prefix K/V once per (kv head, row block); Q and the partials are
// small next to it.  What bounds it: a warp's chain of MMAs and softmax per tile (2.1 us, a quarter where four warps share it; see
// attn_tile.cuh), start, first tile and partials around it.
#include <climits>
#include <mutex>

#include "attn_tile.cuh"

namespace q40 {

struct PrefixArgs {
  const __half* q;    // branch b, head h at q + b*q_stride + h*D
  int64_t q_stride;
  const __half* pk;   // key t of kv head h at pk + t*key_stride + h*head_stride
  const __half* pv;
  float* pm;          // [nsp][B*H]
  float* pl;
  float* po;          // [nsp][B*H][D]
  int64_t key_stride, head_stride;   // elements between consecutive keys / kv heads of pk, pv
  const int32_t* prefix_len_dev;     // optional device scalar overriding prefix_len (<= prefix_len)
  int B, H, Hkv, prefix_len, keys_per_split;
  float scale_log2;
  const __half* cos_tbl;             // ROT: q is rotated here, at its branch's position
  const __half* sin_tbl;
  const int32_t* pos;
  int n_pos;
};

// grid: (nsp, Hkv, row blocks); block: NWARPS*32 threads, 16 query rows per KW warps, which share the keys of a tile.
template <int NWARPS, int KW, bool ROT>
__global__ void __launch_bounds__(NWARPS * 32)
attn_prefix_kernel(const PrefixArgs a) {
  constexpr int D = ATTN_D;
  constexpr int RB = NWARPS / KW * 16, KEYS = TILE_KEYS / KW;
  constexpr int NT = NWARPS * 32;
  extern __shared__ __align__(128) unsigned char smem[];
  // [Q rows][stage][K tile | V tile]
  const uint32_t sbase = smem_u32(smem);
  asm volatile("griddepcontrol.wait;" ::: "memory");               // nothing of the previous launch is read before it is done
  // the branch kernel behind this one starts when that holds for all of these CTAs, and walks its own keys beside them
  asm volatile("griddepcontrol.launch_dependents;");

  const int sp = blockIdx.x, hk = blockIdx.y, rblk = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rep = a.H / a.Hkv;
  const int rows = a.B * rep;                 // query rows of this kv head
  const int row0 = rblk * RB;
  const int plen = a.prefix_len_dev ? min(max(a.prefix_len_dev[0], 0), a.prefix_len) : a.prefix_len;
  const int k_begin = sp * a.keys_per_split;
  const int k_end = min(plen, k_begin + a.keys_per_split);
  const int ntiles = (k_end > k_begin) ? (k_end - k_begin + TILE_KEYS - 1) / TILE_KEYS : 0;

  const uint32_t stages = sbase + RB * TILE_ROW_BYTES;
  auto load = [&](int tile, int stage) {
    const int key0 = k_begin + tile * TILE_KEYS;
    const uint32_t kdst = stages + stage * 2 * TILE_BYTES;
    const int64_t off = (int64_t)key0 * a.key_stride + (int64_t)hk * a.head_stride;
    load_tile<NT>(kdst, kdst + TILE_BYTES, a.pk + off, a.pv + off, a.key_stride, a.key_stride, k_end - key0, tid);
  };
  // ---- Q rows -> shared (swizzled) -> A fragments in registers, with the first tile on its way ----
  for (int idx = tid; !ROT && idx < RB * 16; idx += NT) {
    const int r = idx >> 4, ch = idx & 15;
    const int gr = row0 + r;
    const bool ok = gr < rows;
    const int b = ok ? gr / rep : 0, j = ok ? gr % rep : 0;
    const __half* src = a.q + (int64_t)b * a.q_stride + (hk * rep + j) * D + ch * 8;
    cp_async16(sbase + tile_off(r, ch), src, ok);
  }
  cp_async_commit();
  if (ntiles > 0) load(0, 0);
  cp_async_commit();
  if constexpr (ROT) {
    // eight dims of a row and the eight 64 further
#pragma unroll
    for (int i = 0; i < RB * 8 / NT; ++i) {
      const int idx = tid + i * NT, r = idx >> 3, ch = idx & 7, gr = row0 + r;
      uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
      if (gr < rows) {
        const int b = gr / rep, j = gr % rep;
        const __half* src = a.q + (int64_t)b * a.q_stride + (hk * rep + j) * D + ch * 8;
        const int64_t at = (int64_t)min(max(a.pos[b], 0), a.n_pos - 1) * 64 + ch * 8;
        lo = *reinterpret_cast<const uint4*>(src);
        hi = *reinterpret_cast<const uint4*>(src + 64);
        rotate_dims(lo, hi, __ldg(reinterpret_cast<const uint4*>(a.cos_tbl + at)), __ldg(reinterpret_cast<const uint4*>(a.sin_tbl + at)));
      }
      *reinterpret_cast<uint4*>(smem + tile_off(r, ch)) = lo;
      *reinterpret_cast<uint4*>(smem + tile_off(r, ch + 8)) = hi;
    }
  }
  cp_async_wait<1>();
  __syncthreads();
  WarpRows w;
  w.init();
  const int wrow = warp / KW * 16, kfirst = warp % KW * KEYS;   // of this warp
  w.load_q(sbase, wrow, lane);

  const bool any_row = row0 + wrow < rows;      // a warp without rows only helps to load
  for (int tile = 0; tile < ntiles; ++tile) {
    const int stage = tile & 1;
    if (tile + 1 < ntiles) load(tile + 1, stage ^ 1);
    cp_async_commit();
    cp_async_wait<1>();   // the tile for this iteration has landed
    __syncthreads();
    const uint32_t kt = stages + stage * 2 * TILE_BYTES + kfirst * TILE_ROW_BYTES, vt = kt + TILE_BYTES;
    const int n = k_end - k_begin - tile * TILE_KEYS - kfirst;
    if (any_row && n > 0) {
      if (n >= KEYS) w.template step<false, KEYS>(kt, vt, a.scale_log2, 0, 0, lane);
      else w.template step<true, KEYS>(kt, vt, a.scale_log2, n, n, lane);
    }
    __syncthreads();  // all warps are done with this stage before it is refilled
  }
  cp_async_wait<0>();

  // ---- write the partial (m, l, O) of rows g and g+8 ----
  w.finish();
  const int64_t total_rows = (int64_t)a.B * a.H;
  if constexpr (KW > 1) {
    // the warps of a row meet in the tiles' memory; eight threads a row, 16 dims each
    constexpr int LD = D + 4;
    float *so = reinterpret_cast<float*>(smem), *sm = so + KW * RB * LD, *sl = sm + KW * RB;
    __syncthreads();                                  // (no tile: the queries are still being read)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int at = warp % KW * RB + wrow + g + r * 8;
      if (t == 0) { sm[at] = w.m[r]; sl[at] = w.l[r]; }
#pragma unroll
      for (int dt = 0; dt < 16; ++dt) *reinterpret_cast<float2*>(so + at * LD + dt * 8 + 2 * t) = make_float2(w.o[dt][2 * r], w.o[dt][2 * r + 1]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RB * 8 / NT; ++i) {
      const int r = (tid + i * NT) >> 3, part = tid & 7, gr = row0 + r;
      if (gr >= rows) continue;
      float M = -CUDART_INF_F, l = 0.f, f[KW];
#pragma unroll
      for (int k = 0; k < KW; ++k) M = fmaxf(M, sm[k * RB + r]);
#pragma unroll
      for (int k = 0; k < KW; ++k) {                  // no finite score: sums and outputs are 0
        f[k] = M > -CUDART_INF_F ? ex2(sm[k * RB + r] - M) : 1.f;
        l = fmaf(sl[k * RB + r], f[k], l);
      }
      const int64_t ridx = (int64_t)sp * total_rows + (int64_t)(gr / rep) * a.H + hk * rep + gr % rep;
      if (part == 0) { a.pm[ridx] = M; a.pl[ridx] = l; }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < KW; ++k) {
          const float4 x = *reinterpret_cast<const float4*>(so + (k * RB + r) * LD + 32 * c + 4 * part);
          v.x = fmaf(x.x, f[k], v.x); v.y = fmaf(x.y, f[k], v.y); v.z = fmaf(x.z, f[k], v.z); v.w = fmaf(x.w, f[k], v.w);
        }
        *reinterpret_cast<float4*>(a.po + ridx * D + 32 * c + 4 * part) = v;
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int gr = row0 + wrow + g + r * 8;
      if (gr >= rows) continue;
      const int b = gr / rep, j = gr % rep;
      const int64_t ridx = (int64_t)sp * total_rows + (int64_t)b * a.H + hk * rep + j;
      if (t == 0) { a.pm[ridx] = w.m[r]; a.pl[ridx] = w.l[r]; }
      float* dst = a.po + ridx * D;
#pragma unroll
      for (int dt = 0; dt < 16; ++dt)
        *reinterpret_cast<float2*>(dst + dt * 8 + 2 * t) = make_float2(w.o[dt][2 * r], w.o[dt][2 * r + 1]);
    }
  }
}

// `own`: keys that the branches have of their own in front of a head, about; 0: not known
static int prefix_splits(int B, int H, int Hkv, int prefix_len, int64_t own) {
  const int rep = H / Hkv;
  const int rows = B * rep;
  const int rblocks = (rows + 127) / 128;
  const int tiles = (prefix_len + TILE_KEYS - 1) / TILE_KEYS;
  // CTAs per SM to aim for: two for the 64-row variant (128 threads; measured best for 2048 keys x 64
  // rows), one for the 128-row variant; never round up past whole waves (a 149th CTA doubles the time
  // of one SM)
  // ... one, too, where the branches' own keys are so many that the pass is over long before they are: it then gets by with half of the
  // partials and leaves SMs to them (64 branches of 256 own keys behind 512: 52.0 us with two, 47.6; of up to 256 35.0 and 32.0, 34 behind 471 18.5
  // and 17.6; below some times the prefix one is slower: 10 of up to 64 behind 2048 9.1 and 11.1; and with fewer than eight tiles: 64
  // of up to 100 behind 300 15.1 and 15.8)
  const bool hidden = tiles >= 8 && own > 6 * (int64_t)prefix_len;
  const int per_sm = rows <= 64 && !hidden ? 2 : 1;
  int want = (148 * per_sm) / (Hkv * rblocks);
  if (want < 1) want = 1;
  if (want > tiles) want = tiles;
  // How many tiles a split has.  A tile costs it 1.0 us (1.9 with eight warps, 0.8 where two warps share a row's keys, 0.56 where four do); the merge has 16 splits of a row on their way at once (8 where a row has two
  // warps) and reads further ones one by one, 0.07 us each, more behind many own keys; a second CTA on an SM costs 2.3 us that matter less the longer splits are.  Us by splits, 8 query heads a kv head:
  // 1 kv head, 1 branch, 2048 keys 16 splits 4.5, 32 6.5; 8192 keys 16 8.0, 32 8.1, 128 12.8; 32768 keys 16 21.4, 64 12.6, 256 24.4; 8 kv heads
  // x 4, 4 branches, 2048 keys 16 6.2, 32 8.7; 32768 keys 16 31.6, 32 27.9.  Before warps shared tiles, over 448 sizes of 1 to 32 kv heads and 512 to
  // 32768 keys, 5 % less time than with as many splits as SMs take, four of them 3 to 9 % more (1 kv head x 4, 34 branches, 8192 keys 15.9 and
  // 17.3).  The line is that of tiles that no warps share: up to 16 rows it has more splits than are best from 8192 keys on (1 kv head, 8192 keys 43, 9.4)
  int best = tiles, least = INT_MAX;
  for (int per = (tiles + want - 1) / want;; ++per) {
    const int n = (tiles + per - 1) / per;                  // every split is non-empty
    const int cost = 14 * per + (n > 16 ? n - 16 : 0) + (n * Hkv * rblocks > 148 ? 32 / per : 0);
    if (cost < least) { least = cost; best = n; }
    if (n <= 16) return best;
  }
}

// pa.prefix_len is the (maximum) prefix length the grid is sized for
static int launch_prefix(PrefixArgs& pa, int nsp, cudaStream_t st) {
  const int tiles = (pa.prefix_len + TILE_KEYS - 1) / TILE_KEYS;
  pa.keys_per_split = ((tiles + nsp - 1) / nsp) * TILE_KEYS;
  const int rep = pa.H / pa.Hkv, rows = pa.B * rep;
  const auto launch = [&](std::atomic<uint64_t>& ready, auto kern, int warps, int kw) {
    const int rb = warps / kw * 16;
    // the Q rows, two stages of K and V; as much with shared tiles, so that no three CTAs crowd on an SM (20 branches, 200 own
    // keys: 19.3 us, 17.7 so)
    const size_t smem = (size_t)warps * 16 * TILE_ROW_BYTES + 4 * TILE_BYTES;
    const cudaError_t e = q40_allow_smem(ready, (const void*)kern, (int)smem);
    return e != cudaSuccess ? e : q40_launch_pdl(kern, dim3(nsp, pa.Hkv, (rows + rb - 1) / rb), dim3(warps * 32), smem, st, pa);
  };
  static std::atomic<uint64_t> ready[8];
  const bool rot = pa.cos_tbl != nullptr;
  cudaError_t e;
  // Warps that would have no rows take a part of each tile's keys: up to 16 rows all four, up to 32 two a row where splits have more than one tile
  // (half of one tile is what the merge of the warps takes again).  The same with and without rotation, whose results are the same bits.  Us with one
  // warp a row and so, with the branch pass: 10 branches behind 2048 keys 11.6 and 9.9, 2 behind 70 5.1 and 4.5; rotating, 5 behind 512 8.9 and 8.5, 10
  // 9.6 and 9.1, 16 10.6 and 9.9; 17 behind 2048 13.7 and 11.6, behind 600 9.1 and 8.4; but rotating, 20 behind 512 (eight splits) 11.3 and 11.6
  if (rows <= 16) e = rot ? launch(ready[0], attn_prefix_kernel<4, 4, true>, 4, 4) : launch(ready[1], attn_prefix_kernel<4, 4, false>, 4, 4);
  else if (rows <= 32 && pa.keys_per_split > TILE_KEYS)
    e = rot ? launch(ready[2], attn_prefix_kernel<4, 2, true>, 4, 2) : launch(ready[3], attn_prefix_kernel<4, 2, false>, 4, 2);
  else if (rows <= 64) e = rot ? launch(ready[4], attn_prefix_kernel<4, 1, true>, 4, 1) : launch(ready[5], attn_prefix_kernel<4, 1, false>, 4, 1);
  else e = rot ? launch(ready[6], attn_prefix_kernel<8, 1, true>, 8, 1) : launch(ready[7], attn_prefix_kernel<8, 1, false>, 8, 1);
  if (e != cudaSuccess) return (int)e;
  return Q40_OK;
}

}  // namespace q40

extern "C" size_t q40_attn_shared_prefix_workspace_bytes(int B, int H, int D, int prefix_len) {
  if (B <= 0 || H <= 0 || D != q40::ATTN_D || prefix_len <= 0) return 0;
  // the split count depends on Hkv; Hkv = 1 with 128-row blocks gives the largest count
  const int tiles = (prefix_len + q40::TILE_KEYS - 1) / q40::TILE_KEYS;
  const int max_sp = tiles < 296 ? tiles : 296;
  return (size_t)max_sp * B * H * (D + 2) * sizeof(float);
}

extern "C" int q40_attn_shared_prefix(const void* q, const void* prefix_k, const void* prefix_v,
                                      int prefix_len, int64_t prefix_key_stride,
                                      int64_t prefix_head_stride, const void* page_tbl, int idx_bytes,
                                      int64_t tbl_stride, const int32_t* seq_lens, const void* kpool,
                                      const void* vpool, void* o, int P, int B, int Lmax, int H, int Hkv,
                                      int D, int page_size, void* workspace, size_t workspace_bytes,
                                      void* stream) {
  using namespace q40;
  if (!q || !o) return Q40_E_NULL;
  if (D != ATTN_D) return Q40_E_UNSUPPORTED;
  if (B < 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0 || prefix_len < 0 || Lmax < 0 || P < 0 || page_size <= 0)
    return Q40_E_SHAPE;
  if (idx_bytes != 2 && idx_bytes != 4) return Q40_E_UNSUPPORTED;
  if (prefix_len > 0 && (!prefix_k || !prefix_v)) return Q40_E_NULL;
  if (prefix_len > 0 && (prefix_key_stride % 8 != 0 || prefix_head_stride % 8 != 0)) return Q40_E_ALIGN;
  if (Lmax > 0 && (!page_tbl || !kpool || !vpool || P == 0)) return Q40_E_NULL;
  if (Lmax > 0 && tbl_stride < (Lmax + page_size - 1) / page_size) return Q40_E_SHAPE;
  if (B == 0) return Q40_OK;
  if (!q40_aligned(q, 16) || !q40_aligned(prefix_k, 16) || !q40_aligned(prefix_v, 16) ||
      !q40_aligned(kpool, 16) || !q40_aligned(vpool, 16))
    return Q40_E_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows_total = (int64_t)B * H;

  BranchArgs br{};
  br.q = (const __half*)q; br.q_stride = (int64_t)H * D; br.k = (const __half*)kpool; br.v = (const __half*)vpool; br.o = (__half*)o;
  br.tbl = page_tbl; br.tbl_stride = tbl_stride; br.seq_lens = seq_lens;
  br.L = Lmax; br.H = H; br.Hkv = Hkv; br.P = P; br.page_size = page_size;
  br.scale_log2 = attn_scale_log2(D);

  // The first of two launches leaves the other its partial results in the scratch.  Callers that share one, as threads on one stream may, enqueue both before
  // the next does (a lock from Python costs 0.3 us of a call)
  static std::mutex turns[64];
  std::unique_lock<std::mutex> turn;
  if (prefix_len > 0) {
    turn = std::unique_lock<std::mutex>(turns[(uintptr_t)workspace / 512 % 64]);
    // lengths are on the device; Lmax is taken for twice their mean up to 256 keys.  A wider table is more likely one that branches can grow
    // into (64 branches of 64 keys with room for 4096, behind 8192: 71 us if they count as 2048 each, 47), and long rows gain nothing (34
    // branches of 1000 behind 512: 89.7 and 89.9).  (So Lmax may move a result's last bits, by another number of splits, behind 449 keys and more)
    const int nsp = prefix_splits(B, H, Hkv, prefix_len, Lmax <= 256 ? (int64_t)B * Lmax / 2 : 0);
    const size_t need = (size_t)nsp * rows_total * (D + 2) * sizeof(float);
    if (!workspace || workspace_bytes < need) return Q40_E_WORKSPACE;
    if (!q40_aligned(workspace, 16)) return Q40_E_ALIGN;
    float* po = (float*)workspace;
    float* pm = po + (size_t)nsp * rows_total * D;
    float* pl = pm + (size_t)nsp * rows_total;
    PrefixArgs pa{};
    pa.q = (const __half*)q; pa.q_stride = (int64_t)H * D; pa.pk = (const __half*)prefix_k; pa.pv = (const __half*)prefix_v;
    pa.pm = pm; pa.pl = pl; pa.po = po;
    pa.key_stride = prefix_key_stride; pa.head_stride = prefix_head_stride;
    pa.B = B; pa.H = H; pa.Hkv = Hkv; pa.prefix_len = prefix_len;
    pa.scale_log2 = br.scale_log2;
    int rc = launch_prefix(pa, nsp, st);
    if (rc != Q40_OK) return rc;
    br.pm = pm; br.pl = pl; br.po = po; br.nsp = nsp; br.beside_prefix = 1;
  }
  // Lmax == 0: the branch kernel only merges the prefix partials
  const int mode = (Lmax == 0) ? 0 : (idx_bytes == 2 ? 1 : 2);
  if (Lmax == 0) { br.seq_lens = nullptr; br.L = 0; }
  return launch_branch(br, mode, B, prefix_len, st);
}

// cos_tbl != NULL: q and cur_k are rotated and the token is appended (q40_attn_tree_step)
static int tree_decode(const void* q, int64_t q_stride, const void* prefix_k, const void* prefix_v, int max_prefix_len,
                       const int32_t* prefix_len_dev, int64_t prefix_key_stride, int64_t prefix_head_stride, const void* cache_kq,
                       const void* cache_ks, const void* cache_vq, const void* cache_vs, int max_t, const int32_t* pos_dev, const void* cur_k,
                       const void* cur_v, int64_t cur_stride, const void* cos_tbl, const void* sin_tbl, int n_pos, void* o, int B, int H,
                       int Hkv, int D, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace q40;
  if (!q || !o || !prefix_k || !prefix_v || !prefix_len_dev || !pos_dev) return Q40_E_NULL;
  if (!cache_kq || !cache_ks || !cache_vq || !cache_vs) return Q40_E_NULL;
  if ((cur_k == nullptr) != (cur_v == nullptr)) return Q40_E_NULL;
  if (D != ATTN_D) return Q40_E_UNSUPPORTED;
  if (B < 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0 || max_prefix_len <= 0 || max_t <= 0) return Q40_E_SHAPE;
  if (prefix_key_stride % 8 != 0 || prefix_head_stride % 8 != 0 || cur_stride % 8 != 0 || q_stride % 8 != 0)
    return Q40_E_ALIGN;
  if (q_stride < (int64_t)H * D) return Q40_E_SHAPE;
  if (B == 0) return Q40_OK;
  if (!q40_aligned(q, 16) || !q40_aligned(prefix_k, 16) || !q40_aligned(prefix_v, 16) ||
      !q40_aligned(cache_kq, 16) || !q40_aligned(cache_vq, 16) || !q40_aligned(cur_k, 16) ||
      !q40_aligned(cur_v, 16))
    return Q40_E_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows_total = (int64_t)B * H;
  const int nsp = prefix_splits(B, H, Hkv, max_prefix_len, 0);
  const size_t need = (size_t)nsp * rows_total * (D + 2) * sizeof(float);
  if (!workspace || workspace_bytes < need) return Q40_E_WORKSPACE;
  if (!q40_aligned(workspace, 16)) return Q40_E_ALIGN;
  float* po = (float*)workspace;
  float* pm = po + (size_t)nsp * rows_total * D;
  float* pl = pm + (size_t)nsp * rows_total;
  PrefixArgs pa{};
  pa.q = (const __half*)q; pa.q_stride = q_stride; pa.pk = (const __half*)prefix_k; pa.pv = (const __half*)prefix_v;
  pa.pm = pm; pa.pl = pl; pa.po = po;
  pa.key_stride = prefix_key_stride; pa.head_stride = prefix_head_stride;
  pa.prefix_len_dev = prefix_len_dev;
  pa.B = B; pa.H = H; pa.Hkv = Hkv; pa.prefix_len = max_prefix_len;
  pa.scale_log2 = attn_scale_log2(D);
  pa.cos_tbl = (const __half*)cos_tbl; pa.sin_tbl = (const __half*)sin_tbl; pa.n_pos = n_pos; pa.pos = pos_dev;
  int rc = launch_prefix(pa, nsp, st);
  if (rc != Q40_OK) return rc;
  BranchRotArgs br{};
  br.cos_tbl = pa.cos_tbl; br.sin_tbl = pa.sin_tbl; br.n_pos = n_pos;
  br.q = (const __half*)q; br.q_stride = q_stride; br.o = (__half*)o;
  br.H = H; br.Hkv = Hkv; br.L = max_t;
  br.scale_log2 = pa.scale_log2;
  br.pm = pm; br.pl = pl; br.po = po; br.nsp = nsp; br.beside_prefix = 1;
  br.kq = (const int8_t*)cache_kq; br.ksc = (const __half*)cache_ks;
  br.vq = (const int8_t*)cache_vq; br.vsc = (const __half*)cache_vs;
  br.pos = pos_dev; br.prefix_len = prefix_len_dev; br.max_t = max_t;
  br.cur_k = (const __half*)cur_k; br.cur_v = (const __half*)cur_v; br.cur_stride = cur_stride;
  return launch_branch_q4(br, B, st);
}

extern "C" int q40_attn_tree_decode(const void* q, int64_t q_stride, const void* prefix_k, const void* prefix_v,
                                    int max_prefix_len, const int32_t* prefix_len_dev,
                                    int64_t prefix_key_stride, int64_t prefix_head_stride,
                                    const void* cache_kq, const void* cache_ks, const void* cache_vq,
                                    const void* cache_vs, int max_t, const int32_t* pos_dev,
                                    const void* cur_k, const void* cur_v, int64_t cur_stride, void* o, int B,
                                    int H, int Hkv, int D, void* workspace, size_t workspace_bytes,
                                    void* stream) {
  return tree_decode(q, q_stride, prefix_k, prefix_v, max_prefix_len, prefix_len_dev, prefix_key_stride, prefix_head_stride, cache_kq,
                     cache_ks, cache_vq, cache_vs, max_t, pos_dev, cur_k, cur_v, cur_stride, nullptr, nullptr, 0, o, B, H, Hkv, D,
                     workspace, workspace_bytes, stream);
}

// A launch of its own for rotation and append (rope_kv_append_kernel), and the wait for it, took 2.5 us a layer and step of 10 branches
// and 3.8 of 100
extern "C" int q40_attn_tree_step(const void* q, int64_t q_stride, const void* k, const void* v, int64_t kv_stride, const void* prefix_k,
                                  const void* prefix_v, int max_prefix_len, const int32_t* prefix_len_dev, int64_t prefix_key_stride,
                                  int64_t prefix_head_stride, void* cache_kq, void* cache_ks, void* cache_vq, void* cache_vs, int max_t,
                                  const int32_t* pos_dev, const void* cos_tbl, const void* sin_tbl, int n_pos, void* o, int B, int H,
                                  int Hkv, int D, void* workspace, size_t workspace_bytes, void* stream) {
  if (!k || !v || !cos_tbl || !sin_tbl) return Q40_E_NULL;
  if (n_pos <= 0 || kv_stride < (int64_t)Hkv * D) return Q40_E_SHAPE;
  if (!q40_aligned(cos_tbl, 16) || !q40_aligned(sin_tbl, 16) || !q40_aligned(cache_ks, 4) || !q40_aligned(cache_vs, 4)) return Q40_E_ALIGN;
  return tree_decode(q, q_stride, prefix_k, prefix_v, max_prefix_len, prefix_len_dev, prefix_key_stride, prefix_head_stride, cache_kq,
                     cache_ks, cache_vq, cache_vs, max_t, pos_dev, k, v, kv_stride, cos_tbl, sin_tbl, n_pos, o, B, H, Hkv, D, workspace,
                     workspace_bytes, stream);
}
