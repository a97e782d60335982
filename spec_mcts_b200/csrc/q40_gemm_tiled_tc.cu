// Q4_0 dequant-matmul for batches above 8 rows on the 5th-generation tensor cores, reading the
// TILED copy of the weights (the format of q40_gemv_tiled.cu: [span of 256 columns][16 k rows] steps of
// 2176 contiguous bytes), so that the decode step's wide path and its narrow path share one weight copy.
//
// Swap-AB as in q40_gemm_tc.cu: the output features are the M dimension of the tcgen05.mma accumulators in tensor memory, the
// batch rows the N dimension (padded to a multiple of 16).  Two kernels: pairs of CTAs (q40_gemm_pair_tc.cu), and, for
// 129 rows or more of matrices with few tiles, the one below, one CTA per 128 features x up to 256 rows with the k range split
// over a cluster.  In both
//   * elected threads stream weights and activations into rings of shared-memory stages by bulk and tensor copies that
//     complete on mbarriers;
//   * dequantiser warps turn a stage's nibbles into the reference's operand value fp16(code * scale)
//     (triton_kernels.py:444-445) and write it as the A operand straight into TENSOR MEMORY: the tiled format hands every lane the
//     four A-fragment words of mma.m16n8k16 (rows g and g + 8 at four consecutive k per word), and that is the
//     register layout of tcgen05.st.16x256b, so a warp stores two 16-row tiles x 64 k with two instructions and the
//     dequantised weights never touch shared memory (through shared memory they cost 64 KB of traffic per
//     k block of 256 features, more than the operands themselves);
//   * one thread issues the tcgen05.mma (A from tensor memory, B from the stage), in k order: a result depends on nothing but
//     the operands and the k split.
// Every mbarrier wait is bounded: on expiry the kernel records an error code, skips the remaining work, waits (bounded too) for
// its own copies and MMAs, frees its tensor memory and returns.
//
// Replaces matmul_q40_kernel (triton_kernels.py:357-469) for M > 8 when the caller holds tiled weights.
#include <cooperative_groups.h>

#include "q40_tc_common.cuh"

namespace cg = cooperative_groups;

namespace q40 {
namespace ttc {
namespace wide {

// The rows, which are the MMA's N, go up to 256, so that a k block is four large MMAs, and one accumulator of 128 features
// takes half of tensor memory; the other half holds NA = 8 A buffers.  The activations of a k block (32 KB at 256 rows) are
// read once per 128 features, which is what bounds a CTA's main loop (72 bytes a cycle at the MMAs' pace, more than an SM
// gets from L2).  Sixteen dequantiser warps are four sets of four (one warp per tensor-memory quadrant) that take the k
// blocks in turn; one thread issues all MMAs.  Rows are cut into equal chunks of at most 256 inside ONE launch (grid z);
// a tile that is not split along k goes from tensor memory to the output directly, otherwise the ranks of a cluster add
// their fp32 tiles in rank order.
// Microseconds for 144 / 256 rows, here and by pairs (one tile per pair, k not split): x 4096 x 4096 11.7 / 14.5 and 14.6 / 15.7;
// x 11008 x 4096 20.3 / 24.1 and 28.4 / 29.7; x 4096 x 11008 25.8 / 30.0 and 21.7 / 25.3.
constexpr int MAX_STAGES = 8;                   // block i owns the stage's barrier i % stages

struct Params {
  const uint8_t* bw[3];   // tiled streams of up to three matrices that share the activations
  __half* c[3];           // [M, ldc]
  int64_t ldc[3];
  int N[3], spans[3], nprob;
  int M, K, Mpad, rows_per_split, stages;
  int* err;               // device word, set non-zero when a bounded wait expired
};

// A wait ran out: the error word, and a wait (with a limit as well) for the copies still on their way, the last S of the
// `copied` k blocks at most: none may land in shared memory that this CTA has given back.  (The MMAs that were issued are
// waited for through the `done` barrier, which the issuing thread commits to, also after giving up.)
__device__ __noinline__ void give_up(int* err, uint32_t bar_full, int S, int copied) {
  q40_set_error(err);
  for (int i = max(0, copied - S); i < copied; ++i) mbar_wait(bar_full + 8 * (i % S), (uint32_t)((i / S) & 1));
}

constexpr int FEATS = 128;                      // features per CTA: half a span of the tiled format
constexpr int MAX_ROWS = 256;
constexpr int NA = 8;                           // A buffers: 32 columns of tensor memory each
constexpr int DSETS = 4;                        // dequantiser sets of four warps
constexpr int DQ_WARP0 = 4;                     // warp 0: copies, warp 1: MMA issue, warps 4..19: dequantise
constexpr int THREADS = (DQ_WARP0 + 4 * DSETS) * 32;
constexpr int HSTEP = 1024 + 64;                // half a step: two 64-column groups and their scales
constexpr int RAW_BYTES = 4 * HSTEP;
constexpr int RAW_PAD = 5120;                   // next multiple of 1024 (the B tile wants that alignment)
constexpr int A_COL0 = MAX_ROWS;

__global__ void __launch_bounds__(THREADS, 1)
gemm_tiled_wide_kernel(const Params p, const __grid_constant__ CUtensorMap amap) {
  extern __shared__ unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int pi = 0, span = blockIdx.x >> 1;
  const int half = blockIdx.x & 1;
  while (pi < p.nprob - 1 && span >= p.spans[pi]) { span -= p.spans[pi]; ++pi; }
  const int kb = blockIdx.y * p.rows_per_split;
  const int ke = min(p.K, kb + p.rows_per_split);
  const int nblk = (ke - kb) / BK;                           // host guarantees >= 1 and exact
  const int m0 = blockIdx.z * p.Mpad;                        // first batch row of this chunk
  const int rows = min(p.Mpad, p.M - m0);
  const int S = p.stages;
  const uint32_t b_bytes = (uint32_t)p.Mpad * 128u;          // B tile: Mpad rows x 64 k x 2 B
  const uint32_t stage_bytes = RAW_PAD + b_bytes;

  const uint32_t raw0 = smem_u32(smem_raw);
  const uint32_t ring = (raw0 + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (ring - raw0);
  const size_t ring_bytes = max((size_t)S * stage_bytes, ((size_t)p.Mpad * FEATS + 64) * 4);
  // full[s]: the stage's copies have landed; afull / mdone [i % NA]: the A operand of block i is written / the MMAs
  // of block i are complete (its stage and its A buffer may be refilled; S <= NA, so neither waiter can
  // miss a phase); done: all MMAs complete
  const uint32_t bar_full = ring + (uint32_t)ring_bytes, bar_afull = bar_full + 8 * MAX_STAGES;
  const uint32_t bar_mdone = bar_afull + 8 * NA, bar_done = bar_mdone + 8 * NA;
  unsigned char* tail = gbase + ring_bytes + 8 * MAX_STAGES + 16 * NA + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail);
  volatile int* s_failed = reinterpret_cast<volatile int*>(tail + 8);
  volatile int* s_copied = reinterpret_cast<volatile int*>(tail + 12);     // k blocks whose copies were requested

  if (tid == 0) {
    *s_failed = 0;
    for (int s = 0; s < MAX_STAGES; ++s) mbar_init(bar_full + 8 * s, 1);
    for (int s = 0; s < NA; ++s) { mbar_init(bar_afull + 8 * s, 4); mbar_init(bar_mdone + 8 * s, 1); }
    mbar_init(bar_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;");
  // the time that the launch in front takes, whose waits may run out, is not that of this one's waits
  if (warp != 0) asm volatile("griddepcontrol.wait;" ::: "memory");

  bool failed = false;
  if (warp == 0) {
    if (elect_one()) {
      const int ksteps = p.K / 16;
      const uint8_t* src = p.bw[pi] + ((int64_t)span * ksteps + kb / 16) * STEP_BYTES;
      auto weights = [&](int i, int s) {
#pragma unroll
        for (int st = 0; st < 4; ++st) {
          const uint8_t* step = src + (int64_t)(4 * i + st) * STEP_BYTES;
          const uint32_t dst = ring + s * stage_bytes + st * HSTEP;
          bulk_g2s(dst, step + half * 1024, 1024, bar_full + 8 * s);
          bulk_g2s(dst + 1024, step + 2048 + half * 64, 64, bar_full + 8 * s);
        }
      };
      // weights do not depend on the previous launch, the activations do
      const int first = min(S, nblk);
      for (int i = 0; i < first; ++i) {
        mbar_expect_tx(bar_full + 8 * i, RAW_BYTES + b_bytes);
        weights(i, i);
      }
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int i = 0; i < first; ++i)
        tma_2d(ring + i * stage_bytes + RAW_PAD, &amap, kb + i * BK, m0, bar_full + 8 * i);
      int i = first;
      for (; i < nblk; ++i) {
        const int s = i % S, j = i - S;                      // block j was the stage's last user
        if (!mbar_wait(bar_mdone + 8 * (j % NA), (uint32_t)((j / NA) & 1))) { failed = true; break; }
        mbar_expect_tx(bar_full + 8 * s, RAW_BYTES + b_bytes);
        tma_2d(ring + s * stage_bytes + RAW_PAD, &amap, kb + i * BK, m0, bar_full + 8 * s);
        weights(i, s);
      }
      *s_copied = i;
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | ((uint32_t)(p.Mpad >> 3) << 17) | ((uint32_t)(FEATS >> 4) << 24);
    if (elect_one()) {
      for (int i = 0; i < nblk; ++i) {
        const int ab = i % NA;
        // the dequantisers' arrival also covers the stage's copies, which they waited for
        if (!mbar_wait(bar_afull + 8 * ab, (uint32_t)((i / NA) & 1))) { failed = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t bd0 = kmajor_desc(ring + (i % S) * stage_bytes + RAW_PAD);
#pragma unroll
        for (int ks = 0; ks < BK / 16; ++ks)
          mma_ts(tmem, tmem + A_COL0 + ab * 32 + ks * 8, bd0 + (uint64_t)((ks * 32) >> 4), idesc,
                 (i > 0 || ks > 0) ? 1u : 0u);
        commit(bar_mdone + 8 * ab);
      }
      commit(bar_done);
    }
    __syncwarp();
  } else if (warp >= DQ_WARP0) {
    // warp = (set, quadrant): 32 feature rows = two 16-row tiles of one 64-column group, see above
    const int quad = warp & 3, dset = (warp - DQ_WARP0) >> 2;
    const int q = quad >> 1, t = lane & 3;
    const unsigned char* lane_w = gbase + (q * 32 + lane) * 16 + (quad & 1) * 8;
    const unsigned char* lane_s = gbase + 1024 + q * 32 + t * 8;
    for (int i = dset; i < nblk; i += DSETS) {
      const int s = i % S, ab = i % NA;
      // block i - S first: its MMAs free this block's A buffer (S <= NA), and the full barrier, which tells only odd
      // from even phases, has then left the phase of block i - S (the copies of different blocks land in any order)
      const int w = i - S;
      if (w >= 0 && !mbar_wait(bar_mdone + 8 * (w % NA), (uint32_t)((w / NA) & 1))) { failed = true; break; }
      if (!mbar_wait(bar_full + 8 * s, (uint32_t)((i / S) & 1))) { failed = true; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const size_t so = (size_t)s * stage_bytes;
      uint32_t r[2][16];
#pragma unroll
      for (int st = 0; st < 4; ++st) dequant_step(lane_w + so + st * HSTEP, lane_s + so + st * HSTEP, r, st);
      const uint32_t ta = tmem + ((uint32_t)(32 * quad) << 16) + A_COL0 + ab * 32;
      st_16x256b_x4(ta, r[0]);
      st_16x256b_x4(ta + (16u << 16), r[1]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_afull + 8 * ab);
    }
  }
  if (!mbar_wait(bar_done, 0) || failed) *s_failed = 1;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  failed = *s_failed != 0;
  if (failed && tid == 0) give_up(p.err, bar_full, S, *s_copied);

  const int nranks = (int)cluster.num_blocks();
  const int n0 = span * SPAN + half * FEATS;
  __half* c = p.c[pi] + (int64_t)m0 * p.ldc[pi] + n0;
  float* tile_f = reinterpret_cast<float*>(gbase);
  if (!failed && warp >= DQ_WARP0) {
    const int quad = warp & 3, dset = (warp - DQ_WARP0) >> 2;
    const int feat = 32 * quad + lane;                // MMA row = feature
    for (int ch = dset; ch < p.Mpad / 16; ch += DSETS) {
      uint32_t r[16];
      ld16(tmem + ((uint32_t)(32 * quad) << 16) + ch * 16, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (nranks > 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) tile_f[(ch * 16 + j) * FEATS + feat] = __uint_as_float(r[j]);
      } else {
        // a warp's store is 64 contiguous bytes of one row: whole sectors, no staging
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (ch * 16 + j < rows) c[(int64_t)(ch * 16 + j) * p.ldc[pi] + feat] = __float2half_rn(__uint_as_float(r[j]));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512));
  }
  if (nranks == 1) return;
  // split-K: rank r finishes the r-th slice of the (row, feature) pairs, adding the ranks' tiles in rank order
  const int rank = (int)cluster.block_rank();
  const int total = rows * FEATS;
  const int per = ((total / 4 + nranks - 1) / nranks) * 4;
  const int e0 = rank * per, e1 = min(total, e0 + per);
  if (!failed) {
    for (int e = e0 + tid * 4; e < e1; e += THREADS * 4) {
      float4 tt[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        tt[r] = (r < nranks) ? *reinterpret_cast<const float4*>(cluster.map_shared_rank(tile_f + e, r))
                             : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int r = 0; r < 8; ++r) { v.x += tt[r].x; v.y += tt[r].y; v.z += tt[r].z; v.w += tt[r].w; }
      __half2* dst = reinterpret_cast<__half2*>(c + (int64_t)(e / FEATS) * p.ldc[pi] + e % FEATS);
      dst[0] = __floats2half2_rn(v.x, v.y);
      dst[1] = __floats2half2_rn(v.z, v.w);
    }
  }
  cluster.sync();       // every rank has read the tiles: shared memory may go away
}

}  // namespace wide
}  // namespace ttc
}  // namespace q40

// How many clusters of (1, nsplit) CTAs with this much dynamic shared memory run at once (an answer is
// kept per device, split and padded row class; 0, not kept, when the runtime cannot tell).
static int wide_max_clusters(int mpad, int nsplit, size_t smem) {
  using namespace q40::ttc;
  static std::atomic<int> cache_all[16][9][17] = {};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* cached = dev < 16 ? &cache_all[dev][nsplit][mpad / 16] : nullptr;
  if (cached && cached->load(std::memory_order_relaxed)) return cached->load(std::memory_order_relaxed) - 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1024, nsplit, 1);
  cfg.blockDim = dim3(wide::THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = nsplit;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, wide::gemm_tiled_wide_kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  if (cached) cached->store(n + 1, std::memory_order_relaxed);
  return n;
}

// Argument rules that both entries share
static int tiled_tc_check(int nmat, const void* a, int64_t lda, const void* const* bw_tiled, void* const* c,
                          const int64_t* ldc, const int* n_cols, int M, int K, const int* err) {
  using namespace q40::ttc;
  if (!a || !bw_tiled || !c || !ldc || !n_cols || !err) return Q40_E_NULL;
  if (nmat < 1 || nmat > 3) return Q40_E_UNSUPPORTED;
  if (M < 1 || K <= 0 || K % BK != 0 || lda < K || lda % 8 != 0) return Q40_E_SHAPE;
  if (!q40_aligned(a, 16)) return Q40_E_ALIGN;
  for (int i = 0; i < nmat; ++i) {
    if (!bw_tiled[i] || !c[i]) return Q40_E_NULL;
    if (n_cols[i] <= 0 || n_cols[i] % SPAN != 0 || ldc[i] < n_cols[i] || ldc[i] % 2 != 0) return Q40_E_SHAPE;
    if (!q40_aligned(bw_tiled[i], 16) || !q40_aligned(c[i], 4)) return Q40_E_ALIGN;
  }
  return Q40_OK;
}

// C[M, N_i] = A[M, K] @ deq(B_i)[K, N_i] for 1..3 matrices given as TILED copies (q40_relayout_tiled),
// K % 64 == 0, N_i % 256 == 0, on tcgen05.  `err` is a device int the kernels set to 1 if one of their
// bounded waits expires (results are then undefined); the caller zeroes it beforehand and may read it after
// synchronising.
//
// Up to 128 rows: pairs of CTAs.  Above, the k range is cut where the kernel of this file would split it: by the largest
// power of two with which all tiles of the widest matrix run at once at one row chunk.  That is how
// q40_gemm_kn_tc splits k, and as all of them sum a range's products in order and then the ranges, a prompt pass of whole
// 256-row chunks has the same bits on either layout and by either kernel (the 512-row prompt pass of the 7B geometry with the
// split of least cost flips greedy tokens at near-ties).  The faster of the two kernels by their estimates is launched.
static int tiled_tc(int nmat, const void* a, int64_t lda, const void* const* bw_tiled, void* const* c, const int64_t* ldc,
                    const int* n_cols, int M, int K, int silu, void* workspace, size_t workspace_bytes, int* err, int use_pdl,
                    void* stream) {
  using namespace q40;
  using namespace q40::ttc;
  if (M <= 128)
    return q40_pair_gemm(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, 1, silu, workspace, workspace_bytes, 1e30, err, use_pdl, stream);
  // a grid has 65535 row chunks at most: more rows go in several launches
  constexpr int LAUNCH_ROWS = 65535 * wide::MAX_ROWS;
  if (M > LAUNCH_ROWS) {
    for (int64_t m0 = 0; m0 < M; m0 += LAUNCH_ROWS) {
      void* cm[3];
      for (int i = 0; i < nmat; ++i) cm[i] = (__half*)c[i] + m0 * ldc[i];
      const int rc = tiled_tc(nmat, (const __half*)a + m0 * lda, lda, bw_tiled, cm, ldc, n_cols,
                              M - m0 < LAUNCH_ROWS ? (int)(M - m0) : LAUNCH_ROWS, K, silu, workspace, workspace_bytes, err, use_pdl, stream);
      if (rc != Q40_OK) return rc;
    }
    return Q40_OK;
  }
  wide::Params p{};
  int spans = 0, widest = 0;
  for (int i = 0; i < nmat; ++i) {
    p.bw[i] = (const uint8_t*)bw_tiled[i];
    p.c[i] = (__half*)c[i]; p.ldc[i] = ldc[i];
    p.N[i] = n_cols[i]; p.spans[i] = n_cols[i] / SPAN;
    spans += p.spans[i];
    widest = p.spans[i] > widest ? p.spans[i] : widest;
  }
  EncodeTiledFn encode = ttc_encode_fn();
  if (!encode) return Q40_E_UNSUPPORTED;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return Q40_E_UNSUPPORTED;
  const int kblocks = K / BK;
  const int chunks = (M + wide::MAX_ROWS - 1) / wide::MAX_ROWS;
  p.nprob = nmat;
  p.M = M; p.K = K; p.Mpad = ((M + chunks - 1) / chunks + 15) / 16 * 16;
  p.err = err;
  // ring depth: what fits, at most MAX_STAGES; the fp32 tile of the epilogue reuses the ring
  const size_t stage_bytes = (size_t)wide::RAW_PAD + (size_t)p.Mpad * 128;
  const size_t fixed = 1024 /* alignment slack */ + 256 /* barriers, tmem slot, flag */;
  int stages = (int)((SMEM_MAX - fixed) / stage_bytes);
  if (stages > wide::MAX_STAGES) stages = wide::MAX_STAGES;
  if (stages < 2) return Q40_E_UNSUPPORTED;
  p.stages = stages;
  size_t ring_bytes = (size_t)stages * stage_bytes;
  const size_t tile_f = ((size_t)p.Mpad * wide::FEATS + 64) * 4;   // slices are rounded up to 4 elements per rank
  if (tile_f > ring_bytes) ring_bytes = tile_f;
  const size_t smem = fixed + ring_bytes;
  static std::atomic<uint64_t> ready;
  cudaError_t e = q40_allow_smem(ready, (const void*)wide::gemm_tiled_wide_kernel, SMEM_MAX);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return Q40_E_UNSUPPORTED; }
  int nsplit = 1, fit = sms;
  for (int ns = 2; ns <= 8; ns *= 2) {
    const int bps = (kblocks + ns - 1) / ns;
    if (bps < 4 || (ns - 1) * bps >= kblocks) continue;
    const int f = wide_max_clusters(p.Mpad, ns, smem);
    if (f >= widest * (SPAN / wide::FEATS)) { nsplit = ns; fit = f; }
  }
  const int tiles = spans * (SPAN / wide::FEATS), bps = (kblocks + nsplit - 1) / nsplit;
  // nanoseconds of the kernel of this file, for q40_pair_gemm to beat (it alone has SiLU)
  const double waves = (double)(((int64_t)tiles * chunks + fit - 1) / fit);
  const double ns_wide = silu ? 1e30 : waves * (bps * (270 + 0.33 * p.Mpad) + 4000 + 18.0 * p.Mpad);
  const int rc = q40_pair_gemm(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, (kblocks + bps - 1) / bps, silu, nullptr, 0, ns_wide, err, use_pdl, stream);
  if (rc != Q40_E_UNSUPPORTED || silu) return rc;
  // activations [M rows, K] as a 2-D tensor, box {64 k, Mpad rows}, 128-byte swizzle, zero fill beyond row M
  CUtensorMap amap;
  const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t gstride[1] = {(cuuint64_t)lda * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)p.Mpad};
  const cuuint32_t estr[2] = {1, 1};
  if (ttc_encode(encode, &amap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)a, gdim, gstride, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q40_E_UNSUPPORTED;
  p.rows_per_split = bps * BK;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles, nsplit, chunks);
  cfg.blockDim = dim3(wide::THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = nsplit;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, wide::gemm_tiled_wide_kernel, p, amap);
  if (e != cudaSuccess) return (int)e;
  return Q40_OK;
}

extern "C" int q40_gemm_tiled_tc_multi(int nmat, const void* a, int64_t lda, const void* const* bw_tiled,
                                       void* const* c, const int64_t* ldc, const int* n_cols, int M, int K, int* err,
                                       int use_pdl, void* stream) {
  const int rc = tiled_tc_check(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, err);
  return rc ? rc : tiled_tc(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, 0, nullptr, 0, err, use_pdl, stream);
}

// The same with scratch, and SiLU(A @ deq(B_0)) * (A @ deq(B_1)) in place of two products
extern "C" int q40_gemm_tiled_tc_ws(int nmat, const void* a, int64_t lda, const void* const* bw_tiled, void* const* c,
                                    const int64_t* ldc, const int* n_cols, int M, int K, int silu_mul, void* workspace,
                                    size_t workspace_bytes, int* err, int use_pdl, void* stream) {
  const int rc = tiled_tc_check(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, err);
  if (rc) return rc;
  if (silu_mul && (nmat != 2 || n_cols[0] != n_cols[1])) return Q40_E_UNSUPPORTED;
  if (q40_gemm_tiled_tc_ws_bytes(M) && (!workspace || workspace_bytes < q40_gemm_tiled_tc_ws_bytes(M))) return Q40_E_WORKSPACE;
  if (!q40_aligned(workspace, 16)) return Q40_E_ALIGN;
  return tiled_tc(nmat, a, lda, bw_tiled, c, ldc, n_cols, M, K, silu_mul != 0, workspace, workspace_bytes, err, use_pdl, stream);
}
