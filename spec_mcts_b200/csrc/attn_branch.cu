// Decode attention for one query token per branch over that branch's own keys: a
// contiguous [B,Hkv,L,D] cache or a paged pool (the packed Q4_0 cache: attn_branch_q4.cu).  Two, four or eight warps per row
// (branch, query head), one or two rows per CTA: see launch_branch_mode.  Calls that several heads of a kv head, or matrix instructions,
// make faster go to attn_branch_f16.cu, which says which.
//
// Eight lanes share a key: lane i owns dims 8i..8i+7 and 64+8i..64+8i+7 of the head (two 16-byte loads of K, two of
// V, each of which covers 128 contiguous bytes over the lanes), the partial dot products are summed with three shuffles, and every group of
// eight lanes keeps its own online-softmax state (running max, sum, 16 output dims) in
// fp32.  A row's groups (four per warp) are merged through shared memory at the end; the same
// merge can fold in partial results of a shared-prefix pass (see attn_prefix.cu), which is
// how the shared-prefix entry point finishes.
//
// Stands in for flash_attn_kernel2 / page_flash_attn_kernel2 of the reference
// (triton_kernels.py:559-647, 700-789), with fp32 softmax state and exact masking of the
// tail instead of the reference's fp16 state and multiple-of-32 length requirement.
#include <math_constants.h>

#include "attn_common.cuh"

namespace q40 {

// Page ids are looked up one iteration ahead of the keys they lead to, so that an iteration waits for one memory latency
// and not for two.
//
// A CTA has NW warps; WPR of them share a row (branch, head).  What bounds a row is latency (ids -> keys -> sums
// -> merge), so the split is the one that keeps the warps of all rows resident at once: see launch_branch_mode.

template <int MODE, int NW, int WPR, int U>    // U: keys per 8-lane group in flight
__global__ void __launch_bounds__(NW * 32, U > 2 ? 16 / NW : NW == 8 ? 3 : 5)
attn_branch_kernel(const BranchArgs a) {
  constexpr int D = ATTN_D;
  constexpr int RT = WPR * 32;                // threads of a row
  constexpr int NG = WPR * 4;                 // key groups of a row
  asm volatile("griddepcontrol.launch_dependents;");   // a dependent may start prefetching its weights
  // ... but nothing of the previous launch is read before it is done.  Behind a prefix pass, which lets this launch start only
  // when everything in front of it is done, that is the pass's results alone: the branch's own keys are read beside it
  if (!a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31;
  const int slot = (NW == WPR) ? 0 : (tid >> 5) / WPR;      // row of this CTA
  const int64_t bh = (int64_t)blockIdx.x * (NW / WPR) + slot;
  const int64_t rows = a.rows;
  if (bh >= rows) return;                     // whole warps; rows of a CTA meet at no barrier unless NW == WPR
  const int b = (int)(bh / a.H), h = (int)(bh % a.H);
  const int hk = h / (a.H / a.Hkv);
  const int tr = tid - slot * RT;             // thread of the row
  const int grp = tr >> 3, sub = tid & 7;
  // the 8 lanes that share a key; groups of one warp may run different numbers of iterations,
  // so every shuffle names only its own group
  const unsigned gmask = 0xffu << (lane & 24);

  const int len = a.seq_lens ? min(max(a.seq_lens[b], 0), a.L) : a.L;
  // first page ids.  They wait for the length: entries beyond it need not exist (the last row of a table that is a
  // column range of a wider one ends with the allocation).  Ids of every row but the last ahead of the length, by a
  // branch around two copies of these loads: 2 to 9 % slower on short rows, also without lengths
  const void* const table = MODE == 1 ? (const void*)(reinterpret_cast<const int16_t*>(a.tbl) + (int64_t)b * a.tbl_stride)
                                      : (const void*)(reinterpret_cast<const int32_t*>(a.tbl) + (int64_t)b * a.tbl_stride);
  int slots[U];
  if (MODE == 1 || MODE == 2) {
#pragma unroll
    for (int u = 0; u < U; ++u) slots[u] = (grp + u * NG < len) ? key_slot<MODE>(a, table, grp + u * NG) : 0;
  }

  __shared__ float sm_m[NW * 4], sm_l[NW * 4];
  __shared__ __align__(16) float sm_o[NW * 4][D];

  __half2 qh[8];                              // this lane's 16 query dims
  {
    const __half* qp = a.q + (int64_t)b * a.q_stride + h * D + sub * 8;
    *reinterpret_cast<uint4*>(qh) = *reinterpret_cast<const uint4*>(qp);
    *reinterpret_cast<uint4*>(qh + 4) = *reinterpret_cast<const uint4*>(qp + 64);
  }
  float m = -CUDART_INF_F, l = 0.f, o[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i] = 0.f;

  // first key of this head and branch, at this lane's dims
  const int64_t kv0 = (MODE == 0 ? (int64_t)(b * a.Hkv + hk) * a.L : (int64_t)hk * a.P) * D + sub * 8;
  for (int t0 = grp; t0 < len; t0 += NG * U) {
    uint4 kv[U][4];
    float s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u * NG;
      if (t < len) {
        const int64_t off = kv0 + (int64_t)(MODE == 0 ? t : slots[u]) * D;
        kv[u][0] = __ldg(reinterpret_cast<const uint4*>(a.k + off));
        kv[u][1] = __ldg(reinterpret_cast<const uint4*>(a.k + off + 64));
        kv[u][2] = __ldg(reinterpret_cast<const uint4*>(a.v + off));
        kv[u][3] = __ldg(reinterpret_cast<const uint4*>(a.v + off + 64));
      } else {
        kv[u][0] = kv[u][1] = kv[u][2] = kv[u][3] = make_uint4(0, 0, 0, 0);
      }
    }
    if (MODE == 1 || MODE == 2) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + (U + u) * NG;
        slots[u] = (t < len) ? key_slot<MODE>(a, table, t) : 0;
      }
    }
    float mnew = m;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const __half2* kh = reinterpret_cast<const __half2*>(&kv[u][0]);  // 8 half2 = 16 dims
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc = dot2(qh[i], kh[i], acc);
      acc += __shfl_xor_sync(gmask, acc, 1);
      acc += __shfl_xor_sync(gmask, acc, 2);
      acc += __shfl_xor_sync(gmask, acc, 4);
      s[u] = (t0 + u * NG < len) ? acc * a.scale_log2 : -CUDART_INF_F;
      mnew = fmaxf(mnew, s[u]);
    }
    // t0 < len, so mnew is finite here
    const float corr = ex2(m - mnew);
    l *= corr;
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] *= corr;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float p = ex2(s[u] - mnew);
      l += p;
      const __half2* vh = reinterpret_cast<const __half2*>(&kv[u][2]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 f = __half22float2(vh[i]);
        o[2 * i] = fmaf(p, f.x, o[2 * i]);
        o[2 * i + 1] = fmaf(p, f.y, o[2 * i + 1]);
      }
    }
    m = mnew;
  }

  if (a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  RowMerge<NG, RT> merge;
  merge.load(a, rows, bh, tr, lane);

  const int g0 = slot * NG;
  if (sub == 0) { sm_m[g0 + grp] = m; sm_l[g0 + grp] = l; }
#pragma unroll
  for (int i = 0; i < 16; i += 4)
    *reinterpret_cast<float4*>(&sm_o[g0 + grp][(i & 8) * 8 + sub * 8 + (i & 4)]) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
  if (NW == WPR) __syncthreads();
  else if (WPR == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(RT) : "memory");

  merge.finish(a, rows, bh, tr, lane, sm_m + g0, sm_l + g0, sm_o[g0]);
}

template <int MODE, int NW, int WPR, int U>
static int launch_rows(const BranchArgs& a, cudaStream_t st) {
  const unsigned grid = (unsigned)((a.rows + NW / WPR - 1) / (NW / WPR));
  const cudaError_t e = q40_launch_pdl(attn_branch_kernel<MODE, NW, WPR, U>, dim3(grid), dim3(NW * 32), 0, st, a);
  return e == cudaSuccess ? Q40_OK : (int)e;
}

// Warps per row and keys per 8-lane group by the number of rows; CTAs an SM at 128 registers a thread: two of eight warps with
// four keys, three with two keys, four of four warps with four keys, five with two.  A row's chain of iterations is its
// time while all rows are resident: eight warps while they are, then four; then what counts is that a row's start and
// merge occupy few warps: two, with two rows a CTA.  Microseconds, written warps / keys (2 / 4 has two rows a CTA):
//   paged, 512 keys: 256 rows 8 / 4 10.2, 8 / 2 13.3, 4 / 4 14.7; 256 keys: 512 rows
//     4 / 4 10.1, 4 / 2 12.3, 8 / 4 12.0; 608 rows 4 / 2 13.1, 4 / 4 14.9, 2 / 4 15.3; 1024 rows 2 / 4 17.0, 4 / 4 19.0; 3200 rows
//     2 / 4 50, 4 / 4 53.8; of up to 64: 768 rows 2 / 4 5.8, 4 / 4 6.5, 4 / 2 7.4.  Behind a prefix: 3200 rows of up to 64
//     2 / 4 23.2, 4 / 4 30.1, of up to 256 49.7 and 52.1
//   contiguous, 512 keys: 256 rows 8 / 4 12.6, 4 / 4 14.7; 416 rows 8 / 2 19.3, 4 / 4 19.9; 768 rows 4 / 4 35.9, 2 / 4 36.1; 3200 rows
//     of 256 4 / 4 63.1, 2 / 4 67.0; of 64: 64 rows 4 / 4 2.6, 8 / 4 3.1; 768 rows 2 / 4 5.1, 4 / 4 5.9
// (a.L is the length here.  Rows whose lengths are on the device are split by their number alone, see f16_form_of_rows)
template <int MODE>
static int launch_branch_mode(const BranchArgs& a, cudaStream_t st) {
  const int64_t rows = a.rows;
  if constexpr (MODE == 1 || MODE == 2) {
    if (rows <= 2 * 148) return launch_rows<MODE, 8, 8, 4>(a, st);
    if (rows > 5 * 148 || (rows > 4 * 148 && (a.L <= 128 || a.seq_lens))) return launch_rows<MODE, 4, 2, 4>(a, st);
    if (rows > 4 * 148) return launch_rows<MODE, 4, 4, 2>(a, st);
  } else {
    if (a.L > 128 && rows <= 2 * 148) return launch_rows<MODE, 8, 8, 4>(a, st);
    if (a.L > 128 && rows <= 3 * 148) return launch_rows<MODE, 8, 8, 2>(a, st);
    if (a.L <= 128 && rows > 4 * 148) return launch_rows<MODE, 4, 2, 4>(a, st);
  }
  return launch_rows<MODE, 4, 4, 4>(a, st);
}

static void fill_derived(BranchArgs& a, int B) {
  a.page_shift = -1;
  if (a.page_size > 0 && (a.page_size & (a.page_size - 1)) == 0)
    for (a.page_shift = 0; (1 << a.page_shift) < a.page_size;) ++a.page_shift;
  a.last_page = a.page_size > 0 && a.P > 0 ? (a.P - 1) / a.page_size : 0;
  a.rows = (int64_t)B * a.H;
}

int launch_branch(BranchArgs a, int mode, int B, int prompt, cudaStream_t st) {
  fill_derived(a, B);
  if (int rc; launch_branch_f16(a, mode, prompt, st, rc)) return rc;
  if (mode == 0) return launch_branch_mode<0>(a, st);
  if (mode == 1) return launch_branch_mode<1>(a, st);
  return launch_branch_mode<2>(a, st);
}

int launch_branch_q4(BranchRotArgs a, int B, cudaStream_t st) {
  fill_derived(a, B);
  return launch_branch_q4(a, a.cos_tbl != nullptr, st);
}

}  // namespace q40

static int check_common(int B, int H, int Hkv, int D) {
  if (D != q40::ATTN_D) return Q40_E_UNSUPPORTED;
  if (B < 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0) return Q40_E_SHAPE;
  if ((int64_t)B * H > 0x7fffffffLL) return Q40_E_SHAPE;
  return Q40_OK;
}

extern "C" int q40_attn_decode(const void* q, const void* k, const void* v, void* o, int B, int L, int H,
                               int Hkv, int D, void* stream) {
  if (!q || !o) return Q40_E_NULL;
  int rc = check_common(B, H, Hkv, D);
  if (rc) return rc;
  if (L < 0) return Q40_E_SHAPE;
  if (L > 0 && (!k || !v)) return Q40_E_NULL;
  if (B == 0) return Q40_OK;
  if (!q40_aligned(q, 16) || !q40_aligned(k, 16) || !q40_aligned(v, 16) || !q40_aligned(o, 2))
    return Q40_E_ALIGN;
  q40::BranchArgs a{};
  a.q = (const __half*)q; a.q_stride = (int64_t)H * D; a.k = (const __half*)k; a.v = (const __half*)v; a.o = (__half*)o;
  a.L = L; a.H = H; a.Hkv = Hkv; a.P = 0; a.page_size = 1;
  a.scale_log2 = q40::attn_scale_log2(D);
  return q40::launch_branch(a, 0, B, 0, (cudaStream_t)stream);
}

extern "C" int q40_attn_paged(const void* page_tbl, int idx_bytes, int64_t tbl_stride,
                              const int32_t* seq_lens, const void* q, const void* kpool, const void* vpool,
                              void* o, int P, int B, int Lmax, int H, int Hkv, int D, int page_size,
                              void* stream) {
  if (!q || !o) return Q40_E_NULL;
  int rc = check_common(B, H, Hkv, D);
  if (rc) return rc;
  if (Lmax < 0 || P < 0 || page_size <= 0) return Q40_E_SHAPE;
  if (idx_bytes != 2 && idx_bytes != 4) return Q40_E_UNSUPPORTED;
  if (Lmax > 0 && (!page_tbl || !kpool || !vpool || P == 0)) return Q40_E_NULL;
  if (tbl_stride < (Lmax + page_size - 1) / page_size) return Q40_E_SHAPE;
  if (B == 0) return Q40_OK;
  if (!q40_aligned(q, 16) || !q40_aligned(kpool, 16) || !q40_aligned(vpool, 16)) return Q40_E_ALIGN;
  q40::BranchArgs a{};
  a.q = (const __half*)q; a.q_stride = (int64_t)H * D; a.k = (const __half*)kpool; a.v = (const __half*)vpool; a.o = (__half*)o;
  a.tbl = page_tbl; a.tbl_stride = tbl_stride; a.seq_lens = seq_lens;
  a.L = Lmax; a.H = H; a.Hkv = Hkv; a.P = P; a.page_size = page_size;
  a.scale_log2 = q40::attn_scale_log2(D);
  return q40::launch_branch(a, idx_bytes == 2 ? 1 : 2, B, 0, (cudaStream_t)stream);
}
