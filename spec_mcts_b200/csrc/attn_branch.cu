// Decode attention for one query token per branch over that branch's own keys: a
// contiguous [B,Hkv,L,D] cache, a paged pool or the packed Q4_0 cache.  Two, four or eight warps per row
// (branch, query head), one or two rows per CTA: see launch_branch_mode.
//
// Eight lanes share a key: lane i owns dims 8i..8i+7 and 64+8i..64+8i+7 of the head (two 16-byte loads of K, two of
// V, each of which covers 128 contiguous bytes over the lanes; in the Q4_0 cache the same dims are the two
// nibbles of 8 bytes), the partial dot products are summed with three shuffles, and every group of
// eight lanes keeps its own online-softmax state (running max, sum, 16 output dims) in
// fp32.  A row's groups (four per warp) are merged through shared memory at the end; the same
// merge can fold in partial results of a shared-prefix pass (see attn_prefix.cu), which is
// how the shared-prefix entry point finishes.
//
// Stands in for flash_attn_kernel2 / page_flash_attn_kernel2 of the reference
// (triton_kernels.py:559-647, 700-789), with fp32 softmax state and exact masking of the
// tail instead of the reference's fp16 state and multiple-of-32 length requirement.
#include <math_constants.h>

#include <type_traits>

#include "attn_common.cuh"

namespace q40 {

// Page ids are looked up one iteration ahead of the keys they lead to, so that an iteration waits for one memory latency
// and not for two.
//
// A CTA has NW warps; WPR of them share a row (branch, head).  What bounds a row is latency (ids -> keys -> sums
// -> merge), so the split is the one that keeps the warps of all rows resident at once: see launch_branch_mode.

// Slot of key t of branch b: in the pool (paged), or just t (contiguous).  `row` is the branch's first page id.  (With a division
// by the page size and 64-bit products per key, slots were a third of a paged row's instructions.)
template <int MODE>  // 0 contiguous, 1 paged with int16 ids, 2 paged with int32 ids, 3 Q4_0 cache, 4 the same with rotation and append (see BranchRotArgs)
__device__ __forceinline__ int key_slot(const BranchArgs& a, const void* row, int t) {
  if (MODE == 0 || MODE >= 3) return t;
  const int pg = a.page_shift >= 0 ? t >> a.page_shift : t / a.page_size, in = t - pg * a.page_size;
  const int id = MODE == 1 ? (int)(uint16_t) reinterpret_cast<const int16_t*>(row)[pg] : reinterpret_cast<const int32_t*>(row)[pg];
  // a bad page id must not turn into a wild read: clamp into the pool
  return min(min(max(id, 0), a.last_page) * a.page_size + in, a.P - 1);
}

// acc + a.x b.x + a.y b.y: the products of fp16 values are exact, each sum rounds once
__device__ __forceinline__ float dot2(__half2 a, __half2 b, float acc) {
  asm("{\n\t.reg .b16 a0, a1, b0, b1;\n\tmov.b32 {a0, a1}, %1;\n\tmov.b32 {b0, b1}, %2;\n\t"
      "fma.rn.f32.f16 %0, a0, b0, %0;\n\tfma.rn.f32.f16 %0, a1, b1, %0;\n\t}" : "+f"(acc) : "r"(h2_as_u32(a)), "r"(h2_as_u32(b)));
  return acc;
}

// a row's two scales in one word
__device__ __forceinline__ uint32_t load_scales(const __half* p, bool aligned4) {
  if (aligned4) return __ldg(reinterpret_cast<const uint32_t*>(p));
  return h2_as_u32(__halves2half2(__ldg(p), __ldg(p + 1)));
}

// Rotary embedding of a lane's 16 dims at branch b's position
__device__ __forceinline__ void rotate_at(const BranchRotArgs& a, int b, int sub, uint4& lo, uint4& hi) {
  const int64_t at = (int64_t)min(max(a.pos[b], 0), a.n_pos - 1) * 64 + 8 * sub;
  rotate_dims(lo, hi, __ldg(reinterpret_cast<const uint4*>(a.cos_tbl + at)), __ldg(reinterpret_cast<const uint4*>(a.sin_tbl + at)));
}

template <int MODE>
using ModeArgs = std::conditional_t<MODE == 4, BranchRotArgs, BranchArgs>;

template <int MODE, int NW, int WPR, int U>    // U: keys per 8-lane group in flight
__global__ void __launch_bounds__(NW * 32, U > 2 ? 16 / NW : NW == 8 ? 3 : 5)
attn_branch_kernel(const ModeArgs<MODE> a) {
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

  int len;
  // mode 4 appends at the position that the tables allow, so that is the length too: the row that is written is never one that is read
  if constexpr (MODE == 4) len = min(max(min(max(a.pos[b], 0), a.n_pos - 1) - a.prefix_len[0], 0), a.max_t);
  else if (MODE == 3) len = min(max(a.pos[b] - a.prefix_len[0], 0), a.max_t);
  else len = a.seq_lens ? min(max(a.seq_lens[b], 0), a.L) : a.L;
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
  if constexpr (MODE == 4) rotate_at(a, b, sub, *reinterpret_cast<uint4*>(qh), *reinterpret_cast<uint4*>(qh + 4));
  float m = -CUDART_INF_F, l = 0.f, o[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i] = 0.f;

  // first key of this head and branch, at this lane's dims
  const int64_t kv0 = (MODE == 0 ? (int64_t)(b * a.Hkv + hk) * a.L : (int64_t)hk * a.P) * D + sub * 8;
  if (MODE < 3)
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

  if (MODE >= 3) {
    // Q4_0 cache: lane `sub` owns bytes 8*sub..8*sub+7 of a row, both nibbles; a word's bytes come out as (0, 2) and (1, 3)
    __half2 q4[8];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      q4[i] = __lows2half2(qh[i], qh[i + 1]);
      q4[i + 1] = __highs2half2(qh[i], qh[i + 1]);
    }
    const bool sc4 = (((uintptr_t)a.ksc | (uintptr_t)a.vsc) & 3) == 0;
    for (int t0 = grp; t0 < len; t0 += NG * U) {
      uint2 kb[U], vb[U];
      uint32_t ksv[U], vsv[U];
      float s[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * NG;
        if (t < len) {
          const int64_t row = ((int64_t)b * a.max_t + t) * a.Hkv + hk;
          kb[u] = __ldg(reinterpret_cast<const uint2*>(a.kq + row * 64 + 8 * sub));
          vb[u] = __ldg(reinterpret_cast<const uint2*>(a.vq + row * 64 + 8 * sub));
          ksv[u] = load_scales(a.ksc + row * 2, sc4);
          vsv[u] = load_scales(a.vsc + row * 2, sc4);
        } else {
          kb[u] = vb[u] = make_uint2(0, 0);
          ksv[u] = vsv[u] = 0u;
        }
      }
      float mnew = m;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const __half2 sh = __low2half2(u32_as_h2(ksv[u])), sl = __high2half2(u32_as_h2(ksv[u]));
        float acc = 0.f;
#pragma unroll
        for (int wi = 0; wi < 2; ++wi) {
          const uint32_t w = wi ? kb[u].y : kb[u].x;
          acc = dot2(q4[2 * wi], __hmul2(codes_hi_to_h2(w), sh), acc);                // bytes 0, 2
          acc = dot2(q4[2 * wi + 1], __hmul2(codes_hi_to_h2(w >> 8), sh), acc);       // bytes 1, 3
          acc = dot2(q4[4 + 2 * wi], __hmul2(codes_lo_to_h2(w), sl), acc);
          acc = dot2(q4[4 + 2 * wi + 1], __hmul2(codes_lo_to_h2(w >> 8), sl), acc);
        }
        acc += __shfl_xor_sync(gmask, acc, 1);
        acc += __shfl_xor_sync(gmask, acc, 2);
        acc += __shfl_xor_sync(gmask, acc, 4);
        s[u] = (t0 + u * NG < len) ? acc * a.scale_log2 : -CUDART_INF_F;
        mnew = fmaxf(mnew, s[u]);
      }
      const float corr = ex2(m - mnew);
      l *= corr;
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i] *= corr;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float p = ex2(s[u] - mnew);
        l += p;
        const __half2 sh = __low2half2(u32_as_h2(vsv[u])), sl = __high2half2(u32_as_h2(vsv[u]));
#pragma unroll
        for (int wi = 0; wi < 2; ++wi) {
          const uint32_t w = wi ? vb[u].y : vb[u].x;
          const float2 h02 = __half22float2(__hmul2(codes_hi_to_h2(w), sh));
          const float2 h13 = __half22float2(__hmul2(codes_hi_to_h2(w >> 8), sh));
          const float2 l02 = __half22float2(__hmul2(codes_lo_to_h2(w), sl));
          const float2 l13 = __half22float2(__hmul2(codes_lo_to_h2(w >> 8), sl));
          o[4 * wi + 0] = fmaf(p, h02.x, o[4 * wi + 0]);
          o[4 * wi + 2] = fmaf(p, h02.y, o[4 * wi + 2]);
          o[4 * wi + 1] = fmaf(p, h13.x, o[4 * wi + 1]);
          o[4 * wi + 3] = fmaf(p, h13.y, o[4 * wi + 3]);
          o[8 + 4 * wi + 0] = fmaf(p, l02.x, o[8 + 4 * wi + 0]);
          o[8 + 4 * wi + 2] = fmaf(p, l02.y, o[8 + 4 * wi + 2]);
          o[8 + 4 * wi + 1] = fmaf(p, l13.x, o[8 + 4 * wi + 1]);
          o[8 + 4 * wi + 3] = fmaf(p, l13.y, o[8 + 4 * wi + 3]);
        }
      }
      m = mnew;
    }
  }
  // the token being decoded attends to its own, un-quantised K/V: one extra key for group 0
  if (a.cur_k != nullptr && grp == 0) {
    const __half* kp = a.cur_k + (int64_t)b * a.cur_stride + hk * D + sub * 8;
    const __half* vp = a.cur_v + (int64_t)b * a.cur_stride + hk * D + sub * 8;
    uint4 k0 = *reinterpret_cast<const uint4*>(kp), k1 = *reinterpret_cast<const uint4*>(kp + 64);
    const uint4 v0 = *reinterpret_cast<const uint4*>(vp), v1 = *reinterpret_cast<const uint4*>(vp + 64);
    if constexpr (MODE == 4) {
      rotate_at(a, b, sub, k0, k1);
      const int t = min(max(a.pos[b], 0), a.n_pos - 1) - a.prefix_len[0];
      if (h % (a.H / a.Hkv) == 0 && t >= 0 && t < a.max_t) {             // the first query head of a kv head
        const int64_t row = ((int64_t)b * a.max_t + t) * a.Hkv + hk;
        append_row(k0, k1, const_cast<int8_t*>(a.kq) + row * 64, const_cast<__half*>(a.ksc) + row * 2, sub, 0xffu);
        append_row(v0, v1, const_cast<int8_t*>(a.vq) + row * 64, const_cast<__half*>(a.vsc) + row * 2, sub, 0xffu);
      }
    }
    const __half2* kh0 = reinterpret_cast<const __half2*>(&k0);
    const __half2* kh1 = reinterpret_cast<const __half2*>(&k1);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc = dot2(qh[4 + i], kh1[i], dot2(qh[i], kh0[i], acc));
    acc += __shfl_xor_sync(0x000000ffu, acc, 1);
    acc += __shfl_xor_sync(0x000000ffu, acc, 2);
    acc += __shfl_xor_sync(0x000000ffu, acc, 4);
    acc *= a.scale_log2;
    const float mnew = fmaxf(m, acc);
    const float corr = ex2(m - mnew), p = ex2(acc - mnew);
    l = l * corr + p;
    const __half2* vh0 = reinterpret_cast<const __half2*>(&v0);
    const __half2* vh1 = reinterpret_cast<const __half2*>(&v1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f0 = __half22float2(vh0[i]), f1 = __half22float2(vh1[i]);
      o[2 * i] = fmaf(p, f0.x, o[2 * i] * corr);
      o[2 * i + 1] = fmaf(p, f0.y, o[2 * i + 1] * corr);
      o[8 + 2 * i] = fmaf(p, f1.x, o[8 + 2 * i] * corr);
      o[8 + 2 * i + 1] = fmaf(p, f1.y, o[8 + 2 * i + 1] * corr);
    }
    m = mnew;
  }

  if (a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  // prefix partials: lane sp holds the maximum and the sum of split sp (further splits are read at the merge)
  const float pm_l = lane < a.nsp ? a.pm[(int64_t)lane * rows + bh] : -CUDART_INF_F;
  const float pl_l = lane < a.nsp ? a.pl[(int64_t)lane * rows + bh] : 0.f;
  // ... and the first splits' outputs at this thread's dims, all requested together and before the groups meet
  constexpr int DP = RT >= D ? 1 : D / RT, PB = 16 / DP;
  float po[PB][DP];
  if (a.nsp > 0) {
#pragma unroll
    for (int i = 0; i < PB; ++i)
#pragma unroll
      for (int j = 0; j < DP; ++j)
        po[i][j] = i < a.nsp && (RT <= D || tr < D) ? a.po[((int64_t)i * rows + bh) * D + tr + j * RT] : 0.f;
  }

  const int g0 = slot * NG;
  if (sub == 0) { sm_m[g0 + grp] = m; sm_l[g0 + grp] = l; }
#pragma unroll
  for (int i = 0; i < 16; i += 4)
    *reinterpret_cast<float4*>(&sm_o[g0 + grp][(i & 8) * 8 + sub * 8 + (i & 4)]) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
  if (NW == WPR) __syncthreads();
  else if (WPR == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(RT) : "memory");

  // merge: thread tr owns output dims tr, tr + RT, ... (WPR = 8: the first four warps)
  if (RT > D && tr >= D) return;
  float M = -CUDART_INF_F;
#pragma unroll
  for (int gI = 0; gI < NG; ++gI) M = fmaxf(M, sm_m[g0 + gI]);
  M = fmaxf(M, warp_max(pm_l));
  for (int sp = 32; sp < a.nsp; ++sp) M = fmaxf(M, a.pm[(int64_t)sp * rows + bh]);
  float Lsum = 0.f, acc[DP];
#pragma unroll
  for (int j = 0; j < DP; ++j) acc[j] = 0.f;
  if (M > -CUDART_INF_F) {
#pragma unroll
    for (int gI = 0; gI < NG; ++gI) {
      const float w = ex2(sm_m[g0 + gI] - M);   // exp2(-inf) = 0 for empty groups
      Lsum = fmaf(sm_l[g0 + gI], w, Lsum);
#pragma unroll
      for (int j = 0; j < DP; ++j) acc[j] = fmaf(sm_o[g0 + gI][tr + j * RT], w, acc[j]);
    }
    if (a.nsp > 0) {
      const float pw_l = ex2(pm_l - M);
#pragma unroll
      for (int i = 0; i < PB; ++i) {                // splits from nsp on: weight and sum are 0
        const float w = __shfl_sync(0xffffffffu, pw_l, i);
        Lsum = fmaf(__shfl_sync(0xffffffffu, pl_l, i), w, Lsum);
#pragma unroll
        for (int j = 0; j < DP; ++j) acc[j] = fmaf(po[i][j], w, acc[j]);
      }
      for (int sp = PB; sp < min(a.nsp, 32); ++sp) {
        const float w = __shfl_sync(0xffffffffu, pw_l, sp);
        Lsum = fmaf(__shfl_sync(0xffffffffu, pl_l, sp), w, Lsum);
#pragma unroll
        for (int j = 0; j < DP; ++j) acc[j] = fmaf(a.po[((int64_t)sp * rows + bh) * D + tr + j * RT], w, acc[j]);
      }
    }
    for (int sp = 32; sp < a.nsp; ++sp) {
      const int64_t r = (int64_t)sp * rows + bh;
      const float w = ex2(a.pm[r] - M);
      Lsum = fmaf(a.pl[r], w, Lsum);
#pragma unroll
      for (int j = 0; j < DP; ++j) acc[j] = fmaf(a.po[r * D + tr + j * RT], w, acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < DP; ++j)
    a.o[bh * D + tr + j * RT] = __float2half_rn((Lsum > 0.f) ? acc[j] / Lsum : 0.f);
}

template <int MODE, int NW, int WPR, int U>
static int launch_rows(const ModeArgs<MODE>& a, cudaStream_t st) {
  const unsigned grid = (unsigned)((a.rows + NW / WPR - 1) / (NW / WPR));
  const cudaError_t e = q40_launch_pdl(attn_branch_kernel<MODE, NW, WPR, U>, dim3(grid), dim3(NW * 32), 0, st, a);
  return e == cudaSuccess ? Q40_OK : (int)e;
}

// Warps per row and keys per 8-lane group by the number of rows; CTAs an SM at 128 registers a thread: two of eight warps with
// four keys, three with two keys, four of four warps with four keys, five with two.  A row's chain of iterations is its
// time while all rows are resident: eight warps while they are, then four; then what counts is that a row's start and
// merge occupy few warps: two, with two rows a CTA.  Microseconds, written warps / keys (2 / 4 has two rows a CTA):
//   paged, 512 keys: 256 rows 8 / 4 10.2, 8 / 2 13.3, 4 / 4 14.7; 416 rows 8 / 2 15.2, 4 / 4 16.7, 8 / 4 18.2; 256 keys: 512 rows
//     4 / 4 10.1, 4 / 2 12.3, 8 / 4 12.0; 608 rows 4 / 2 13.1, 4 / 4 14.9, 2 / 4 15.3; 1024 rows 2 / 4 17.0, 4 / 4 19.0; 3200 rows
//     2 / 4 50, 4 / 4 53.8; of up to 64: 768 rows 2 / 4 5.8, 4 / 4 6.5, 4 / 2 7.4.  Behind a prefix: 3200 rows of up to 64
//     2 / 4 23.2, 4 / 4 30.1, of up to 256 49.7 and 52.1
//   contiguous, 512 keys: 256 rows 8 / 4 12.6, 4 / 4 14.7; 416 rows 8 / 2 19.3, 4 / 4 19.9; 768 rows 4 / 4 35.9, 2 / 4 36.1; 3200 rows
//     of 256 4 / 4 63.1, 2 / 4 67.0; of 64: 64 rows 4 / 4 2.6, 8 / 4 3.1; 768 rows 2 / 4 5.1, 4 / 4 5.9
//   Q4_0 cache, whose length the host does not know, 20 / 64 / 200 keys, with the prefix pass: 64 rows 4 / 4 6.2 / 6.3 / 8.8, 8 / 2
//     6.5 / 6.8 / 8.7; 320 rows 8 / 2 8.5 / 9.1 / 12.7, 4 / 4 8.8 / 9.0 / 13.5, 2 / 4 8.1 / 10.2 / 18.6; 640 rows 2 / 4 8.2 / 9.9 /
//     18.4, 4 / 4 10.5 / 10.9 / 16.6; 960 rows 9.3 / 11.4 / 20.2 and 12.7 / 13.1 / 20.7; 3200 rows 19.3 / 23.8 / 46.8 and 29.5 / 30.4 / 53.5
//     (a whole step of 320 rows with 64 keys: 8 / 2 2280, 4 / 4 2251)
template <int MODE>
static int launch_branch_mode(const ModeArgs<MODE>& a, cudaStream_t st) {
  const int64_t rows = a.rows;
  if constexpr (MODE == 1 || MODE == 2) {
    if (rows <= 2 * 148) return launch_rows<MODE, 8, 8, 4>(a, st);
    if (rows <= 3 * 148) return launch_rows<MODE, 8, 8, 2>(a, st);
    if (rows > 5 * 148 || (rows > 4 * 148 && a.L <= 128)) return launch_rows<MODE, 4, 2, 4>(a, st);
    if (rows > 4 * 148) return launch_rows<MODE, 4, 4, 2>(a, st);
  } else if constexpr (MODE == 0) {
    if (a.L > 128 && rows <= 2 * 148) return launch_rows<MODE, 8, 8, 4>(a, st);
    if (a.L > 128 && rows <= 3 * 148) return launch_rows<MODE, 8, 8, 2>(a, st);
    if (a.L <= 128 && rows > 4 * 148) return launch_rows<MODE, 4, 2, 4>(a, st);
  } else {
    if (rows > 4 * 148) return launch_rows<MODE, 4, 2, 4>(a, st);
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

int launch_branch(BranchArgs a, int mode, int B, cudaStream_t st) {
  fill_derived(a, B);
  if (mode == 0) return launch_branch_mode<0>(a, st);
  if (mode == 1) return launch_branch_mode<1>(a, st);
  if (mode == 2) return launch_branch_mode<2>(a, st);
  return launch_branch_mode<3>(a, st);
}

int launch_branch(BranchRotArgs a, int B, cudaStream_t st) {
  fill_derived(a, B);
  return launch_branch_mode<4>(a, st);
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
  return q40::launch_branch(a, 0, B, (cudaStream_t)stream);
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
  return q40::launch_branch(a, idx_bytes == 2 ? 1 : 2, B, (cudaStream_t)stream);
}
