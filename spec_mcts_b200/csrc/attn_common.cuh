// Declarations shared by the attention kernels.
#pragma once
#include <math_constants.h>

#include "q40_common.cuh"

namespace q40 {

constexpr int ATTN_D = 128;  // head dim of every supported model (CodeLlama 7B/70B)

inline float attn_scale_log2(int D) { return (1.0f / sqrtf((float)D)) * 1.4426950408889634f; }

// 2^x by the approximate instruction; results below 2^-126, which are nothing beside a row's largest weight, 1, become 0
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// acc + a.x b.x + a.y b.y: the products of fp16 values are exact, each sum rounds once
__device__ __forceinline__ float dot2(__half2 a, __half2 b, float acc) {
  asm("{\n\t.reg .b16 a0, a1, b0, b1;\n\tmov.b32 {a0, a1}, %1;\n\tmov.b32 {b0, b1}, %2;\n\t"
      "fma.rn.f32.f16 %0, a0, b0, %0;\n\tfma.rn.f32.f16 %0, a1, b1, %0;\n\t}" : "+f"(acc) : "r"(h2_as_u32(a)), "r"(h2_as_u32(b)));
  return acc;
}

struct BranchArgs {
  const __half* q;        // branch b, head h at q + b*q_stride + h*D
  int64_t q_stride;
  const __half* k;        // contiguous: [B,Hkv,L,D]; paged: pool [Hkv,P,D]
  const __half* v;
  __half* o;              // [B, H, D]
  const void* tbl;        // page table or nullptr
  int64_t tbl_stride;
  const int32_t* seq_lens;  // per-branch length or nullptr (= L)
  int L, H, Hkv, P, page_size;
  int page_shift, last_page;   // log2 of the page size or -1; id of the pool's last page (set by launch_branch)
  // optional partial results of a prefix pass over rows (b, h), log2 domain, un-normalised
  int64_t rows;           // B*H (set by launch_branch)
  const float* pm;        // [nsp][B*H]
  const float* pl;        // [nsp][B*H]
  const float* po;        // [nsp][B*H][128]
  int nsp;
  int beside_prefix;      // the prefix pass is the launch in front of this one: its results are waited for at the merge
  float scale_log2;       // 1/sqrt(D) * log2(e)
  // Q4_0 suffix cache: packed rows [B, max_t, Hkv, 64] + scales [B, max_t, Hkv, 2];
  // the branch's suffix length is pos[b] - prefix_len[0] (device values)
  const int8_t* kq;
  const __half* ksc;
  const int8_t* vq;
  const __half* vsc;
  const int32_t* pos;
  const int32_t* prefix_len;
  int max_t;
  // optional un-quantised K/V of the token being decoded, [B, Hkv*D] rows of stride cur_stride
  const __half* cur_k;
  const __half* cur_v;
  int64_t cur_stride;
};

// The Q4_0 cache; with tables ([n_pos, 64], 16-byte aligned) q and cur_k are from before their rotary embedding, which is done here, and
// the token's key and value are appended to the cache.  A struct of its own: a launch takes longer with more arguments, also where they are not
// used (a call of q40_attn_decode 3.33 us with 216 bytes, 3.68 with 240).
struct BranchRotArgs : BranchArgs {
  const __half* cos_tbl;
  const __half* sin_tbl;
  int n_pos;
};

// A weight p as two fp16: fp16(p) and what that leaves.  Weights come times 2^14, so that 22 bits are kept of all above 2^-28 of a row's
// largest, and 2^-39 of it of the others (root mean square errors against 64 bits are those of weights in fp32 to a thousandth: 2.07e-4 over 11
// sizes of paged and contiguous keys, which is the rounding of the result).  The first is never 0: an infinite value has to come out infinite, however small its weight
constexpr float WEIGHT_BITS = 14.f;
__device__ __forceinline__ uint32_t weight_parts(float p) {
  const __half h = __hmax_nan(__float2half_rn(p), __ushort_as_half(1));
  return h2_as_u32(__halves2half2(h, __float2half_rn(p - __half2float(h))));
}
// A row's sum from those over the two parts.  An infinite value is infinite in the first, and no number times a rest of 0
__device__ __forceinline__ float both_parts(float a, float b) { return fabsf(a) <= 3.402823466e38f ? a + b : a; }

// Slot of key t of branch b: in the pool (paged), or just t (contiguous).  `row` is the branch's first page id.  (With a division
// by the page size and 64-bit products per key, slots were a third of a paged row's instructions.)
template <int MODE>  // 0 contiguous, 1 paged with int16 ids, 2 paged with int32 ids
__device__ __forceinline__ int key_slot(const BranchArgs& a, const void* row, int t) {
  if (MODE == 0) return t;
  const int pg = a.page_shift >= 0 ? t >> a.page_shift : t / a.page_size, in = t - pg * a.page_size;
  const int id = MODE == 1 ? (int)(uint16_t) reinterpret_cast<const int16_t*>(row)[pg] : reinterpret_cast<const int32_t*>(row)[pg];
  // a bad page id must not turn into a wild read: clamp into the pool
  return min(min(max(id, 0), a.last_page) * a.page_size + in, a.P - 1);
}

// The end of a row (branch, head) of RT threads: its own keys' partial results, NG of them in shared memory, and those of a prefix pass
// become the output.  Thread tr owns output dims tr, tr + RT, ... (RT above the head's 128: the first four warps)
template <int NG, int RT>
struct RowMerge {
  static constexpr int DP = RT >= ATTN_D ? 1 : ATTN_D / RT, PB = 16 / DP;
  float pm_l, pl_l, po[PB][DP];
  // The prefix partials, once they are there and before the row's warps meet: lane sp holds the maximum and the sum of split sp
  // (further splits are read at the end), and the first splits' outputs are all requested together
  __device__ __forceinline__ void load(const BranchArgs& a, int64_t rows, int64_t bh, int tr, int lane) {
    pm_l = lane < a.nsp ? a.pm[(int64_t)lane * rows + bh] : -CUDART_INF_F;
    pl_l = lane < a.nsp ? a.pl[(int64_t)lane * rows + bh] : 0.f;
    if (a.nsp > 0) {
#pragma unroll
      for (int i = 0; i < PB; ++i)
#pragma unroll
        for (int j = 0; j < DP; ++j)
          po[i][j] = i < a.nsp && (RT <= ATTN_D || tr < ATTN_D) ? a.po[((int64_t)i * rows + bh) * ATTN_D + tr + j * RT] : 0.f;
    }
  }
  template <int STRIDE = ATTN_D>                // floats between the outputs of two
  __device__ __forceinline__ void finish(const BranchArgs& a, int64_t rows, int64_t bh, int tr, int lane, const float* sm_m, const float* sm_l,
                                         const float* sm_o) {
    if (RT > ATTN_D && tr >= ATTN_D) return;
    float M = -CUDART_INF_F;
#pragma unroll
    for (int g = 0; g < NG; ++g) M = fmaxf(M, sm_m[g]);
    M = fmaxf(M, warp_max(pm_l));
    for (int sp = 32; sp < a.nsp; ++sp) M = fmaxf(M, a.pm[(int64_t)sp * rows + bh]);
    float Lsum = 0.f, acc[DP];
#pragma unroll
    for (int j = 0; j < DP; ++j) acc[j] = 0.f;
    if (M > -CUDART_INF_F) {
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const float w = ex2(sm_m[g] - M);         // exp2(-inf) = 0 for empty groups
        Lsum = fmaf(sm_l[g], w, Lsum);
#pragma unroll
        for (int j = 0; j < DP; ++j) acc[j] = fmaf(sm_o[g * STRIDE + tr + j * RT], w, acc[j]);
      }
      if (a.nsp > 0) {
        const float pw_l = ex2(pm_l - M);
#pragma unroll
        for (int i = 0; i < PB; ++i) {            // splits from nsp on: weight and sum are 0
          const float w = __shfl_sync(0xffffffffu, pw_l, i);
          Lsum = fmaf(__shfl_sync(0xffffffffu, pl_l, i), w, Lsum);
#pragma unroll
          for (int j = 0; j < DP; ++j) acc[j] = fmaf(po[i][j], w, acc[j]);
        }
        for (int sp = PB; sp < min(a.nsp, 32); ++sp) {
          const float w = __shfl_sync(0xffffffffu, pw_l, sp);
          Lsum = fmaf(__shfl_sync(0xffffffffu, pl_l, sp), w, Lsum);
#pragma unroll
          for (int j = 0; j < DP; ++j) acc[j] = fmaf(a.po[((int64_t)sp * rows + bh) * ATTN_D + tr + j * RT], w, acc[j]);
        }
      }
      for (int sp = 32; sp < a.nsp; ++sp) {
        const int64_t r = (int64_t)sp * rows + bh;
        const float w = ex2(a.pm[r] - M);
        Lsum = fmaf(a.pl[r], w, Lsum);
#pragma unroll
        for (int j = 0; j < DP; ++j) acc[j] = fmaf(a.po[r * ATTN_D + tr + j * RT], w, acc[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < DP; ++j) a.o[bh * ATTN_D + tr + j * RT] = __float2half_rn((Lsum > 0.f) ? acc[j] / Lsum : 0.f);
  }
};

// defined in attn_branch_q4.cu; `rotate`: see BranchRotArgs
int launch_branch_q4(const BranchRotArgs& a, bool rotate, cudaStream_t st);
// defined in attn_branch.cu; mode 0 contiguous, 1 paged/int16 ids, 2 paged/int32 ids; `prompt`: keys of the prefix pass, 0: none
int launch_branch(BranchArgs a, int mode, int B, int prompt, cudaStream_t st);
// defined in attn_branch_f16.cu; false, and nothing launched, where attn_branch_kernel is faster
bool launch_branch_f16(const BranchArgs& a, int mode, int prompt, cudaStream_t st, int& rc);
int launch_branch_q4(BranchRotArgs a, int B, cudaStream_t st);         // the Q4_0 cache, with rotation where there are tables

}  // namespace q40
