// Declarations shared by the attention kernels.
#pragma once
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
  // Q4_0 suffix cache (mode 3): packed rows [B, max_t, Hkv, 64] + scales [B, max_t, Hkv, 2];
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

// mode 4: mode 3 with q and cur_k from before their rotary embedding (tables [n_pos, 64], 16-byte aligned), which is done here, and the
// token's key and value appended to the cache.  A struct of its own: a launch takes longer with more arguments, also where they are not
// used (a call of q40_attn_decode 3.33 us with 216 bytes, 3.68 with 240).
struct BranchRotArgs : BranchArgs {
  const __half* cos_tbl;
  const __half* sin_tbl;
  int n_pos;
};

// defined in attn_branch.cu; mode 0 contiguous, 1 paged/int16 ids, 2 paged/int32 ids, 3 Q4_0 cache
int launch_branch(BranchArgs a, int mode, int B, cudaStream_t st);
int launch_branch(BranchRotArgs a, int B, cudaStream_t st);   // mode 4

}  // namespace q40
