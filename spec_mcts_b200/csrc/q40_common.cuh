// Shared helpers for the q40b200 kernels (sm_100a only).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/q40b200.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "q40b200 kernels are written for sm_100a only"
#endif

#define Q40_LAUNCH_CHECK()                          \
  do {                                              \
    cudaError_t e__ = cudaGetLastError();           \
    if (e__ != cudaSuccess) return (int)e__;        \
  } while (0)

// A bounded wait has run out: the caller's error word, which may be mapped host memory (all writers store the same)
__device__ __forceinline__ void q40_set_error(int* err) { *reinterpret_cast<volatile int*>(err) = 1; }

static inline bool q40_aligned(const void* p, size_t a) { return ((uintptr_t)p % a) == 0; }

// Allow `kern` that much dynamic shared memory, once per device (`ready`: one bit each).  The limit is a property of the
// kernel, not of a launch: set to the most any call needs, threads that meet here do not lower each other's.
static inline cudaError_t q40_allow_smem(std::atomic<uint64_t>& ready, const void* kern, int bytes) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (ready.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) ready.fetch_or(bit, std::memory_order_release);
  return e;
}

// Launch with programmatic stream serialization.  Kernels launched this way execute griddepcontrol.wait
// before their first access to global memory (the branch attention behind a prefix pass: before the first to what that
// pass writes, see attn_branch_kernel), so for the caller the launch orders exactly like a plain
// one; what changes is that the CTAs may become resident while the previous launch on the stream drains
// (and, where that launch triggered early, while it runs), which takes the launch latency off the
// critical path of a chain of small dependent launches.
template <typename... KArgs, typename... Args>
static inline cudaError_t q40_launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                         cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Optional stage timestamps (builds with -DQ40_TRACE only; compiled out otherwise): thread 0 of a CTA
// reads the global nanosecond timer at up to 8 points and appends one record of 10 words
// {kind, linear CTA id, t0..t7} to the buffer given to q40_debug_trace (word 0 = record counter,
// word 1 = capacity in records, records from word 16).
#ifdef Q40_TRACE
extern void* q40_trace_ptr;
#define Q40_TRACE_DECL unsigned long long q40_ts_[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#define Q40_STAMP(i) \
  do { if (threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(q40_ts_[i])::"memory"); } while (0)
#define Q40_STAMP_DEP(i, v) /* not before the float v is available */ \
  do { if (threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(q40_ts_[i]) : "f"(v) : "memory"); } while (0)
#define Q40_TRACE_FLUSH(buf, kind)                                                                   \
  do {                                                                                               \
    unsigned long long* tb_ = (unsigned long long*)(buf);                                            \
    if (threadIdx.x == 0 && tb_) {                                                                   \
      const unsigned long long slot_ = atomicAdd(tb_, 1ull);                                         \
      if (slot_ < tb_[1]) {                                                                          \
        unsigned long long* r_ = tb_ + 16 + slot_ * 10;                                              \
        r_[0] = (kind);                                                                              \
        r_[1] = (unsigned long long)blockIdx.x + (unsigned long long)gridDim.x * blockIdx.y;         \
        for (int i_ = 0; i_ < 8; ++i_) r_[2 + i_] = q40_ts_[i_];                                     \
      }                                                                                              \
    }                                                                                                \
  } while (0)
#else
#define Q40_TRACE_DECL
#define Q40_STAMP(i) do { } while (0)
#define Q40_STAMP_DEP(i, v) do { } while (0)
#define Q40_TRACE_FLUSH(buf, kind) do { } while (0)
#endif

namespace q40 {

__device__ __forceinline__ uint32_t lop3_and_xor(uint32_t a, uint32_t mask, uint32_t x) {
  uint32_t r;
  // (a & mask) ^ x : immLut = (0xF0 & 0xCC) ^ 0xAA
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(mask), "r"(x));
  return r;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

__device__ __forceinline__ __half2 u32_as_h2(uint32_t v) {
  return *reinterpret_cast<__half2*>(&v);
}
__device__ __forceinline__ uint32_t h2_as_u32(__half2 v) {
  return *reinterpret_cast<uint32_t*>(&v);
}

// Two signed 4-bit codes sitting in the LOW nibbles of bytes 0 and 2 of `p` -> exact half2.
// (nib ^ 8) | 0x6400 is the half 1024 + (code + 8); subtracting 1032 is exact.
__device__ __forceinline__ __half2 codes_lo_to_h2(uint32_t p) {
  uint32_t v = lop3_and_xor(p, 0x000F000Fu, 0x64086408u);
  return __hsub2(u32_as_h2(v), u32_as_h2(0x64086408u));
}
// Same for the HIGH nibbles of bytes 0 and 2: the half is 1024 + 16*(code + 8);
// fma(v, 1/16, -72) is exact.
__device__ __forceinline__ __half2 codes_hi_to_h2(uint32_t p) {
  uint32_t v = lop3_and_xor(p, 0x00F000F0u, 0x64806480u);
  return __hfma2(u32_as_h2(v), u32_as_h2(0x2C002C00u) /* 1/16 */, u32_as_h2(0xD480D480u) /* -72 */);
}

// The format's fp16(w / scale) without a division per element.  w and s are fp16: write w = A 2^i, s = S 2^j with
// integers A, S < 2^11.  An fp16 rounding boundary of the quotient is M 2^g with an odd 12-bit M, and
// A/S = M 2^h has no solution (S M has more significant bits than A), so |A 2^h' - S M| >= 1 and the quotient stays
// at least 1 / (2047 * 4095) = 2^-23 * 1.0007 away from every boundary, relatively.  fl(w * fl(1/s)) in fp32 is at
// most 2^-23 + 2^-48 off.  So it lies on the quotient's side of the boundary and rounds to the same fp16 value.
// (Quotients below the normal fp16 range round to a code of 0 either way.)
// x + 1536 in fp16 then rounds to the nearest integer, ties to even, and leaves the two's complement code in the low
// bits; the clamp makes NaN and infinite quotients (NaN loses against a number in min/max) leave 0 there, which
// is what the x86 float->int conversion of the reference makes of them.
__device__ __forceinline__ uint32_t quant_pair(uint32_t w2, float inv) {
  const float2 f = __half22float2(u32_as_h2(w2));
  __half2 h = __floats2half2_rn(f.x * inv, f.y * inv);
  h = __hmin2(__hmax2(h, u32_as_h2(0xE000E000u)), u32_as_h2(0x60006000u));   // [-512, 512]
  return h2_as_u32(__hadd2(h, u32_as_h2(0x66006600u)));                      // 1536 + code
}

// Eight values of a pair's even group and the same of its odd group: their (even, odd) maxima.  max drops NaN like
// torch.max would not, but NaN inputs are outside the format.
__device__ __forceinline__ __half2 quant_max(const uint32_t (&ew)[4], const uint32_t (&ow)[4]) {
  __half2 ae = __habs2(u32_as_h2(ew[0])), ao = __habs2(u32_as_h2(ow[0]));
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    ae = __hmax2(ae, __habs2(u32_as_h2(ew[i])));
    ao = __hmax2(ao, __habs2(u32_as_h2(ow[i])));
  }
  return __hmax2(__lows2half2(ae, ao), __highs2half2(ae, ao));
}

// ... and, with the maxima m over the whole groups, their 8 finished bytes and the two scales
__device__ __forceinline__ uint2 quant_codes(const uint32_t (&ew)[4], const uint32_t (&ow)[4], __half2 m, __half2& sc) {
  const float me = fmaxf(0.f, __low2float(m)), mo = fmaxf(0.f, __high2float(m));    // all-NaN group: 0
  // scale = fp16(absmax / 7): fp32 division, one rounding to fp16
  const __half se = __float2half_rn(__fdiv_rn(me, 7.0f)), so = __float2half_rn(__fdiv_rn(mo, 7.0f));
  // a scale of zero makes every code 0 (x/0 and 0/0 both do)
  const float fe = __half2float(se), fo = __half2float(so);
  const float ie = fe > 0.f ? __frcp_rn(fe) : 0.f, io = fo > 0.f ? __frcp_rn(fo) : 0.f;
  uint32_t out[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t ce = quant_pair(ew[2 * k + i], ie), co = quant_pair(ow[2 * k + i], io);
      b[i] = ((ce << 4) & 0x00F000F0u) | (co & 0x000F000Fu);      // bytes 0 and 2 of the word
    }
    out[k] = prmt(b[0], b[1], 0x6420);
  }
  sc = __halves2half2(se, so);
  return make_uint2(out[0], out[1]);
}

// Rotary embedding of eight dims (lo) and the eight 64 further (hi), with their cosines and sines, in fp16: the reference's roundings
__device__ __forceinline__ void rotate_dims(uint4& lo, uint4& hi, const uint4& c, const uint4& s) {
  const __half2 *ch = reinterpret_cast<const __half2*>(&c), *sh = reinterpret_cast<const __half2*>(&s);
  __half2 *l2 = reinterpret_cast<__half2*>(&lo), *h2 = reinterpret_cast<__half2*>(&hi);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2 x1 = l2[j], x2 = h2[j];
    l2[j] = __hadd2_rn(__hmul2_rn(x1, ch[j]), __hmul2_rn(__hneg2(x2), sh[j]));
    h2[j] = __hadd2_rn(__hmul2_rn(x2, ch[j]), __hmul2_rn(x1, sh[j]));
  }
}

// dims 8i.. (high nibbles) and 64 + 8i.. (low nibbles) of a head -> 8 packed bytes per lane and the row's two scales.  The eight lanes of a
// head are STRIDE apart; of others that hold the same, `writes` is false
template <int STRIDE = 1>
__device__ __forceinline__ void append_row(const uint4& lo, const uint4& hi, int8_t* codes, __half* scales, int i,
                                           unsigned gmask, bool writes = true) {
  const uint32_t ew[4] = {lo.x, lo.y, lo.z, lo.w}, ow[4] = {hi.x, hi.y, hi.z, hi.w};
  __half2 m = quant_max(ew, ow);
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) m = __hmax2(m, u32_as_h2(__shfl_xor_sync(gmask, h2_as_u32(m), off * STRIDE)));
  __half2 sc;
  const uint2 out = quant_codes(ew, ow, m, sc);
  if (writes) {
    *reinterpret_cast<uint2*>(codes + 8 * i) = out;
    if (i == 0) *reinterpret_cast<__half2*>(scales) = sc;
  }
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace q40
