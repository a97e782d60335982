// What the tensor-core matmuls on the tiled weight copies share: mbarriers, bulk and tensor copies, tcgen05
// instructions, and the step from a tile word to the A operand.
#pragma once
#include <cuda.h>

#include <atomic>

#include "q40_common.cuh"

namespace q40 {
namespace ttc {

constexpr int BK = 64;                          // k rows per pipeline stage
constexpr int SPAN = 256;                       // features of a span of the tiled stream
constexpr int STEP_BYTES = 2048 + 128;
constexpr int SMEM_MAX = 227 * 1024;            // of a CTA
constexpr unsigned SPIN_LIMIT = 1u << 17;       // polls before giving up
constexpr unsigned POLL_NS = 20000;             // ... each of which suspends the thread until the barrier's phase ends or this time is
                                                // over: warps that wait otherwise take a third of the issue slots

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// One lane of a converged warp, chosen so that the compiler knows the branch to be taken by a single thread: operands
// of copies and MMAs issued under `lane == 0` go through a loop that moves them to uniform registers, which bound a
// k block (100 rows x 4096 x 11008: 19.4 -> 16.9 us; 512 rows: 94.9 -> 58.5 us).
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
// K-major operand with 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)(16 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;      // descriptor version of this architecture
  d |= (uint64_t)2 << 61;      // 128-byte swizzle
  return d;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
// A bounded wait: false if it ran out
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (unsigned it = 0; it < SPIN_LIMIT; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(POLL_NS) : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// 2-D tiled copy: box {64 k, Mpad rows} at (k element x, row y); x * 2 bytes is a multiple of 128
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// fp16 pair (offset + code) -> fp16(code * scale), the reference's operand rounding: offset + code and code
// are exact in fp16, the product rounds once
template <uint32_t OFFSET>
__device__ __forceinline__ uint32_t deq_pair(uint32_t v, __half2 scale) {
  return h2_as_u32(__hmul2(__hsub2(u32_as_h2(v), u32_as_h2(OFFSET)), scale));
}

// One 16-row step of a lane's two 16-row tiles: the tile words w0, w1 and the scales of k = 4t .. 4t + 3 to the
// registers of columns 8 st + 2t, + 1 of st_16x256b_x4
__device__ __forceinline__ void dequant_step(const unsigned char* w, const unsigned char* sc, uint32_t (&r)[2][16], int st) {
  const uint2 wv = *reinterpret_cast<const uint2*>(w);
  const uint2 sv = *reinterpret_cast<const uint2*>(sc);
  const __half2 s01 = u32_as_h2(sv.x), s23 = u32_as_h2(sv.y);     // scales of k = 4t, 4t+1 and 4t+2, 4t+3
  const uint32_t wds[2] = {wv.x, wv.y};
#pragma unroll
  for (int j2 = 0; j2 < 2; ++j2) {
    const uint32_t v = wds[j2];
    // bits 4..7 of a 16-bit half under the exponent of 64: 72 + code; bits 0..3 under that of 1024: 1032 + code (the
    // sign bit of the code flipped; in the low nibbles of a copy it is so already).  One shift a word instead of three
    constexpr uint32_t HI = 0x54805480u, LO = 0x64086408u, LO_EXP = 0x64006400u;
    const uint32_t v8 = v >> 8;
    r[j2][4 * st + 0] = deq_pair<HI>(lop3_and_xor(v, 0x00F000F0u, HI), s01);      // row g,     k + 0, 1: column 8 st + 2t
    r[j2][4 * st + 1] = deq_pair<HI>(lop3_and_xor(v8, 0x00F000F0u, HI), s23);     // row g,     k + 2, 3: column 8 st + 2t + 1
    r[j2][4 * st + 2] = deq_pair<LO>(lop3_and_xor(v, 0x000F000Fu, LO_EXP), s01);      // row g + 8, column 8 st + 2t
    r[j2][4 * st + 3] = deq_pair<LO>(lop3_and_xor(v8, 0x000F000Fu, LO_EXP), s23);     // row g + 8, column 8 st + 2t + 1
  }
}

// 16 rows x 16 columns of 32 bits to tensor memory: lane (g, t) gives, per group of 8 columns, rows g and
// g + 8 at columns 2t and 2t + 1 — the accumulator-fragment layout of mma.m16n8, which is also how the
// tiled weight format hands out its words
__device__ __forceinline__ void st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor]
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}

}  // namespace ttc
}  // namespace q40

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against the driver library)
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static inline EncodeTiledFn ttc_encode_fn() {
  static std::atomic<void*> cached{nullptr};
  void* fn = cached.load(std::memory_order_acquire);
  if (fn) return (EncodeTiledFn)fn;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess || !fn) {
    (void)cudaGetLastError();
    return nullptr;
  }
  cached.store(fn, std::memory_order_release);
  return (EncodeTiledFn)fn;
}
// A call of it.  The driver wants the device's context current in the calling thread, which a thread that has made no call of the runtime so far
// does not have (all that a launch asks of the runtime before may be known already)
template <typename... Args>
static CUresult ttc_encode(EncodeTiledFn fn, Args... args) {
  const CUresult r = fn(args...);
  int dev = 0;
  if (r == CUDA_SUCCESS || cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return r;
  return fn(args...);
}

// q40_gemm_pair_tc.cu: C_i[M, N_i] = A[M, K] @ deq(B_i) on tiled copies by pairs of CTAs, or, with `silu` and two matrices, c[0] =
// silu(A @ deq(B_0)) * (A @ deq(B_1)).  M <= 128: any order of the sums over k; above: the sums of `ranges` equal k
// ranges (64-row steps, rounded up), added in order.  `workspace` (may be NULL): see q40_gemm_tiled_tc_ws.
// Q40_E_UNSUPPORTED also if the launch is estimated to take `beat_ns` or longer.
int q40_pair_gemm(int nmat, const void* a, int64_t lda, const void* const* bw_tiled, void* const* c, const int64_t* ldc,
                  const int* n_cols, int M, int K, int ranges, int silu, void* workspace, size_t workspace_bytes, double beat_ns,
                  int* err, int use_pdl, void* stream);
