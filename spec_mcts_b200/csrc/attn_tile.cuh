// What the two tensor-core attention kernels (attn_prefix.cu, attn_causal.cu) share: 64-key tiles of keys and values in shared
// memory, and a warp's step over one of them.
#pragma once
#include <math_constants.h>

#include "attn_common.cuh"

namespace q40 {

constexpr int TILE_KEYS = 64;
constexpr int TILE_ROW_BYTES = ATTN_D * 2;                      // 256 B per key
constexpr int TILE_BYTES = TILE_KEYS * TILE_ROW_BYTES;          // 16 KB

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool pred) {
  const int sz = pred ? 16 : 0;  // size 0 = write zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// byte offset of 16-byte chunk `chunk` (0..15) of row `row` in a [rows][256 B] tile, XOR-swizzled so
// that the 8 rows of an ldmatrix 8x8 block fall in different bank groups
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  return (uint32_t)(row * TILE_ROW_BYTES + ((chunk ^ (row & 7)) << 4));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// NT threads request 64 keys and values: row r of the tile is key r of src, zeros from `keys` on.  A thread's rows are NT / 16
// apart, so that its addresses are sums of what does not change.
template <int NT>
__device__ __forceinline__ void load_tile(uint32_t kdst, uint32_t vdst, const __half* k, const __half* v, int64_t ldk, int64_t ldv,
                                          int keys, int tid) {
  constexpr int STEP = NT / 16;                     // a multiple of 8: the swizzle of a thread's rows is the same
  const int r0 = tid >> 4, ch = tid & 15;
  const uint32_t off = tile_off(r0, ch);
  const __half *kp = k + r0 * ldk + ch * 8, *vp = v + r0 * ldv + ch * 8;
#pragma unroll
  for (int i = 0; i < TILE_KEYS / STEP; ++i) {
    const bool ok = r0 + i * STEP < keys;
    cp_async16(kdst + off + i * STEP * TILE_ROW_BYTES, ok ? kp + i * STEP * ldk : k, ok);
    cp_async16(vdst + off + i * STEP * TILE_ROW_BYTES, ok ? vp + i * STEP * ldv : v, ok);
  }
}

// Maximum of a row that has met no score above it: below every finite score, and finite, since -inf - -inf is no number
// (with a test for -inf in each tile: attention of 100 branches over 400 + 64 keys 25.34 us instead of 25.17, a prompt of 512 18.27
// instead of 18.17)
constexpr float NO_KEY = -3e38f;

// State of a warp's 16 query rows; lane (g, t) has rows g and g + 8
struct WarpRows {
  uint32_t qa[8][4];                                // A fragments of Q
  float m[2], l[2], o[16][4];                       // running maximum (log2 domain), this lane's part of the sum, outputs

  __device__ __forceinline__ void init() {
    m[0] = m[1] = NO_KEY;
    l[0] = l[1] = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
  }
  // 16 rows from a swizzled tile, `row0` the warp's first
  __device__ __forceinline__ void load_q(uint32_t tile, int row0, int lane) {
    const int mi = lane >> 3, row = row0 + (lane & 7) + (mi & 1) * 8;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) ldsm_x4(tile + tile_off(row, 2 * ks + (mi >> 1)), qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
  }

  // KEYS keys of a tile: S = Q K^T, online softmax, O += P V.  With MASK, key i of the tile counts for row g below n0 and for row g + 8
  // below n1.  A row all of whose scores so far are -inf keeps its sum and outputs at zero.
  template <bool MASK, int KEYS = TILE_KEYS>
  __device__ __forceinline__ void step(uint32_t kt, uint32_t vt, float scale_log2, int n0, int n1, int lane) {
    const int t = lane & 3;
    constexpr int NT = KEYS / 8;
    float s[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ks += 2) {
      // eight sums in turn: one after the other, each MMA would wait for the one before it
      uint32_t kb[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        ldsm_x4(kt + tile_off(nt * 8 + (lane & 7), 2 * ks + (lane >> 3)), kb[nt][0], kb[nt][1], kb[nt][2], kb[nt][3]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) mma_f16(s[nt], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[nt][0], kb[nt][1]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        mma_f16(s[nt], qa[ks + 1][0], qa[ks + 1][1], qa[ks + 1][2], qa[ks + 1][3], kb[nt][2], kb[nt][3]);
    }
    float mx[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[nt][j] *= scale_log2;
        if (MASK && nt * 8 + 2 * t + (j & 1) >= ((j >> 1) ? n1 : n0)) s[nt][j] = -CUDART_INF_F;
        mx[j >> 1] = fmaxf(mx[j >> 1], s[nt][j]);
      }
    float corr[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      const float mnew = fmaxf(m[r], mx[r]);
      corr[r] = ex2(m[r] - mnew);
      m[r] = mnew;
      l[r] *= corr[r];
    }
    float ls[2] = {0.f, 0.f};
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = ex2(s[nt][j] - m[j >> 1]);
        s[nt][j] = p;
        ls[j >> 1] += p;
      }
    l[0] += ls[0];       // combined across the quad at the end
    l[1] += ls[1];
    if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {      // a maximum has moved
#pragma unroll
      for (int dt = 0; dt < 16; ++dt) {
        o[dt][0] *= corr[0]; o[dt][1] *= corr[0];
        o[dt][2] *= corr[1]; o[dt][3] *= corr[1];
      }
    }
#pragma unroll
    for (int kk = 0; kk < KEYS / 16; ++kk) {
      const uint32_t a0 = pack_h2(s[2 * kk][0], s[2 * kk][1]);
      const uint32_t a1 = pack_h2(s[2 * kk][2], s[2 * kk][3]);
      const uint32_t a2 = pack_h2(s[2 * kk + 1][0], s[2 * kk + 1][1]);
      const uint32_t a3 = pack_h2(s[2 * kk + 1][2], s[2 * kk + 1][3]);
      const int vrow = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int dt = 0; dt < 16; dt += 2) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4_t(vt + tile_off(vrow, dt + (lane >> 4)), b0, b1, b2, b3);
        mma_f16(o[dt], a0, a1, a2, a3, b0, b1);
        mma_f16(o[dt + 1], a0, a1, a2, a3, b2, b3);
      }
    }
  }
  // the rows' sums over the quad; the maximum of a row without a finite score is -inf
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (m[r] == NO_KEY) m[r] = -CUDART_INF_F;
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
  }
};

}  // namespace q40
