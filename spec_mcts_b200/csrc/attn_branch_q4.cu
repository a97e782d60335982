// Decode attention for one query token per branch over that branch's packed Q4_0 cache, and the merge with a shared prefix's
// partial results; with rotary tables also the rotation of the new token and its append.  One, two or four warps per row (branch, query head).
//
// A row is a matrix-vector product, so the tensor cores' products are mostly unused columns; what counts is that an MMA takes the
// place of 16 x 16 multiply-adds and of the shuffles that sum them: 22 instructions a key and 35 cycles of a scheduler where
// scalar products take 36 and 60.  Per 16 keys:
//   scores   A = codes of K as fp16 (16 keys x 128 dims, exact), B = the query in every column; the two scales of a key multiply the
//            fp32 sums of its two halves
//   output   A = V transposed (dims x 16 keys), fp16(code * scale), B = the weights: column pairs hold fp16(p) and fp16(p - fp16(p)),
//            so that weights keep 22 bits and the sums of both columns are the row's (weight_parts)
// Dims and keys of a contraction may be in any order as long as both operands agree, so lanes take them as memory has them: lane
// (g, t) of eight times four holds bytes 16t.. of keys g and g + 8 for the scores (a warp's load covers eight whole rows) and bytes 8g.. of
// keys 2t, 2t + 1, 2t + 8 and 2t + 9 for the output.  All four lanes of a key end up with its score, and all four lanes t with the
// output's dims 8g.. and 64 + 8g.. .
//
// Stands in for the reference's dequantisation of the whole suffix and SDPA on it (hf_model_q40_kv_shared.py:346-405).
#include <type_traits>

#include "attn_tile.cuh"

namespace q40 {

constexpr int Q4_NW = 4;                        // warps of a CTA
constexpr int CHUNK = 32;                       // keys of a warp's iteration
constexpr int STAGES = 2;                       // of a warp's ring: [keys' codes][values' codes][keys' scales][values' scales]
constexpr int V_OFF = CHUNK * 64, KS_OFF = 2 * V_OFF, VS_OFF = KS_OFF + CHUNK * 4, STAGE_BYTES = VS_OFF + CHUNK * 4;
constexpr int RING_BYTES = Q4_NW * STAGES * STAGE_BYTES;
// Byte `at` of row r of the values' codes: two rows share 128 bytes, whose 32-byte quarters are permuted so that the quarters that lanes
// (g, t) of half a warp read of rows 2t lie in different banks
__device__ __forceinline__ int v_at(int r, int at) {
  return (r >> 1) * 128 + 32 * ((2 * (r & 1) + (at >> 5)) ^ ((r >> 1) & 3)) + (at & 31);
}

template <bool ROT>
using Q4Args = std::conditional_t<ROT, BranchRotArgs, BranchArgs>;

// The codes of a word's bytes 0 and 2 in its high or low nibbles, exactly
__device__ __forceinline__ __half2 nibbles_hi(uint32_t w) {
  return __hsub2(u32_as_h2(lop3_and_xor(w, 0x00F000F0u, 0x54805480u)), u32_as_h2(0x54805480u));      // 72 + code
}

// sum over the eight lanes g of (g, t)
__device__ __forceinline__ float sum_g(float v) {
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float max_g(float v) {
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src));
}
// The first of a sum's products
__device__ __forceinline__ void mma_f16_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// SC4: the scales of a row are one aligned word
template <bool ROT, int WPR, bool SC4>
__global__ void __launch_bounds__(Q4_NW * 32, 4)
attn_branch_q4_kernel(const Q4Args<ROT> a) {
  constexpr int D = ATTN_D, RT = WPR * 32;       // threads of a row
  asm volatile("griddepcontrol.launch_dependents;");
  // behind a prefix pass, which lets this launch start only when everything in front of it is done: see attn_branch_kernel
  if (!a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int slot = warp / WPR, part = warp % WPR;           // row of this CTA, warp of the row
  const int64_t bh = (int64_t)blockIdx.x * (Q4_NW / WPR) + slot;
  const int64_t rows = a.rows;
  if (bh >= rows) return;                        // whole rows, which meet at no common barrier
  const int b = (int)(bh / a.H), h = (int)(bh % a.H), hk = h / (a.H / a.Hkv);

  int at = a.pos[b];                             // with rotation the tables bound the position, at which the token is appended too
  if constexpr (ROT) at = min(max(at, 0), a.n_pos - 1);
  const int own = at - a.prefix_len[0], len = min(max(own, 0), a.max_t);

  // the query: dims 16t .. and 64 + 16t .., as column of the scores' B operand
  uint32_t qf[8][2];
  {
    uint4 lo[2], hi[2];
    const __half* qp = a.q + (int64_t)b * a.q_stride + h * D + 16 * t;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      lo[i] = *reinterpret_cast<const uint4*>(qp + 8 * i);
      hi[i] = *reinterpret_cast<const uint4*>(qp + 64 + 8 * i);
      if constexpr (ROT) {
        const int64_t o = (int64_t)at * 64 + 16 * t + 8 * i;
        rotate_dims(lo[i], hi[i], __ldg(reinterpret_cast<const uint4*>(a.cos_tbl + o)), __ldg(reinterpret_cast<const uint4*>(a.sin_tbl + o)));
      }
    }
    const uint32_t *l = reinterpret_cast<const uint32_t*>(lo), *u = reinterpret_cast<const uint32_t*>(hi);
#pragma unroll
    for (int j = 0; j < 4; ++j) {                // a word's bytes come out as (0, 2) and (1, 3)
      qf[j][0] = prmt(l[2 * j], l[2 * j + 1], 0x5410);
      qf[j][1] = prmt(l[2 * j], l[2 * j + 1], 0x7632);
      qf[4 + j][0] = prmt(u[2 * j], u[2 * j + 1], 0x5410);
      qf[4 + j][1] = prmt(u[2 * j], u[2 * j + 1], 0x7632);
    }
  }
  // 72 times the sum of the query's halves: high nibbles come as 72 + code (exact; the sums' 24 bits are plenty), low ones as codes
  float q72 = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float2 f = __half22float2(u32_as_h2(qf[j][r]));
      q72 += f.x + f.y;
    }
  q72 += __shfl_xor_sync(0xffffffffu, q72, 1);
  q72 = 72.f * (q72 + __shfl_xor_sync(0xffffffffu, q72, 2));
  float m = -CUDART_INF_F, l = 0.f;              // m: WEIGHT_BITS below the largest score; l: of this lane's keys
  float acc[8][4];                               // dims 8g + 2i (columns: both parts of the weights) and 8g + 2i + 1; from 4: 64 + ..
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  const int64_t row0 = (int64_t)b * a.max_t * a.Hkv + hk;
  // A warp's chunks come through a ring of its own: 16 bytes of keys (lane >> 2) + 8j at a time, a key's scales by its lane.  Keys beyond
  // the length: the last one's bytes, with a weight of 0
  extern __shared__ __align__(128) unsigned char rings[];
  unsigned char* const ring = rings + warp * (STAGES * STAGE_BYTES);
  const uint32_t ring0 = smem_u32(ring);
  const int8_t *kbase = a.kq + row0 * 64 + 16 * t, *vbase = a.vq + row0 * 64 + 16 * t;
  const __half *ksbase = a.ksc + row0 * 2, *vsbase = a.vsc + row0 * 2;
  const auto request = [&](int t0, int stage) {
    const uint32_t st = ring0 + stage * STAGE_BYTES;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t row = (uint32_t)(min(t0 + 8 * j + g, len - 1) * a.Hkv);
      cp_async16(st + (8 * j + g) * 64 + 16 * t, kbase + row * 64, true);
      cp_async16(st + V_OFF + v_at(8 * j + g, 16 * t), vbase + row * 64, true);
    }
    const size_t row = (uint32_t)(min(t0 + lane, len - 1) * a.Hkv);
    if (SC4) {
      cp_async4(st + KS_OFF + 4 * lane, ksbase + row * 2);
      cp_async4(st + VS_OFF + 4 * lane, vsbase + row * 2);
    } else {
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(st + KS_OFF + 4 * lane), "r"(h2_as_u32(__halves2half2(__ldg(ksbase + row * 2), __ldg(ksbase + row * 2 + 1)))));
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(st + VS_OFF + 4 * lane), "r"(h2_as_u32(__halves2half2(__ldg(vsbase + row * 2), __ldg(vsbase + row * 2 + 1)))));
    }
  };
#pragma unroll
  for (int i = 0; i < STAGES; ++i) {
    const int t0 = (part + i * WPR) * CHUNK;
    if (t0 < len) request(t0, i);
    cp_async_commit();
  }
  int stage = 0;
#pragma unroll 1
  for (int t0 = part * CHUNK; t0 < len; t0 += WPR * CHUNK) {
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const unsigned char* st = ring + stage * STAGE_BYTES;
    float s[2][2], mnew = m;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float ch[4], cl[4];
      const uint4 ka = *reinterpret_cast<const uint4*>(st + (16 * i + g) * 64 + 16 * t), kb = *reinterpret_cast<const uint4*>(st + (16 * i + 8 + g) * 64 + 16 * t);
      const uint32_t wa[4] = {ka.x, ka.y, ka.z, ka.w}, wb[4] = {kb.x, kb.y, kb.z, kb.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t x = wa[j], y = wb[j], x8 = x >> 8, y8 = y >> 8;
        constexpr uint32_t M = 0x00F000F0u, E = 0x54805480u;
        const uint32_t h0 = lop3_and_xor(x, M, E), h1 = lop3_and_xor(y, M, E), h2 = lop3_and_xor(x8, M, E), h3 = lop3_and_xor(y8, M, E);
        const uint32_t l0 = h2_as_u32(codes_lo_to_h2(x)), l1 = h2_as_u32(codes_lo_to_h2(y)), l2 = h2_as_u32(codes_lo_to_h2(x8)),
                       l3 = h2_as_u32(codes_lo_to_h2(y8));
        if (j == 0) {
          mma_f16_zero(ch, h0, h1, h2, h3, qf[j][0], qf[j][1]);
          mma_f16_zero(cl, l0, l1, l2, l3, qf[4 + j][0], qf[4 + j][1]);
        } else {
          mma_f16(ch, h0, h1, h2, h3, qf[j][0], qf[j][1]);
          mma_f16(cl, l0, l1, l2, l3, qf[4 + j][0], qf[4 + j][1]);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {              // columns are alike: rows g and g + 8 of one
        const float2 sc = __half22float2(*reinterpret_cast<const __half2*>(st + KS_OFF + 4 * (16 * i + 8 * r + g)));
        s[i][r] = t0 + 16 * i + 8 * r + g < len ? fmaf(sc.x, ch[2 * r] - q72, sc.y * cl[2 * r]) * a.scale_log2 : -CUDART_INF_F;
        mnew = fmaxf(mnew, s[i][r] - WEIGHT_BITS);
      }
    }
    mnew = max_g(mnew);
    if (mnew != m) {
      const float corr = ex2(m - mnew);
      l *= corr;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= corr;
      m = mnew;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t pk[2];                            // of keys g and g + 8: fp16(p) and what that leaves
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float p = ex2(s[i][r] - m);
        l += p;
        pk[r] = weight_parts(p);
      }
      const auto of_key = [&](const uint32_t (&v)[2], int r) { return __shfl_sync(0xffffffffu, v[r >> 1], 8 * t + 4 * (r & 1)); };
      const uint32_t sel = g & 1 ? 0x7632u : 0x5410u;                     // odd columns: the rest
      const uint32_t b0 = prmt(of_key(pk, 0), of_key(pk, 1), sel), b1 = prmt(of_key(pk, 2), of_key(pk, 3), sel);
      const uint2 s01 = *reinterpret_cast<const uint2*>(st + VS_OFF + 4 * (16 * i + 2 * t)), s23 = *reinterpret_cast<const uint2*>(st + VS_OFF + 4 * (16 * i + 8 + 2 * t));
      const __half2 h01 = u32_as_h2(prmt(s01.x, s01.y, 0x5410)), l01 = u32_as_h2(prmt(s01.x, s01.y, 0x7632));
      const __half2 h23 = u32_as_h2(prmt(s23.x, s23.y, 0x5410)), l23 = u32_as_h2(prmt(s23.x, s23.y, 0x7632));
      uint2 vw[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) vw[r] = *reinterpret_cast<const uint2*>(st + V_OFF + v_at(16 * i + 8 * (r >> 1) + 2 * t + (r & 1), 8 * g));
#pragma unroll
      for (int j = 0; j < 4; ++j) {              // bytes 2j and 2j + 1 of the four keys
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int by = 2 * (j & 1) + e;
          const uint32_t pick = by | by << 4 | (4 + by) << 8 | (4 + by) << 12;
          const uint32_t x = j < 2 ? prmt(vw[0].x, vw[1].x, pick) : prmt(vw[0].y, vw[1].y, pick);
          const uint32_t y = j < 2 ? prmt(vw[2].x, vw[3].x, pick) : prmt(vw[2].y, vw[3].y, pick);
          hi[e] = h2_as_u32(__hmul2(nibbles_hi(x), h01));
          hi[2 + e] = h2_as_u32(__hmul2(nibbles_hi(y), h23));
          lo[e] = h2_as_u32(__hmul2(codes_lo_to_h2(x), l01));
          lo[2 + e] = h2_as_u32(__hmul2(codes_lo_to_h2(y), l23));
        }
        mma_f16(acc[j], hi[0], hi[1], hi[2], hi[3], b0, b1);
        mma_f16(acc[4 + j], lo[0], lo[1], lo[2], lo[3], b0, b1);
      }
    }
    __syncwarp();
    if (t0 + STAGES * WPR * CHUNK < len) request(t0 + STAGES * WPR * CHUNK, stage);
    cp_async_commit();
    if (++stage == STAGES) stage = 0;
  }
  l = sum_g(l);
  float o[16];                                   // dims 8g .. and 64 + 8g ..
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o[2 * i] = both_parts(acc[i][0], acc[i][1]);
    o[2 * i + 1] = both_parts(acc[i][2], acc[i][3]);
  }

  // the token being decoded attends to its own, un-quantised K/V: one more key for a row's first warp
  if (a.cur_k != nullptr && part == 0) {
    const int64_t off = (int64_t)b * a.cur_stride + hk * D + 8 * g;
    uint4 k0 = *reinterpret_cast<const uint4*>(a.cur_k + off), k1 = *reinterpret_cast<const uint4*>(a.cur_k + off + 64);
    const uint4 v0 = *reinterpret_cast<const uint4*>(a.cur_v + off), v1 = *reinterpret_cast<const uint4*>(a.cur_v + off + 64);
    const __half* qp = a.q + (int64_t)b * a.q_stride + h * D + 8 * g;
    uint4 q0 = *reinterpret_cast<const uint4*>(qp), q1 = *reinterpret_cast<const uint4*>(qp + 64);
    if constexpr (ROT) {
      const uint4 c = __ldg(reinterpret_cast<const uint4*>(a.cos_tbl + (int64_t)at * 64 + 8 * g)),
                  sn = __ldg(reinterpret_cast<const uint4*>(a.sin_tbl + (int64_t)at * 64 + 8 * g));
      rotate_dims(q0, q1, c, sn);
      rotate_dims(k0, k1, c, sn);
      if (h % (a.H / a.Hkv) == 0 && own >= 0 && own < a.max_t) {             // the first query head of a kv head
        const int64_t row = row0 + (int64_t)own * a.Hkv;
        append_row<4>(k0, k1, const_cast<int8_t*>(a.kq) + row * 64, const_cast<__half*>(a.ksc) + row * 2, g, 0xffffffffu, t == 0);
        append_row<4>(v0, v1, const_cast<int8_t*>(a.vq) + row * 64, const_cast<__half*>(a.vsc) + row * 2, g, 0xffffffffu, t == 0);
      }
    }
    const __half2 *qh0 = reinterpret_cast<const __half2*>(&q0), *qh1 = reinterpret_cast<const __half2*>(&q1);
    const __half2 *kh0 = reinterpret_cast<const __half2*>(&k0), *kh1 = reinterpret_cast<const __half2*>(&k1);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) dot = dot2(qh1[i], kh1[i], dot2(qh0[i], kh0[i], dot));
    const float sc = sum_g(dot) * a.scale_log2, mnew = fmaxf(m, sc), corr = ex2(m - mnew), p = ex2(sc - mnew);
    l = l * corr + p;
    const __half2 *vh0 = reinterpret_cast<const __half2*>(&v0), *vh1 = reinterpret_cast<const __half2*>(&v1);
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

  __shared__ float sm_m[Q4_NW], sm_l[Q4_NW];
  __shared__ __align__(16) float sm_o[Q4_NW][D];
  if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
  // lane t writes four of its dims
  *reinterpret_cast<float4*>(&sm_o[warp][(t >> 1) * 64 + 8 * g + 4 * (t & 1)]) =
      t == 0 ? make_float4(o[0], o[1], o[2], o[3]) : t == 1 ? make_float4(o[4], o[5], o[6], o[7])
      : t == 2 ? make_float4(o[8], o[9], o[10], o[11]) : make_float4(o[12], o[13], o[14], o[15]);
  if (a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  RowMerge<WPR, RT> merge;
  merge.load(a, rows, bh, part * 32 + lane, lane);
  if (WPR == 1) __syncwarp();
  else if (WPR == Q4_NW) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(RT) : "memory");
  merge.finish(a, rows, bh, part * 32 + lane, lane, sm_m + slot * WPR, sm_l + slot * WPR, sm_o[slot * WPR]);
}

template <bool ROT, int WPR, bool SC4>
static int launch_q4(const BranchRotArgs& a, cudaStream_t st) {
  static std::atomic<uint64_t> ready;
  cudaError_t e = q40_allow_smem(ready, (const void*)attn_branch_q4_kernel<ROT, WPR, SC4>, RING_BYTES);
  const unsigned grid = (unsigned)((a.rows + Q4_NW / WPR - 1) / (Q4_NW / WPR));
  if (e == cudaSuccess)
    e = q40_launch_pdl(attn_branch_q4_kernel<ROT, WPR, SC4>, dim3(grid), dim3(Q4_NW * 32), RING_BYTES, st, (const Q4Args<ROT>&)a);
  return e == cudaSuccess ? Q40_OK : (int)e;
}

// Warps of a row by the number of rows: as many as keep all SMs busy, no more, since every warp starts, and is merged, by itself.  (The
// host does not know a row's length.)  Us with the prefix pass (512 keys) and rotation, 20 / 64 / 128 / 220 own keys, one, two and four warps:
// 320 rows 7.9 / 9.2 / 11.6 / 15.1, 9.0 / 10.3 / 12.9 / 16.1, 8.9 / 9.3 / 10.6 / 12.7; 640 rows 10.6 / 11.9 / 14.6 / 18.3,
// 9.9 / 11.3 / 13.9 / 17.4, 11.6 / 12.3 / 13.7 / 16.4; 1408 rows 13.4 / 16.4 / 21.2 / 27.7, 14.8 / 16.8 / 20.3 / 25.3,
// 19.6 / 21.5 / 24.1 / 29.0; 2048 rows 14.7 / 18.2 / 22.6 / 30.0, 17.4 / 20.1 / 24.6 / 31.4, 25.6 / ..
// By scalar products (eight lanes a key): 9.5 / 9.6 / 11.6 / 15.3, 10.1 / 12.0 / 15.7 / 21.5, 14.4 / 18.1 / 24.4 / 33.3, 17.0 / 21.4 / 28.5 /
// 40.2, 3200 rows 23.6 / 29.9 / 41.1 / 57.9 (18.8 / 22.9 / 29.4 / 41.9 here).  Keys and values straight to registers instead of through
// the ring: 20.4 / 25.2 / 33.8 / 47.6; three stages, which leave the prefix pass no room beside: 18.8 / 23.3 / 32.6 / 45.6; five CTAs
// an SM, with spills: 19.5 / 23.5 / 30.9 / 44.2
// Scales off four bytes by the same rule (without rotation, 32 heads, 200 own keys behind 40, two warps a row and so: 6 branches 14.3 us and 10.2, 10
// 14.4 and 11.1; 20 own keys behind 512, 100 branches 19.7 and 16.4)
int launch_branch_q4(const BranchRotArgs& a, bool rotate, cudaStream_t st) {
  const int w = a.rows <= 3 * 148 ? 4 : a.rows <= 10 * 148 ? 2 : 1;
  if (rotate) return w == 1 ? launch_q4<true, 1, true>(a, st) : w == 2 ? launch_q4<true, 2, true>(a, st) : launch_q4<true, 4, true>(a, st);
  if (!q40_aligned(a.ksc, 4) || !q40_aligned(a.vsc, 4))
    return w == 1 ? launch_q4<false, 1, false>(a, st) : w == 2 ? launch_q4<false, 2, false>(a, st) : launch_q4<false, 4, false>(a, st);
  return w == 1 ? launch_q4<false, 1, true>(a, st) : w == 2 ? launch_q4<false, 2, true>(a, st) : launch_q4<false, 4, true>(a, st);
}

}  // namespace q40
