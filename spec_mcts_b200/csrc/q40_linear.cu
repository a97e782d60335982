// y[M, N] = x[M, K] @ deq(W)^T for W [N, K] with groups of 64 along K (the layout of quantize_q40 on a Linear weight), up to 32 rows a
// launch (from 9 on where q40_pair_linear, on tcgen05, is not the faster one: see q40_gemm_nk).
//
// One CTA per SM: up to five 16-row tiles of W over the whole k range, or, where the activations do not fit shared memory or
// tiles are few, a cluster of two or four CTAs that share it.  The activations are staged once, W comes straight into the
// registers of the lanes that expand it, the 16 warps split k (and tiles) and their sums meet in shared memory: no scratch
// in global memory.  Operands are the reference's: fp16(code * scale), fp32 sums.
//
// What bounds it: instructions of the expansion (about 230 a warp and 128 k of 16 rows, of which 100 make operands) and a warp's chain
// of loads, four of 1 KB on their way.  Microseconds of the launch alone with W in L2, here and by gemv_nk_kernel (64 rows x part of k per CTA,
// scratch and tickets): 10 rows x 4096 x 11008 13.7 and 18.2 (calls of linear_q40 one after the other: 12.0, without programmatic launch
// 14.3, and 18.4), x 11008 x 4096 17.8 and 18.7; 1 row x 4096 x 4096 5.8 and 7.6, x 11008 x 11008 24.0 and 27.7; 10 rows x 1024 x 1000 4.0 and
// 7.0; 20 rows x 4096 x 11008 20.1 and 29.3.  No gain: weights prefetched to L2 at the start (14.2).
#include <cooperative_groups.h>

#include <algorithm>

#include "q40_common.cuh"

namespace cg = cooperative_groups;

namespace q40 {
namespace nk {

constexpr int WARPS = 16, THREADS = WARPS * 32;
constexpr int STEP = 128;                          // k of a step: one packed row of two groups, 64 bytes
constexpr int XPAD = 8;                            // halves: rows of activations start 16 bytes further in the banks
constexpr int M_LD = 20;                           // floats between rows of a 16 x 16 tile's sums
constexpr int TILES = 5;                           // 16-row tiles of W of a cluster, at most
constexpr int SMEM_MAX = 227 * 1024;

struct Args {
  const __half* x;
  int64_t ldx;
  const uint8_t* w;
  const __half* s;
  __half* y;
  int64_t ldy;
  int M, N, K;
  int tiles, kw, ksteps;     // tiles of a cluster, warps that share a tile's k range, steps of a CTA's k range
  int xk;                    // k of a CTA's range
  int wide_s, wide_x;        // scales of four groups by one 8-byte load; rows of x on 16-byte boundaries (else 8)
  int off_slab, off_out;
};

// Two codes of a packed word (bytes 0 and 2) as fp16, exact: 72 + code (bits 4..7 of a 16-bit half under the exponent of 64, or 1032 + code,
// bits 0..3 under that of 1024; the code's sign bit flipped) less the constant
__device__ __forceinline__ uint32_t codes_hi(uint32_t w) {
  return h2_as_u32(__hsub2(u32_as_h2(lop3_and_xor(w, 0x00F000F0u, 0x54805480u)), u32_as_h2(0x54805480u)));
}
__device__ __forceinline__ uint32_t codes_lo(uint32_t w) { return h2_as_u32(codes_lo_to_h2(w)); }

struct Steps { uint4 a[2], b[2]; uint2 sa, sb; };  // two steps of rows g and g + 8: 16 packed bytes each, and the four groups' scales

__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MT>
__global__ void __launch_bounds__(THREADS, 1) linear_kernel(const Args p) {
  extern __shared__ __align__(16) unsigned char smem[];
  cg::cluster_group cluster = cg::this_cluster();
  // started while the launch in front drains (which may be the one that writes the weights): 0.9 us of a call
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __half* xs = reinterpret_cast<__half*>(smem);                       // [M][xk + XPAD], in fours of the order x0 x2 x1 x3
  float* slab = reinterpret_cast<float*>(smem + p.off_slab);          // [kw][TILES][MT * 8][M_LD]
  float* out = reinterpret_cast<float*>(smem + p.off_out);            // [TILES][MT * 8][16] this CTA's sums
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int c = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int kw = p.kw, tw = WARPS / kw;                               // warps: [tw][kw]
  const int wk = warp % kw, wt = warp / kw;
  const int k0 = rank * p.xk, nk = min(p.xk, p.K - k0);               // this CTA's k range
  const int steps = nk / STEP;
  const int s0 = steps * wk / kw, s1 = steps * (wk + 1) / kw;         // this warp's steps of it
  const int all_tiles = (p.N + 15) / 16;
  const int tile0 = blockIdx.x / c * p.tiles, tile1 = min(all_tiles, tile0 + p.tiles);
  const int64_t w_ld = p.K / 2, s_ld = p.K / 64;
  const int xld = p.xk + XPAD;
  const bool wide_s = p.wide_s && ((k0 / 64 + 2 * s0) & 3) == 0;      // 8-byte aligned, in every row

  // the warp's steps, two at a time, tile by tile; two such pairs are on their way to registers
  int l_tile = tile0 + wt, l_step = s0;
  const uint8_t *la = nullptr, *lb = nullptr;
  const __half *lsa = nullptr, *lsb = nullptr;
  auto rows = [&]() {
    const int64_t na = min(l_tile * 16 + g, p.N - 1), nb = min(l_tile * 16 + g + 8, p.N - 1);      // rows beyond W: not stored
    const int kb = k0 / 2 + s0 * (STEP / 2) + 16 * t, ks = k0 / 64 + 2 * s0;
    la = p.w + na * w_ld + kb;
    lb = p.w + nb * w_ld + kb;
    lsa = p.s + na * s_ld + ks;
    lsb = p.s + nb * s_ld + ks;
  };
  rows();
  auto load = [&](Steps& r) {
    if (l_tile < tile1) {
      r.a[0] = __ldg(reinterpret_cast<const uint4*>(la));
      r.b[0] = __ldg(reinterpret_cast<const uint4*>(lb));
      const bool two = l_step + 1 < s1;
      if (two) {
        r.a[1] = __ldg(reinterpret_cast<const uint4*>(la + STEP / 2));
        r.b[1] = __ldg(reinterpret_cast<const uint4*>(lb + STEP / 2));
      }
      if (two && wide_s) {
        r.sa = __ldg(reinterpret_cast<const uint2*>(lsa));
        r.sb = __ldg(reinterpret_cast<const uint2*>(lsb));
      } else {
        r.sa.x = __ldg(reinterpret_cast<const uint32_t*>(lsa));
        r.sb.x = __ldg(reinterpret_cast<const uint32_t*>(lsb));
        if (two) {
          r.sa.y = __ldg(reinterpret_cast<const uint32_t*>(lsa + 2));
          r.sb.y = __ldg(reinterpret_cast<const uint32_t*>(lsb + 2));
        }
      }
      la += STEP; lb += STEP; lsa += 4; lsb += 4;
      l_step += 2;
      if (l_step >= s1) {
        l_step = s0;
        l_tile += tw;
        rows();
      }
    }
  };
  Steps r0, r1;
  load(r0);
  load(r1);

  // ---- activations ----
  {
    const int per = nk / 8, total = p.M * per;
    constexpr int BATCH = 5;
    for (int i0 = tid; i0 < total; i0 += BATCH * THREADS) {
      uint4 v[BATCH];
      int at[BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int i = i0 + u * THREADS, m = i / per, j = i - m * per;
        at[u] = i < total ? m * xld + j * 8 : -1;
        if (i < total) {
          const __half* src = p.x + (int64_t)m * p.ldx + k0 + j * 8;
          if (p.wide_x) {
            v[u] = __ldg(reinterpret_cast<const uint4*>(src));
          } else {
            const uint2 lo = __ldg(reinterpret_cast<const uint2*>(src)), hi = __ldg(reinterpret_cast<const uint2*>(src + 4));
            v[u] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
        if (at[u] >= 0)
          *reinterpret_cast<uint4*>(xs + at[u]) = make_uint4(prmt(v[u].x, v[u].y, 0x5410), prmt(v[u].x, v[u].y, 0x7632),
                                                             prmt(v[u].z, v[u].w, 0x5410), prmt(v[u].z, v[u].w, 0x7632));
    }
  }
  __syncthreads();

  float acc[MT][4];
  auto clear = [&]() {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[mt][j] = 0.f;
  };
  clear();
  int c_tile = tile0 + wt, c_step = s0;
  // columns of the MMA beyond the last row repeat it; they are not stored
  int xrow[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) xrow[mt] = min(mt * 8 + g, p.M - 1) * xld;
  const __half* xl = xs + 16 * t + s0 * STEP;
  auto step = [&](const uint4& a, const uint4& b, uint32_t s2a, uint32_t s2b, const __half* x) {
    const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int lo = 0; lo < 2; ++lo) {               // the group in the high nibbles, and the one in the low nibbles, 64 k further
      const __half2 sa = lo ? __high2half2(u32_as_h2(s2a)) : __low2half2(u32_as_h2(s2a)), sb = lo ? __high2half2(u32_as_h2(s2b)) : __low2half2(u32_as_h2(s2b));
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        uint4 xv[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) xv[mt] = *reinterpret_cast<const uint4*>(x + xrow[mt] + lo * 64 + 4 * i);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t va = wa[i + e], vb = wb[i + e], va8 = va >> 8, vb8 = vb >> 8;
          const auto operand = [&](uint32_t w, __half2 sc) { return h2_as_u32(__hmul2(u32_as_h2(lo ? codes_lo(w) : codes_hi(w)), sc)); };
          const uint32_t a0 = operand(va, sa), a1 = operand(vb, sb), a2 = operand(va8, sa), a3 = operand(vb8, sb);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma(acc[mt], a0, a1, a2, a3, e ? xv[mt].z : xv[mt].x, e ? xv[mt].w : xv[mt].y);
        }
      }
    }
  };
  auto two_steps = [&](Steps& r) {
    const bool two = c_step + 1 < s1;
    step(r.a[0], r.b[0], r.sa.x, r.sb.x, xl);
    if (two) step(r.a[1], r.b[1], r.sa.y, r.sb.y, xl + STEP);
    load(r);
    c_step += 2;
    xl += 2 * STEP;
    if (c_step >= s1) {                            // the tile's sums over this warp's k
      float* o = slab + ((wk * TILES + c_tile - tile0) * (MT * 8) + 2 * t) * M_LD + g;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        o[mt * 8 * M_LD] = acc[mt][0];
        o[mt * 8 * M_LD + M_LD] = acc[mt][1];
        o[mt * 8 * M_LD + 8] = acc[mt][2];
        o[mt * 8 * M_LD + M_LD + 8] = acc[mt][3];
      }
      clear();
      c_tile += tw;
      c_step = s0;
      xl = xs + 16 * t + s0 * STEP;
    }
  };
#pragma unroll 1
  while (c_tile < tile1) {
    two_steps(r0);
    if (c_tile < tile1) two_steps(r1);
  }
  __syncthreads();
  // ---- sums over the warps, then over the cluster, in a fixed order ----
  const int n_el = (tile1 - tile0) * 16 * p.M;      // [tile][m][n]
  for (int e = tid; e < n_el; e += THREADS) {
    const int n = e & 15, m = (e >> 4) % p.M, tl = (e >> 4) / p.M;
    const float* s = slab + (tl * (MT * 8) + m) * M_LD + n;
    float v = s[0];
#pragma unroll 4
    for (int k = 1; k < kw; ++k) v += s[k * TILES * (MT * 8) * M_LD];
    if (c == 1) {
      const int row = (tile0 + tl) * 16 + n;
      if (row < p.N) p.y[(int64_t)m * p.ldy + row] = __float2half_rn(v);
    } else {
      out[(tl * (MT * 8) + m) * 16 + n] = v;
    }
  }
  if (c == 1) return;
  cluster.sync();
  for (int e = tid + rank * THREADS; e < n_el; e += c * THREADS) {
    const int n = e & 15, m = (e >> 4) % p.M, tl = (e >> 4) / p.M;
    float* at = out + (tl * (MT * 8) + m) * 16 + n;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = q < c ? *cluster.map_shared_rank(at, q) : 0.f;
    const int row = (tile0 + tl) * 16 + n;
    if (row < p.N) p.y[(int64_t)m * p.ldy + row] = __float2half_rn((v[0] + v[1]) + (v[2] + v[3]));
  }
  cluster.sync();                                   // sums have been read
}

template <int MT>
static int launch(Args& p, int c, int clusters, size_t smem, cudaStream_t st) {
  static std::atomic<uint64_t> ready;
  const cudaError_t e = q40_allow_smem(ready, (const void*)linear_kernel<MT>, SMEM_MAX);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(c * clusters, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t l = cudaLaunchKernelEx(&cfg, linear_kernel<MT>, p);
  return l == cudaSuccess ? Q40_OK : (int)l;
}

// The launch of least estimated time (`ns`, of what differs between launches); c == 0: none, gemv_nk_kernel takes the call
struct Plan {
  Args p{};
  int c = 0, clusters = 0, busiest = 0;            // CTAs of a cluster, clusters, steps of the busiest warp
  size_t smem = 0;
  double ns = 1e30;
};
static Plan make_plan(int M, int N, int K) {
  const int mt = M <= 8 ? 1 : (M <= 16 ? 2 : 4), tiles = (N + 15) / 16, ksteps = K / STEP;
  Plan best;
  Args p{};
  p.M = M; p.N = N; p.K = K;
  for (int c = 1; c <= 4; c *= 2) {
    if (c > ksteps) break;
    const int fit = c == 1 ? 148 : (c == 2 ? 74 : 33);
    p.tiles = (tiles + fit - 1) / fit;
    const int clusters = (tiles + p.tiles - 1) / p.tiles;
    p.ksteps = (ksteps + c - 1) / c;
    if ((c - 1) * p.ksteps >= ksteps || p.tiles > TILES) continue;      // a CTA without work; several waves
    p.xk = p.ksteps * STEP;
    for (p.kw = WARPS; p.kw >= 1; p.kw /= 2) {
      if (p.kw > ksteps - (c - 1) * p.ksteps) continue;                   // every warp has a step
      size_t off = (size_t)M * (p.xk + XPAD) * 2;
      off = (off + 15) & ~(size_t)15;
      p.off_slab = (int)off; off += (size_t)p.kw * TILES * mt * 8 * M_LD * 4;
      p.off_out = (int)off; off += c > 1 ? (size_t)TILES * mt * 8 * 16 * 4 : 0;
      if (off > (size_t)SMEM_MAX) continue;
      // steps of the busiest warp (which come in pairs: an odd one counts a quarter more), staging, sums over warps, what a cluster's exchange
      // costs.  (Without the quarter 1 row x 2048 x 10711, where a warp had five single steps, 10.2 us, 8.8 by gemv_nk_kernel; now 7.3)
      const int tw = WARPS / p.kw, warp_tiles = (p.tiles + tw - 1) / tw, warp_steps = (p.ksteps + p.kw - 1) / p.kw;
      const double ns = warp_tiles * (warp_steps + 0.25 * (warp_steps & 1)) * (160.0 + 110.0 * mt) + p.xk * M * 0.03 + p.kw * 20.0 + (c > 1 ? 1200 : 0);
      if (ns < best.ns) best = {p, c, clusters, warp_tiles * warp_steps, off, ns};
    }
  }
  // gemv_nk_kernel instead, where it is the faster one with weights from HBM (us here and there).  Above eight rows, where activations leave room for
  // few warps' sums, so that one has a long chain of steps: 16 rows x 7040 x 9825 45.4 and 31.9, 55 steps; 9 x 11008 x 11008 43.5 and 36.9, 43; 24 x
  // 8320 x 3197 29.7 and 28.1, 33; but 12 x 8704 x 8754 27.8 and 31.1, 34, with tiles spread evenly; 16 x 6528 x 8146 25.9 and 27.7, 26.  Up to four,
  // where CTAs have a quarter less to do on average than the busiest and scales lie so that a step's come in two loads: 1 row x 4224 x 4963 10.0
  // and 9.0, 4 rows x 10880 x 2893 14.2 and 12.3, x 6016 x 5185 12.6 and 12.1; but 1 x 1152 x 2596, 2 steps, 4.3 and 5.0.  (From L2 this
  // kernel is the faster one of most of these: 32.3 and 28.6, 30.6 and 33.4, 22.8 and 24.2 above eight rows, 8.2 and 8.6, 11.7 and 11.5, 10.2 and 10.9.)
  const double even = !best.c ? 1 : (double)tiles * ksteps / (148.0 * best.p.tiles * best.p.ksteps);
  if (best.c && (M > 8 ? best.busiest >= (even < 0.9 ? 30 : 40) : M <= 4 && K % 256 != 0 && even < 0.75 && best.busiest >= 6)) best.c = 0;
  return best;
}

}  // namespace nk
}  // namespace q40

// About how long q40_linear takes for 9 to 32 rows, nanoseconds (1e30: it does not take the call).  Measured, and by this: 10 rows x 1024 x 1000
// 3.6 and 3.8 us, 16 x 2048 x 2048 4.9 and 5.3, x 4096 x 11008 13.1 and 12.9 (14.7 with weights from HBM), 20 rows 17.3 and 17.6
double q40_linear_ns(int M, int N, int K) {
  const q40::nk::Plan p = q40::nk::make_plan(M, N, K);
  return p.c ? 2200 + 1.75 * p.ns : 1e30;
}

// q40_gemm_nk for up to 32 rows and groups of 64, or Q40_E_UNSUPPORTED.  Arguments are checked.
int q40_linear(const void* x, int64_t ldx, const void* wq, const void* ws, void* y, int64_t ldy, int M, int N, int K, void* stream) {
  using namespace q40;
  using namespace q40::nk;
  if (M > 32) return Q40_E_UNSUPPORTED;
  Plan plan = make_plan(M, N, K);
  if (plan.c == 0) return Q40_E_UNSUPPORTED;
  Args& p = plan.p;
  p.wide_s = K % 256 == 0 && q40_aligned(ws, 8);
  p.wide_x = q40_aligned(x, 16) && ldx % 8 == 0;
  p.x = (const __half*)x; p.ldx = ldx; p.w = (const uint8_t*)wq; p.s = (const __half*)ws; p.y = (__half*)y; p.ldy = ldy;
  if (M <= 8) return launch<1>(p, plan.c, plan.clusters, plan.smem, (cudaStream_t)stream);
  if (M <= 16) return launch<2>(p, plan.c, plan.clusters, plan.smem, (cudaStream_t)stream);
  return launch<4>(p, plan.c, plan.clusters, plan.smem, (cudaStream_t)stream);
}
