// All layers of a narrow decode step in one launch: RMSNorm, q/k/v, rotary embedding, cache append, attention, wo, RMSNorm,
// w1 and w3, SiLU product, w2, to the last layer's residual.  One CTA per SM stays for the whole step, in clusters of four (a
// cooperative launch: the clusters wait for one another).
//
// Why: a step of one branch as five launches a layer (q40_gemv_tiled.cu, attn_tree_fused.cu) takes 51.5 us a layer, of which the
// 107 MB of weights need 16.5 at HBM's rate: launches drain and fill, and HBM idles meanwhile.  Here a warp's weights come through
// a ring of its own that does not stop between matmuls (cp.async, 139 KB an SM: the first two passes of a matmul are there when its
// activations are), and matmuls hand over through L2 in words that carry their own step and layer, so that a consumer needs no flag, no
// fence and one trip.  Microseconds of a whole step with its lm_head, 512 + 64 keys: one branch 1075, 1655 as launches; a layer of one branch
// 31.4 and 51.5, of two 38 and 57.
//
// Matmul.  A cluster has whole 64-column groups and each of its CTAs a quarter of their k range; a CTA's share is cut into 16
// contiguous runs, one per warp.  Up to 128 k at a time (a pass), scale * x becomes integers of 22 bits with one exponent per branch, in three
// signed bytes that are three columns of the B operand of an int8 MMA; the A operand is the tiled word itself and its low nibbles, so that
// expanding eight weights costs one instruction (the fp16 fragments of q40_gemv_tiled.cu: seven).  Products and sums of a pass are exact.
// What scale * x loses is 2^-22 of the largest of 128 values, at most 2^-18 of their root mean square; one rounding to fp16, as in
// q40_gemv_tiled.cu, is 2^-12 of each (7B step: logits 0.0095 from 64 bits, 0.0100 by launches).  Sums over warps, then over the
// cluster (distributed shared memory, 16 of 64 columns finished by each CTA), in a fixed order: the same bits every time.
//
// Attention: a cluster per (branch, head), merged through distributed shared memory; keys and values are prefetched to L2 at the
// start of the layer.  The residual stream is kept by every CTA, which normalises for itself: no exchange of row statistics.
//
// What bounds it, per layer of one branch (us): matmuls 13.3 (a pass 1.05: a warp's own chain of staging, MMAs and copies; none of
// its parts alone is more than a fifth of it), of which 1.3 because 172 pairs of groups of w1 and w3 do not divide by 33 clusters; attention 3.7;
// exchanges, normalisation and the way through L2 9; waiting for the slowest cluster 5.  Tried without gain: later passes prefetched to
// L2, warps of a scheduler started one after the other, sums per CTA published to all (45 KB to be read by each CTA instead of 16: 65 us a layer).
//
// Words are written again one layer later.  That is safe because whoever writes has seen words that depend, through the
// matmuls between, on words of every CTA that read the old ones; it takes that each cluster has columns of every matmul.
#include <math_constants.h>

#include <algorithm>

#include "q40_common.cuh"

namespace q40 {
namespace chain {

constexpr int CL = 4;                             // CTAs of a cluster; each has a quarter of the k range of the cluster's columns
constexpr int WARPS = 16, THREADS = WARPS * 32;
constexpr int STEP = 2048 + 128;                  // one 16-row step of a span of the tiled stream
constexpr int PASS = 4;                           // a pass: up to four pairs of 16-row steps of a 64-column group, 128 k, with one exponent
constexpr int SLOT_W = PASS * 2 * 512, SLOT = SLOT_W + PASS * 2 * 32;       // a ring slot: a pass's weights and scales
constexpr int DEPTH = 2;                          // ring slots of a warp
constexpr int SEGS = 16;                          // column groups that a cluster has of one matmul, at most
constexpr int LIST = 28;                          // passes of a warp and layer, at most
constexpr int BF_LD = 72;                         // words of a pair's B fragments, padded to other banks
constexpr int KPB = 4;                            // prompt keys of a half warp per batch; and one of the suffix
constexpr int NR = 2;                             // fours of columns of the residual stream per thread and branch
constexpr uint32_t POLLS = 1u << 21;              // of one thread, before it gives up: about a second
constexpr uint32_t BAR_NS = 20000;
constexpr float MAGIC = 12582912.0f;              // 1.5 * 2^23
constexpr int MAGIC_BITS = 0x4B400000;

struct Layer {
  const uint8_t* w[7];                            // tiled copies: wq, wk, wv, wo, w1, w3, w2
  const __half* norm[2];
  const __half* pk;
  const __half* pv;
  int8_t* kq;
  __half* ks;
  int8_t* vq;
  __half* vs;
  const void* unused;
};

struct Params {
  const Layer* layers;
  int L, dim, hid, H, Hkv;
  int units[4], kpairs[4];                        // of q/k/v, wo, w1 and w3, w2: groups of 64 columns (w1 and w3: of both), 32-row pairs of a quarter
  const int64_t* tok;
  const __half* emb;
  int vocab;
  const int32_t* pos;
  const int32_t* plen;
  const __half* cos_tbl;
  const __half* sin_tbl;
  int n_pos, max_t, max_p;
  float eps;
  uint2* words[5];                                // what CTAs hand on, [branch][columns / 2] {two fp16 values, step and layer}: q/k/v, wo, SiLU product, w2, attention
  uint32_t* ctl;                                  // step number, CTAs that are through
  int* err;
  __half* h_out;
  float* ss_out;
  int xk;                                         // values of a branch's activations in shared memory
  int most[4], recv0[4];                          // segments of a cluster at most; where sums received of a matmul start (floats)
  int off_bf, off_xs, off_slab, off_recv, off_tab;
};

struct Seg { uint32_t off; uint16_t n; uint8_t mat, q; uint32_t k0, pad; };          // a warp's part of one group

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 ld_words(const uint2* a) {        // two words; each is one access
  uint64_t x, y;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(a) : "memory");
  return make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)y, (uint32_t)(y >> 32));
}
__device__ __forceinline__ void st_word(uint2* a, __half2 v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(a), "l"((uint64_t)h2_as_u32(v) | (uint64_t)tag << 32) : "memory");
}
// Four columns (nullptr: none) once they are of this step and layer; a bounded wait
template <int N>
__device__ __forceinline__ void poll(const uint2* const (&a)[N], uint2 (&v)[N], uint32_t tag, uint32_t& limit) {
  uint4 x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = a[i] ? ld_words(a[i]) : make_uint4(0, tag, 0, tag);
  for (;;) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && x[i].y == tag && x[i].w == tag;
    if (ok || !limit) break;
    --limit;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (x[i].y != tag || x[i].w != tag) x[i] = ld_words(a[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = make_uint2(x[i].x, x[i].z);
}
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, uint32_t& limit) {
  for (;;) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(BAR_NS) : "memory");
    if (ok || !limit) return;
    limit = limit > 32 ? limit - 32 : 0;
  }
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void push4(uint32_t dst, float4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar) : "memory");
}
__device__ __forceinline__ void push1(uint32_t dst, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MB>
__global__ void __launch_bounds__(THREADS, 1) decode_chain_kernel(const Params p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int cluster = blockIdx.x / CL, rank = blockIdx.x % CL, nclusters = gridDim.x / CL;
  const uint32_t ring = smem_u32(smem) + warp * (DEPTH * SLOT);
  const unsigned char* ring_g = smem + warp * (DEPTH * SLOT);
  uint32_t* bf = reinterpret_cast<uint32_t*>(smem + p.off_bf) + warp * (PASS * BF_LD);
  __half* xs = reinterpret_cast<__half*>(smem + p.off_xs);                    // [MB][xk] of this CTA's quarter of k
  float* slab = reinterpret_cast<float*>(smem + p.off_slab);                  // [warp][2][MB][64]
  constexpr int SLAB_LD = 2 * MB * 64 + 8;
  float* recv = reinterpret_cast<float*>(smem + p.off_recv);                  // of each matmul [source][segment][MB][16]; attention [2][source][36]
  float* recv_a = recv + p.recv0[3] + CL * p.most[3] * MB * 16;
  // tables
  Seg* segs = reinterpret_cast<Seg*>(smem + p.off_tab);                       // [4][WARPS][2]
  const uint8_t** wptr = reinterpret_cast<const uint8_t**>(segs + 4 * WARPS * 2);       // [L][7]
  uint2* list = reinterpret_cast<uint2*>(wptr + (p.L * 7 + 1) / 2 * 2);       // [WARPS][LIST] passes of a layer: offset, {matrix, pairs, group of the span}
  uint64_t* bars = reinterpret_cast<uint64_t*>(list + WARPS * LIST);               // [6]: exchanges of the four matmuls, two of attention
  int* s_seg = reinterpret_cast<int*>(bars + 6);                              // [4][SEGS]: warps that share a segment
  __half* s_qkv = reinterpret_cast<__half*>(s_seg + 4 * SEGS);                // [3][128] q, k, v of the item
  __half* s_rot = s_qkv + 3 * 128;                                            // [MB][2][64] cos, sin
  __half* s_h = s_rot + MB * 128;                                             // [MB][dim] residual stream
  float* s_red = reinterpret_cast<float*>(s_h + MB * p.dim);                  // [MB][WARPS]
  float* s_ml = s_red + MB * WARPS;                                           // [2][WARPS]
  int* s_u = reinterpret_cast<int*>(s_ml + 2 * WARPS);                        // [2][4]
  int* s_cnt = s_u + 8;                                                       // [WARPS] passes of a warp
  const uint32_t bar0 = smem_u32(bars);

  uint32_t limit = POLLS;
  // units of matmul ph of this cluster: [s_u[ph], s_u[4 + ph])
  if (tid < 8) s_u[tid] = p.units[tid & 3] * (cluster + (tid >> 2)) / nclusters;
  __syncthreads();
  // ---- tables ----
  for (int i = tid; i < p.L * 7; i += THREADS) wptr[i] = p.layers[i / 7].w[i % 7];
  if (tid == 0)
    for (int i = 0; i < 6; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i));
  if (tid < 4 * WARPS) {
    const int ph = tid / WARPS, w = tid % WARPS, G = p.kpairs[ph], mul = ph == 2 ? 2 : 1;
    const int u0 = s_u[ph] * mul, n = (s_u[4 + ph] * mul - u0) * G;
    int a = n * w / WARPS;
    const int b = n * (w + 1) / WARPS;
    Seg e[2] = {};
    for (int s = 0; s < 2 && a < b; ++s) {
      const int k = a % G, m = min(b - a, G - k), gi = u0 + a / G;
      int mat, idx = gi;
      if (ph == 0) {
        mat = 0;
        if (idx >= 2 * p.H) { idx -= 2 * p.H; mat = 1; if (idx >= 2 * p.Hkv) { idx -= 2 * p.Hkv; mat = 2; } }
      } else if (ph == 2) { mat = 4 + (gi & 1); idx = gi >> 1; }
      else mat = ph == 1 ? 3 : 6;
      e[s].off = (uint32_t)(((int64_t)(idx >> 2) * (2 * CL * G) + 2 * (rank * G + k)) * STEP);
      e[s].n = (uint16_t)m; e[s].mat = (uint8_t)mat; e[s].q = (uint8_t)(idx & 3);
      e[s].k0 = k * 32;
      a += m;
    }
    segs[(ph * WARPS + w) * 2] = e[0];
    segs[(ph * WARPS + w) * 2 + 1] = e[1];
  }
  if (tid < 4 * SEGS) {
    // segment s of matmul ph: the first and last warp with a part of it, and whether it is the first one's second segment
    const int ph = tid / SEGS, s = tid % SEGS, G = p.kpairs[ph], mul = ph == 2 ? 2 : 1;
    const int n = (s_u[4 + ph] - s_u[ph]) * mul * G;
    int w0 = 0, w1 = 0;
    if (s * G < n) {
      while (n * (w0 + 1) / WARPS <= s * G) ++w0;
      w1 = w0;
      while (w1 + 1 < WARPS && n * (w1 + 1) / WARPS < (s + 1) * G) ++w1;
    }
    s_seg[tid] = w0 | w1 << 8 | (n * w0 / WARPS < s * G ? 1 : 0) << 16;
  }
  if (tid < MB * 128) {
    const int m = tid >> 7, i = tid & 127;
    s_rot[tid] = (i < 64 ? p.cos_tbl : p.sin_tbl)[(int64_t)min(max(p.pos[m], 0), p.n_pos - 1) * 64 + (i & 63)];
  }
  const int plen = min(max(p.plen[0], 0), p.max_p);
  const uint32_t seq = *reinterpret_cast<volatile uint32_t*>(p.ctl);
  __syncthreads();
  if (tid < WARPS) {
    int n = 0;
    for (int i = 0; i < 8; ++i) {
      const Seg e = segs[((i >> 1) * WARPS + tid) * 2 + (i & 1)];
      for (int k = 0; k < e.n; k += PASS)
        list[tid * LIST + n++] = make_uint2(e.off + 2 * k * STEP, (uint32_t)min(PASS, e.n - k) | e.mat << 4 | e.q << 8);
    }
    s_cnt[tid] = n;
  }
  __syncthreads();
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  // ---- the warp's weight stream: all its pairs of all layers, through a ring that does not stop between matmuls ----
  const uint2* my_list = list + warp * LIST;
  const int my_n = s_cnt[warp];
  int i_layer = my_n ? 0 : p.L, i_at = 0;
  uint32_t i_dst = ring + lane * 16;
  const uint8_t* i_base = nullptr;
  int i_n = 0, i_q = 0;
  auto locate = [&]() {                                      // the next pass
    i_n = 0;
    if (i_layer < p.L) {
      const uint2 e = my_list[i_at];
      i_base = wptr[i_layer * 7 + (e.y >> 4 & 15)] + e.x;
      i_n = e.y & 15;
      i_q = e.y >> 8;
      if (++i_at == my_n) { i_at = 0; ++i_layer; }
    }
  };
  auto issue = [&]() {
    const uint8_t* w = i_base + i_q * 512 + lane * 16;
#pragma unroll
    for (int j = 0; j < PASS; ++j)
      if (j < i_n) {
        cp16(i_dst + j * 1024, w + j * 2 * STEP);
        cp16(i_dst + j * 1024 + 512, w + (j * 2 + 1) * STEP);
      }
    if (lane < 4 * i_n) cp16(i_dst + SLOT_W, i_base + 2048 + i_q * 32 + (lane >> 1) * STEP + (lane & 1) * 16);
    asm volatile("cp.async.commit_group;");
    i_dst ^= (ring + lane * 16) ^ (ring + lane * 16 + SLOT);
  };
#pragma unroll 1
  for (int i = 0; i < DEPTH; ++i) {
    locate();
    issue();
  }
  uint32_t c_off = 0;                                        // the slot of the next pass

  // ---- one matmul: the warp's pairs against xs, sums of 64 columns per segment to the slab ----
  auto matmul = [&](int ph) {
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      const Seg e = segs[(ph * WARPS + warp) * 2 + s];
      if (!e.n) break;
      float acc[8], eight[MB];                               // ... 8 times this lane's sum of scale * x
#pragma unroll
      for (int m = 0; m < MB; ++m) eight[m] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = 0.f;
      const __half* xk = xs + e.k0 + lane * 4;
#pragma unroll 1
      for (int left = e.n; left > 0; left -= PASS, xk += PASS * 32) {
        const int np = min(PASS, left);
        locate();
        asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
        __syncwarp();
        // scale * x of 128 k, four per lane, as 22-bit integers with one exponent per branch: three signed bytes, the columns 4 m + digit
        // of the B operand (bytes in the order k, k + 2, k + 1, k + 3 of the tiled words)
        float wgt = 0.f;
        {
          const int u = lane >> 2;
          const bool on = u < 2 * np;
          uint2 sc = make_uint2(0, 0);
          if (on) sc = *reinterpret_cast<const uint2*>(ring_g + c_off + SLOT_W + lane * 8);
          const float2 s01 = __half22float2(u32_as_h2(sc.x)), s23 = __half22float2(u32_as_h2(sc.y));
#pragma unroll
          for (int m = 0; m < MB; ++m) {
            uint2 xv = make_uint2(0, 0);
            if (on) xv = *reinterpret_cast<const uint2*>(xk + m * p.xk);
            const float2 x01 = __half22float2(u32_as_h2(xv.x)), x23 = __half22float2(u32_as_h2(xv.y));
            const float y0 = x01.x * s01.x, y1 = x01.y * s01.y, y2 = x23.x * s23.x, y3 = x23.y * s23.y;
            const uint32_t b = max(max(__float_as_uint(y0) & 0x7fffffffu, __float_as_uint(y1) & 0x7fffffffu),
                                   max(__float_as_uint(y2) & 0x7fffffffu, __float_as_uint(y3) & 0x7fffffffu));
            const uint32_t ex = max(__reduce_max_sync(0xffffffffu, b) >> 23, 26u);
            const float f = __uint_as_float((274u - ex) << 23);                 // |y| f < 2^21
            const float wm = ex == 255 ? CUDART_NAN_F : __uint_as_float((ex - 20u) << 23);     // 1 / f
            const uint32_t q0 = __float_as_uint(fmaf(y0, f, MAGIC + 32896.f)), q1 = __float_as_uint(fmaf(y1, f, MAGIC + 32896.f)),
                           q2 = __float_as_uint(fmaf(y2, f, MAGIC + 32896.f)), q3 = __float_as_uint(fmaf(y3, f, MAGIC + 32896.f));
            if (MB == 1 || m == (t >> 1)) wgt = wm;
            constexpr float C0 = MAGIC + 32896.f;
            eight[m] = fmaf(8.f * wm, ((__uint_as_float(q0) - C0) + (__uint_as_float(q1) - C0)) + ((__uint_as_float(q2) - C0) + (__uint_as_float(q3) - C0)), eight[m]);
            const uint32_t lo02 = prmt(q0, q2, 0x5140), lo13 = prmt(q1, q3, 0x5140);     // bytes 0 and 1 of two
            const uint32_t hi02 = prmt(q0, q2, 0x0062), hi13 = prmt(q1, q3, 0x0062);     // byte 2
            uint32_t* dst = bf + (u >> 1) * BF_LD + (m * 4) * 8 + t * 2 + (u & 1);
            dst[0] = prmt(lo02, lo13, 0x5410) ^ 0x80808080u;
            dst[8] = prmt(lo02, lo13, 0x7632) ^ 0x80808080u;
            dst[16] = (prmt(hi02, hi13, 0x5410) + 0x40404040u) ^ 0x80808080u;
          }
        }
        __syncwarp();
        int c[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) c[i][j] = MAGIC_BITS;
#pragma unroll
        for (int j = 0; j < PASS; ++j) {
          if (j < np) {
            const unsigned char* sp = ring_g + c_off + j * 1024 + lane * 16;
            const uint4 w0 = *reinterpret_cast<const uint4*>(sp), w1 = *reinterpret_cast<const uint4*>(sp + 512);
            const uint2 b = *reinterpret_cast<const uint2*>(bf + j * BF_LD + (MB == 1 ? (g & 3) : g) * 8 + t * 2);
            const uint32_t a[4] = {w0.x, w0.y, w0.z, w0.w}, a2[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
              imma(c[i], a[i], a[i] & 0x0F0F0F0Fu, a2[i], a2[i] & 0x0F0F0F0Fu, b.x, b.y);
          }
        }
        issue();
        c_off ^= SLOT;
        const float wa = (t & 1) ? wgt * 65536.f : wgt, wb = (t & 1) ? wgt * 0.f : wgt * 256.f;
        // a byte of a tiled word, as a signed number, is 16 code + (code' + 8), code' that of the column 8 further
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float c0 = __int_as_float(c[i][0]), c1 = __int_as_float(c[i][1]), c2 = __int_as_float(c[i][2]), c3 = __int_as_float(c[i][3]);
          acc[2 * i] = fmaf(c0 - c2, wa, fmaf(c1 - c3, wb, acc[2 * i]));
          acc[2 * i + 1] = fmaf(c2 - MAGIC, wa, fmaf(c3 - MAGIC, wb, acc[2 * i + 1]));
        }
      }
      float sub = warp_sum(eight[0]);
      if (MB == 2) {
        const float other = warp_sum(eight[MB - 1]);
        sub = t >> 1 ? other : sub;
      }
      if (t & 1) sub = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[i] = i & 1 ? acc[i] - sub : acc[i] * 0.0625f;
        const float v = acc[i] + __shfl_xor_sync(0xffffffffu, acc[i], 1);
        if (t == 0 || (MB == 2 && t == 2)) slab[warp * SLAB_LD + (s * MB + (t >> 1)) * 64 + 8 * i + g] = v;
      }
    }
  };
  // ---- the cluster's sums of a matmul: each CTA finishes 16 of a group's 64 columns and hands them on ----
  auto exchange = [&](int ph, uint32_t parity, uint32_t tag) {
    const int mul = ph == 2 ? 2 : 1, u0 = s_u[ph], nu = s_u[4 + ph] - u0, nseg = nu * mul;
    const uint32_t bar = bar0 + 8 * ph;
    float* rc = recv + p.recv0[ph];
    const int ld = p.most[ph] * MB * 16;                   // of a source
    if (tid == 0) bar_expect(bar, CL * nseg * MB * 64);
    if (tid < nseg * MB * 16) {
      const int j = tid & 15, s = (tid >> 4) / MB, m = (tid >> 4) % MB;
      const int e = s_seg[ph * SEGS + s], w1 = e >> 8 & 0xff;
      int w = e & 0xff;
      const float* src = slab + w * SLAB_LD + ((e >> 16) * MB + m) * 64 + 4 * j;
      float4 v = *reinterpret_cast<const float4*>(src);
      src = slab + w * SLAB_LD + m * 64 + 4 * j;
#pragma unroll 2
      for (; w < w1; ++w) {
        src += SLAB_LD;
        const float4 x = *reinterpret_cast<const float4*>(src);
        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
      }
      push4(mapa(smem_u32(rc + rank * ld + (s * MB + m) * 16 + (j & 3) * 4), j >> 2), v, mapa(bar, j >> 2));
    }
    if (tid < nu * MB * 8) {
      const int c2 = tid & 7, m = (tid >> 3) % MB, u = (tid >> 3) / MB;
      bar_wait(bar, parity, limit);
      const auto total = [&](int seg) {
        float2 x[CL];
#pragma unroll
        for (int r = 0; r < CL; ++r) x[r] = *reinterpret_cast<const float2*>(rc + r * ld + (seg * MB + m) * 16 + 2 * c2);
        return make_float2((x[0].x + x[1].x) + (x[2].x + x[3].x), (x[0].y + x[1].y) + (x[2].y + x[3].y));
      };
      const float2 v = total(u * mul);
      __half2 o = __floats2half2_rn(v.x, v.y);
      if (ph == 2) {
        const float2 a = __half22float2(o);
        const float2 v3 = total(u * mul + 1);
        o = __hmul2(__floats2half2_rn(a.x / (1.0f + expf(-a.x)), a.y / (1.0f + expf(-a.y))), __floats2half2_rn(v3.x, v3.y));
      }
      st_word(p.words[ph] + (m * p.units[ph] + u0 + u) * 32 + rank * 8 + c2, o, tag);
    }
  };

  // ---- residual stream: every CTA has all of it, columns 4 (tid + r THREADS) .. + 3 of each branch in this thread ----
  // h += sums of matmul `ph` (ph < 0: h is there); xs = RMSNorm(h) * w, this CTA's quarter.  `out`: the finished rows instead, for the
  // launch that multiplies them with the vocabulary
  auto norm_x = [&](int ph, const __half* w, uint32_t tag, bool out) {
    const int q0 = rank * (p.dim / CL);
    uint2 nw[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int c = 4 * (tid + r * THREADS);
      nw[r] = make_uint2(0, 0);
      if (!out && c >= q0 && c < q0 + p.dim / CL) nw[r] = __ldg(reinterpret_cast<const uint2*>(w + c));
    }
    float ss[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) ss[m] = 0.f;
    if (ph >= 0) {
      const uint2* a[MB * NR];
      uint2 v[MB * NR];
#pragma unroll
      for (int i = 0; i < MB * NR; ++i) {
        const int c = 4 * (tid + i % NR * THREADS);
        a[i] = c < p.dim ? p.words[ph] + (i / NR * p.dim + c) / 2 : nullptr;
      }
      poll(a, v, tag, limit);
#pragma unroll
      for (int i = 0; i < MB * NR; ++i) {
        const int c = 4 * (tid + i % NR * THREADS);
        if (c >= p.dim) continue;
        uint2* hp = reinterpret_cast<uint2*>(s_h + i / NR * p.dim + c);
        const uint2 x = *hp;
        *hp = make_uint2(h2_as_u32(__hadd2_rn(u32_as_h2(x.x), u32_as_h2(v[i].x))), h2_as_u32(__hadd2_rn(u32_as_h2(x.y), u32_as_h2(v[i].y))));
      }
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int c = 4 * (tid + r * THREADS);
        if (c >= p.dim) continue;
        const uint2 x = *reinterpret_cast<const uint2*>(s_h + m * p.dim + c);
        const float2 lo = __half22float2(u32_as_h2(x.x)), hi = __half22float2(u32_as_h2(x.y));
        ss[m] = fmaf(lo.x, lo.x, fmaf(lo.y, lo.y, fmaf(hi.x, hi.x, fmaf(hi.y, hi.y, ss[m]))));
      }
      ss[m] = warp_sum(ss[m]);
      if (lane == 0) s_red[m * WARPS + warp] = ss[m];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < WARPS; ++i) s += s_red[m * WARPS + i];
      if (out && blockIdx.x == 0 && tid == 0) p.ss_out[m] = s;
      const float inv = rsqrtf(s / (float)p.dim + p.eps);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int c = 4 * (tid + r * THREADS);
        const uint2* hp = reinterpret_cast<const uint2*>(s_h + m * p.dim + c);
        if (out) {
          if (blockIdx.x == 0 && c < p.dim) *reinterpret_cast<uint2*>(p.h_out + (int64_t)m * p.dim + c) = *hp;
        } else if (c >= q0 && c < q0 + p.dim / CL) {
          const float2 lo = __half22float2(u32_as_h2(hp->x)), hi = __half22float2(u32_as_h2(hp->y));
          uint2 v;
          v.x = h2_as_u32(__hmul2(__floats2half2_rn(lo.x * inv, lo.y * inv), u32_as_h2(nw[r].x)));
          v.y = h2_as_u32(__hmul2(__floats2half2_rn(hi.x * inv, hi.y * inv), u32_as_h2(nw[r].y)));
          *reinterpret_cast<uint2*>(xs + m * p.xk + c - q0) = v;
        }
      }
    }
    __syncthreads();
  };
  // xs = this CTA's quarter of what was handed on as words[src], `cols` columns a branch
  auto words_x = [&](int src, int cols, uint32_t tag) {
    const int n = cols / CL / 4;
#pragma unroll 1
    for (int i0 = tid; i0 < MB * n; i0 += 2 * THREADS) {
      const uint2* a[2];
      uint2 v[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + r * THREADS, m = MB == 1 ? 0 : i / n;
        a[r] = i < MB * n ? p.words[src] + (m * cols + rank * (cols / CL)) / 2 + 2 * (i - m * n) : nullptr;
      }
      poll(a, v, tag, limit);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + r * THREADS, m = MB == 1 ? 0 : i / n;
        if (i < MB * n) *reinterpret_cast<uint2*>(xs + m * p.xk + 4 * (i - m * n)) = v[r];
      }
    }
    __syncthreads();
  };

  // embedding rows (ids are clamped)
#pragma unroll
  for (int m = 0; m < MB; ++m) {
    const int64_t id = p.tok[m];
    const __half* e = p.emb + (id < 0 ? 0 : (id >= p.vocab ? p.vocab - 1 : id)) * p.dim;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int c = 4 * (tid + r * THREADS);
      uint2 v = make_uint2(0, 0);
      if (c < p.dim) v = __ldg(reinterpret_cast<const uint2*>(e + c));
      if (c < p.dim) *reinterpret_cast<uint2*>(s_h + m * p.dim + c) = v;
    }
  }

  // ---- attention: a cluster per (branch, head), its keys round-robin over CTAs and half warps; 8 of the 128 dims per lane ----
  const int hw = warp * 2 + (lane >> 4), sl = lane & 15;
  // eight values of the keys and values of a batch: of the prompt, and of one suffix row its codes, and both scales in z
  uint4 kk[KPB], vv[KPB], ks, vs;
  auto load_keys = [&](const Layer& ly, int ab, int hk, int slen, int batch) {
    const __half* pk = ly.pk + hk * 128 + sl * 8;
    const __half* pv = ly.pv + hk * 128 + sl * 8;
#pragma unroll
    for (int i = 0; i < KPB; ++i) {
      const int key = ((batch * KPB + i) * 2 * WARPS + hw) * CL + rank;
      kk[i] = vv[i] = make_uint4(0, 0, 0, 0);
      if (key < plen) {
        const int64_t off = (int64_t)key * (p.Hkv * 128);
        kk[i] = __ldg(reinterpret_cast<const uint4*>(pk + off));
        vv[i] = __ldg(reinterpret_cast<const uint4*>(pv + off));
      }
    }
    const int j = (batch * 2 * WARPS + hw) * CL + rank;
    ks = vs = make_uint4(0, 0, 0, 0);
    if (j < slen) {
      const int64_t row = ((int64_t)ab * p.max_t + j) * p.Hkv + hk;
      const uint2 a = __ldg(reinterpret_cast<const uint2*>(ly.kq + row * 64 + 8 * (sl & 7)));
      const uint2 b = __ldg(reinterpret_cast<const uint2*>(ly.vq + row * 64 + 8 * (sl & 7)));
      ks.x = a.x; ks.y = a.y; vs.x = b.x; vs.y = b.y;
      ks.z = (uint32_t)__half_as_ushort(__ldg(ly.ks + row * 2 + (sl >> 3)));
      vs.z = (uint32_t)__half_as_ushort(__ldg(ly.vs + row * 2 + (sl >> 3)));
    }
  };
  // ... on their way to L2 long before
  auto prefetch_keys = [&](const Layer& ly) {
    if (sl >= 4) return;
#pragma unroll 1
    for (int it = cluster; it < MB * p.H; it += nclusters) {
      const int ab = MB == 1 ? 0 : it / p.H, hk = (it - ab * p.H) / (p.H / p.Hkv);
      const int slen = min(max(min(max(p.pos[ab], 0), p.n_pos - 1) - plen, 0), p.max_t);
      const __half* pp = (sl & 2 ? ly.pv : ly.pk) + hk * 128 + (sl & 1) * 64;
#pragma unroll 1
      for (int key = hw * CL + rank; key < plen; key += 2 * WARPS * CL) asm volatile("prefetch.global.L2 [%0];" ::"l"(pp + (int64_t)key * (p.Hkv * 128)));
#pragma unroll 1
      for (int j = hw * CL + rank; j < slen; j += 2 * WARPS * CL) {
        const int64_t row = ((int64_t)ab * p.max_t + j) * p.Hkv + hk;
        const void* a = sl & 2 ? (const void*)((sl & 1 ? ly.vs : ly.ks) + row * 2) : (const void*)((sl & 1 ? ly.vq : ly.kq) + row * 64);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
      }
    }
  };
  auto expand = [&](uint4& r) {                        // eight codes (high nibbles: dims 0..63) times the scale
    const __half2 sc = __half2half2(__ushort_as_half((unsigned short)r.z));
    const int sh = sl >> 3 ? 0 : 4;
    const uint32_t c0 = r.x >> sh, c1 = r.y >> sh;
    const uint32_t e0 = h2_as_u32(__hmul2(codes_lo_to_h2(c0), sc)), o0 = h2_as_u32(__hmul2(codes_lo_to_h2(c0 >> 8), sc));      // dims 0, 2 and 1, 3
    const uint32_t e1 = h2_as_u32(__hmul2(codes_lo_to_h2(c1), sc)), o1 = h2_as_u32(__hmul2(codes_lo_to_h2(c1 >> 8), sc));
    r = make_uint4(prmt(e0, o0, 0x5410), prmt(e0, o0, 0x7632), prmt(e1, o1, 0x5410), prmt(e1, o1, 0x7632));
  };
  float* am = slab;                                    // [WARPS][132]: 128 dims of each warp
  uint32_t a_turn = 0;                                 // attention exchanges so far
  auto attention = [&](const Layer& ly, uint32_t tag) {
#pragma unroll 1
    for (int it = cluster; it < MB * p.H; it += nclusters, ++a_turn) {
      const int ab = MB == 1 ? 0 : it / p.H, hq = it - ab * p.H, hk = hq / (p.H / p.Hkv);
      const int apos = min(max(p.pos[ab], 0), p.n_pos - 1);
      const int slen = min(max(apos - plen, 0), p.max_t);
      const bool has_new = slen % CL == rank;             // this CTA takes the new token's key, suffix row slen
      const uint32_t bar = bar0 + 8 * (4 + (a_turn & 1));
      float* rc = recv_a + (a_turn & 1) * CL * 36;
      float qf[8], mx = -CUDART_INF_F, l = 0.f, o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = 0.f;
      const auto dot = [&](const uint4& x) {
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
        float s = 0.f;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const float2 f = __half22float2(u32_as_h2(w[d]));
          s = fmaf(qf[2 * d], f.x, s);
          s = fmaf(qf[2 * d + 1], f.y, s);
        }
        return s;
      };
      const auto add = [&](const uint4& x, float pw) {
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
        l += pw;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const float2 f = __half22float2(u32_as_h2(w[d]));
          o[2 * d] = fmaf(pw, f.x, o[2 * d]);
          o[2 * d + 1] = fmaf(pw, f.y, o[2 * d + 1]);
        }
      };
#pragma unroll 1
      for (int batch = 0; batch * KPB * 2 * WARPS * CL < plen || batch * 2 * WARPS * CL <= slen; ++batch) {
        load_keys(ly, ab, hk, slen, batch);
        if (batch == 0) {
          if (warp < (has_new ? 3 : 1)) {
            // q, k or v of the new token
            const int col = (warp == 0 ? hq : (warp == 1 ? p.H + hk : p.H + p.Hkv + hk)) * 128 + 4 * lane;
            const uint2* a[1] = {p.words[0] + (ab * (p.H + 2 * p.Hkv) * 128 + col) / 2};
            uint2 v[1];
            poll(a, v, tag, limit);
            uint2 x = v[0];
            if (warp < 2) {                                   // rotary embedding: dim d turns with dim d +- 64
              const uint2 o = make_uint2(__shfl_xor_sync(0xffffffffu, x.x, 16), __shfl_xor_sync(0xffffffffu, x.y, 16));
              const __half2* cs = reinterpret_cast<const __half2*>(s_rot + ab * 128 + 4 * (lane & 15));
              const __half2 p0 = lane < 16 ? __hneg2(u32_as_h2(o.x)) : u32_as_h2(o.x), p1 = lane < 16 ? __hneg2(u32_as_h2(o.y)) : u32_as_h2(o.y);
              x.x = h2_as_u32(__hadd2_rn(__hmul2_rn(u32_as_h2(x.x), cs[0]), __hmul2_rn(p0, cs[32])));
              x.y = h2_as_u32(__hadd2_rn(__hmul2_rn(u32_as_h2(x.y), cs[1]), __hmul2_rn(p1, cs[33])));
            }
            *reinterpret_cast<uint2*>(s_qkv + warp * 128 + 4 * lane) = x;
          }
          if (tid == 0) bar_expect(bar, CL * (32 * 4 + 8));
          __syncthreads();
          const float scale_log2 = (1.0f / sqrtf(128.0f)) * 1.4426950408889634f;
#pragma unroll
          for (int i = 0; i < 8; ++i) qf[i] = __half2float(s_qkv[sl * 8 + i]) * scale_log2;
        }
        const int j = (batch * 2 * WARPS + hw) * CL + rank;
        if (batch * 2 * WARPS * CL <= slen) {
          expand(ks);
          expand(vs);
          if (j == slen) {
            ks = *reinterpret_cast<const uint4*>(s_qkv + 128 + sl * 8);
            vs = *reinterpret_cast<const uint4*>(s_qkv + 256 + sl * 8);
          }
        }
        float sd[KPB + 1], mn = mx;
#pragma unroll
        for (int i = 0; i < KPB; ++i) sd[i] = dot(kk[i]);
        sd[KPB] = dot(ks);
#pragma unroll
        for (int x = 1; x < 16; x <<= 1)
#pragma unroll
          for (int i = 0; i <= KPB; ++i) sd[i] += __shfl_xor_sync(0xffffffffu, sd[i], x);
#pragma unroll
        for (int i = 0; i <= KPB; ++i) {
          if (i < KPB ? ((batch * KPB + i) * 2 * WARPS + hw) * CL + rank >= plen : j > slen) sd[i] = -CUDART_INF_F;
          mn = fmaxf(mn, sd[i]);
        }
        if (mn > -CUDART_INF_F) {
          const float corr = mx > -CUDART_INF_F ? exp2f(mx - mn) : 0.f;
          l *= corr;
#pragma unroll
          for (int d = 0; d < 8; ++d) o[d] *= corr;
#pragma unroll
          for (int i = 0; i < KPB; ++i) add(vv[i], exp2f(sd[i] - mn));
          add(vs, exp2f(sd[KPB] - mn));
          mx = mn;
        }
      }
      // the two half warps, then the warps
      {
        const float m2 = __shfl_xor_sync(0xffffffffu, mx, 16), l2 = __shfl_xor_sync(0xffffffffu, l, 16);
        const float M = fmaxf(mx, m2);
        const float w1 = mx > -CUDART_INF_F ? exp2f(mx - M) : 0.f, w2 = m2 > -CUDART_INF_F ? exp2f(m2 - M) : 0.f;
#pragma unroll
        for (int d = 0; d < 8; ++d) o[d] = o[d] * w1 + __shfl_xor_sync(0xffffffffu, o[d], 16) * w2;
        l = l * w1 + l2 * w2;
        mx = M;
      }
      if (lane < 16) {
        *reinterpret_cast<float4*>(am + warp * 132 + lane * 8) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4*>(am + warp * 132 + lane * 8 + 4) = make_float4(o[4], o[5], o[6], o[7]);
      }
      if (lane == 0) { s_ml[warp] = mx; s_ml[WARPS + warp] = l; }
      __syncthreads();
      if (warp < 4) {
        // dim tid of the CTA's keys to the CTA that finishes it
        const float mw = lane < WARPS ? s_ml[lane] : -CUDART_INF_F, M = warp_max(mw);
        const float wl = mw > -CUDART_INF_F ? exp2f(mw - M) : 0.f, L = warp_sum(lane < WARPS ? s_ml[WARPS + lane] * wl : 0.f);
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) v = fmaf(am[w * 132 + tid], __shfl_sync(0xffffffffu, wl, w), v);
        const uint32_t rbar = mapa(bar, warp), dst = mapa(smem_u32(rc + rank * 36), warp);
        push1(dst + lane * 4, v, rbar);
        if (lane < 2) push1(dst + 128 + lane * 4, lane ? L : M, rbar);
        if (warp == 0) {
          bar_wait(bar, a_turn >> 1 & 1, limit);
          if (lane < 16) {
            float Mx = -CUDART_INF_F, Ls = 0.f, a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int r = 0; r < CL; ++r) Mx = fmaxf(Mx, rc[r * 36 + 32]);
#pragma unroll
            for (int r = 0; r < CL; ++r) {
              const float pm = rc[r * 36 + 32], wt = pm > -CUDART_INF_F ? exp2f(pm - Mx) : 0.f;
              Ls = fmaf(rc[r * 36 + 33], wt, Ls);
              a0 = fmaf(rc[r * 36 + 2 * lane], wt, a0);
              a1 = fmaf(rc[r * 36 + 2 * lane + 1], wt, a1);
            }
            const __half2 x = Ls > 0.f ? __floats2half2_rn(a0 / Ls, a1 / Ls) : __floats2half2_rn(0.f, 0.f);
            st_word(p.words[4] + it * 64 + rank * 16 + lane, x, tag);
          }
        }
      }
      // Q4_0 append of the rotated key (warp 1) and the value (warp 2): four dims per lane, byte d = code(d) << 4 | code(d + 64)
      if (has_new && (warp == 1 || warp == 2) && hq % (p.H / p.Hkv) == 0 && apos - plen >= 0 && apos - plen < p.max_t) {
        const uint2 x = *reinterpret_cast<const uint2*>(s_qkv + warp * 128 + 4 * lane);
        const float2 lo = __half22float2(u32_as_h2(x.x)), hi = __half22float2(u32_as_h2(x.y));
        const float f[4] = {lo.x, lo.y, hi.x, hi.y};
        float mxv = fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fmaxf(fabsf(f[2]), fabsf(f[3])));
#pragma unroll
        for (int i = 1; i < 16; i <<= 1) mxv = fmaxf(mxv, __shfl_xor_sync(0xffffffffu, mxv, i));
        const __half sc = __float2half_rn(__fdiv_rn(mxv, 7.0f));
        const float fs = __half2float(sc);
        uint32_t code = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float q = rintf(__half2float(__float2half_rn(__fdiv_rn(f[i], fs))));
          code |= (uint32_t)((fabsf(q) <= 65504.0f ? (int)q : 0) & 0xF) << (8 * i);
        }
        const uint32_t other = __shfl_xor_sync(0xffffffffu, code, 16);
        const int64_t row = ((int64_t)ab * p.max_t + (apos - plen)) * p.Hkv + hk;
        int8_t* dst = warp == 1 ? ly.kq : ly.vq;
        __half* dsc = warp == 1 ? ly.ks : ly.vs;
        if (lane < 16) reinterpret_cast<uint32_t*>(dst + row * 64)[lane] = code << 4 | other;
        if ((lane & 15) == 0) dsc[row * 2 + (lane >> 4)] = sc;
      }
      __syncthreads();                                 // s_qkv, slab and s_ml may be written again
    }
  };

#pragma unroll 1
  for (int layer = 0; layer <= p.L; ++layer) {
    const Layer& ly = p.layers[min(layer, p.L - 1)];
    const uint32_t tag = seq * (uint32_t)p.L + layer + 1;
#pragma unroll 1
    for (int ph = 0; ph < 4; ++ph) {
      const bool last = layer == p.L;
      if (ph == 0 && !last) prefetch_keys(ly);
      if (ph & 1) words_x(ph == 1 ? 4 : 2, ph == 1 ? p.H * 128 : p.hid, tag);
      else norm_x(ph == 0 ? (layer ? 3 : -1) : 1, ly.norm[ph >> 1], ph == 0 ? tag - 1 : tag, last);
      if (last) break;
      matmul(ph);
      __syncthreads();
      exchange(ph, layer & 1, tag);
      if (ph == 0) attention(ly, tag);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (limit == 0) q40_set_error(p.err);
  __syncthreads();
  if (tid == 0 && atomicAdd(p.ctl + 1, 1u) == gridDim.x - 1) {
    p.ctl[1] = 0;
    p.ctl[0] = seq + 1;
  }
  // nobody leaves while sums for it may be on their way
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

using Kernel = void (*)(const Params);

struct Plan { size_t smem, ws; int64_t word0[5]; int clusters; };

static int plan(Params& p, int B, int clusters, Plan& pl) {
  p.units[0] = 2 * (p.H + 2 * p.Hkv); p.kpairs[0] = p.dim / 32 / CL;
  p.units[1] = p.dim / 64;            p.kpairs[1] = p.H * 4 / CL;
  p.units[2] = p.hid / 64;            p.kpairs[2] = p.dim / 32 / CL;
  p.units[3] = p.dim / 64;            p.kpairs[3] = p.hid / 32 / CL;
  pl.clusters = clusters;
  int passes = 0;
  for (int i = 0; i < 4; ++i) {
    // a cluster has work in every matmul (see the note on words that are written again), and so has each of its warps (the sums over warps
    // take every slab between a segment's first and last); its segments fit, a warp has two at most
    const int mul = i == 2 ? 2 : 1, most = (p.units[i] + clusters - 1) / clusters * mul;
    if (p.units[i] / clusters * mul * p.kpairs[i] < WARPS || most > SEGS || most * B * 16 > THREADS || (most * p.kpairs[i] + WARPS - 1) / WARPS > p.kpairs[i]) return Q40_E_UNSUPPORTED;
    p.most[i] = most;
    passes += ((most * p.kpairs[i] + WARPS - 1) / WARPS + PASS - 1) / PASS + 1;      // a warp's share of two segments
    p.recv0[i] = i ? p.recv0[i - 1] + CL * p.most[i - 1] * B * 16 : 0;
  }
  if (passes > LIST || p.dim > 4 * NR * THREADS) return Q40_E_UNSUPPORTED;
  p.xk = std::max(std::max(p.dim, p.hid), p.H * 128) / CL;
  size_t off = (size_t)WARPS * DEPTH * SLOT;
  p.off_bf = (int)off; off += (size_t)WARPS * PASS * BF_LD * 4;
  p.off_xs = (int)off; off += (size_t)B * p.xk * 2;
  p.off_slab = (int)off; off += (size_t)WARPS * (2 * B * 64 + 8) * 4;
  p.off_recv = (int)off; off += (size_t)(p.recv0[3] + CL * p.most[3] * B * 16 + 2 * CL * 36) * 4;
  p.off_tab = (int)off;
  off += 4 * WARPS * 2 * sizeof(Seg) + (size_t)((p.L * 7 + 1) / 2 * 2) * 8 + 6 * 8 + 4 * SEGS * 4 + 3 * 128 * 2 + B * 128 * 2 + (size_t)B * p.dim * 2 + B * WARPS * 4 + 2 * WARPS * 4 + 8 * 4 + WARPS * 4 + WARPS * LIST * 8;
  pl.smem = off;
  const int cols[5] = {(p.H + 2 * p.Hkv) * 128, p.dim, p.hid, p.dim, p.H * 128};
  int64_t n = 16;                                    // the step counter's place
  for (int i = 0; i < 5; ++i) { pl.word0[i] = n; n += (int64_t)B * cols[i] / 2; }
  pl.ws = (size_t)n * 8;
  return Q40_OK;
}

// Clusters that run at once on the current device (an answer is kept per device)
static int max_clusters(Kernel kern) {
  static std::atomic<int> cache[16];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* kept = dev < 16 ? &cache[dev] : nullptr;
  if (kept && kept->load(std::memory_order_relaxed)) return kept->load(std::memory_order_relaxed) - 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(CL * 64, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = 227 * 1024;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0, coop = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  if (kept) kept->store(n + 1, std::memory_order_relaxed);
  return n;
}

static Kernel chain_kernel(int B) {
  static std::atomic<uint64_t> ready[2];
  Kernel k = B == 1 ? decode_chain_kernel<1> : decode_chain_kernel<2>;
  if (q40_allow_smem(ready[B - 1], (const void*)k, 227 * 1024) == cudaSuccess) return k;
  (void)cudaGetLastError();
  return nullptr;
}

static Kernel prepare(Params& p, int B, int L, int dim, int hid, int H, int Hkv, Plan& pl) {
  if (B < 1 || B > 2 || L < 1 || L > 256 || H < 1 || Hkv < 1 || H % Hkv || dim < 256 || dim > 65536 || dim % 256 || hid < 256 || hid > 65536 ||
      hid % 256 || H > 512 || H % 2 || Hkv % 2)
    return nullptr;
  Kernel k = chain_kernel(B);
  if (!k) return nullptr;
  p.L = L; p.dim = dim; p.hid = hid; p.H = H; p.Hkv = Hkv;
  const int n = max_clusters(k);
  if (n < 1 || plan(p, B, n, pl) != Q40_OK || pl.smem > 227 * 1024) return nullptr;
  return k;
}

}  // namespace chain
}  // namespace q40

// Bytes of workspace of q40_decode_chain, zeroed before its first call; 0: not available for these sizes or on this device
extern "C" size_t q40_decode_chain_ws_bytes(int B, int L, int dim, int hid, int H, int Hkv) {
  using namespace q40::chain;
  Params p{};
  Plan pl;
  return prepare(p, B, L, dim, hid, H, Hkv, pl) ? pl.ws : 0;
}

extern "C" int q40_decode_chain(const void* layers, int L, int B, int dim, int hid, int H, int Hkv, const int64_t* tok,
                                const void* emb, int vocab, const int32_t* pos, const int32_t* prefix_len, const void* cos_tbl,
                                const void* sin_tbl, int n_pos, int max_t, int max_p, float eps, void* h_out, float* ss_out,
                                void* workspace, size_t workspace_bytes, int* err, void* stream) {
  using namespace q40::chain;
  if (!layers || !tok || !emb || !pos || !prefix_len || !cos_tbl || !sin_tbl || !h_out || !ss_out || !workspace || !err) return Q40_E_NULL;
  if (vocab < 1 || n_pos < 1 || max_t < 1 || max_p < 1) return Q40_E_SHAPE;
  Params p{};
  Plan pl;
  Kernel kern = prepare(p, B, L, dim, hid, H, Hkv, pl);
  if (!kern) return Q40_E_UNSUPPORTED;
  if (workspace_bytes < pl.ws) return Q40_E_WORKSPACE;
  if (!q40_aligned(workspace, 16) || !q40_aligned(layers, 8) || !q40_aligned(emb, 8) || !q40_aligned(h_out, 8)) return Q40_E_ALIGN;
  p.layers = (const Layer*)layers;
  p.tok = tok; p.emb = (const __half*)emb; p.vocab = vocab; p.pos = pos; p.plen = prefix_len;
  p.cos_tbl = (const __half*)cos_tbl; p.sin_tbl = (const __half*)sin_tbl; p.n_pos = n_pos; p.max_t = max_t; p.max_p = max_p;
  p.eps = eps; p.err = err; p.h_out = (__half*)h_out; p.ss_out = ss_out;
  p.ctl = (uint32_t*)workspace;
  for (int i = 0; i < 5; ++i) p.words[i] = (uint2*)workspace + pl.word0[i];
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(CL * pl.clusters, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
  if (e == cudaErrorCooperativeLaunchTooLarge) {              // a part of the SMs is not this context's
    (void)cudaGetLastError();
    return Q40_E_UNSUPPORTED;
  }
  return e == cudaSuccess ? Q40_OK : (int)e;
}
