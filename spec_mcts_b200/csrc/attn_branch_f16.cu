// Decode attention for one query token per branch over that branch's own fp16 keys, on matrix instructions: a contiguous [B,Hkv,L,D] cache or a paged
// pool.  A row is a branch and up to four query heads of one kv head, whose keys and values are read once for all of them; one to eight warps
// share a row.  The end of a row may fold in partial results of a shared-prefix pass (attn_prefix.cu).
//
// What bounds it: few rows, a warp's chain of 0.7 us per 16 keys; many, the keys' and values' way from memory (100 branches of 300 keys,
// contiguous: 71.4 us, 6.9 TB/s).  A warp takes 16 keys at a time through a ring of its own (cp.async, 8 KB a stage), which is filled while it
// computes.  A tile that does not start on 128 bytes costs a fifth (10 paged branches of 512 keys 13.6 us, 11.5).
//   scores   A = 16 keys (ldmatrix), B = the queries: columns 2i and 2i + 1 are head i's (of two heads, 4i .. 4i + 3; of one, all)
//   output   A = 16 values transposed (ldmatrix.trans), B = the weights: a head's two columns hold the two parts of weight_parts
// Lane (g, t) has the scores of keys g and g + 8 for head t, that head's maximum and sum, and its dims g and g + 8 of every 16.
//
// Stands in for flash_attn_kernel2 / page_flash_attn_kernel2 of the reference
// (triton_kernels.py:559-647, 700-789), with fp32 softmax state and exact masking of the
// tail instead of the reference's fp16 state and multiple-of-32 length requirement.
#include "attn_tile.cuh"

namespace q40 {

constexpr int F16_KEYS = 16;                    // of a stage
constexpr int F16_TILE = F16_KEYS * TILE_ROW_BYTES;
constexpr int Q_ROW = TILE_ROW_BYTES + 16;      // of the queries behind it, so that four heads lie in different banks

template <int WPR>
struct F16Shape { static constexpr int NW = WPR == 8 ? 8 : 4; };
template <int S, int G>
constexpr int f16_warp_bytes = (S * 2 * F16_TILE + G * Q_ROW + 127) / 128 * 128;

template <int MODE, int WPR, int S, int G>             // MODE: see key_slot
__global__ void __launch_bounds__(F16Shape<WPR>::NW * 32, F16Shape<WPR>::NW == 8 ? 1 : S == 3 ? 2 : 3)
attn_branch_f16_kernel(const BranchArgs a) {
  constexpr int D = ATTN_D, NW = F16Shape<WPR>::NW, RT = WPR * 32;       // RT: threads of a row
  constexpr int GL = G == 4 ? 0 : G == 2 ? 1 : 2;                         // lane t works for head t >> GL
  asm volatile("griddepcontrol.launch_dependents;");
  // nothing of the previous launch is read before it is done: see attn_branch_kernel
  if (!a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, mi = lane >> 3;
  const int slot = warp / WPR, part = warp % WPR;           // row of this CTA, warp of the row
  const int64_t row = (int64_t)blockIdx.x * (NW / WPR) + slot;
  const int HG = a.H / G;                        // rows of a branch
  if (row >= a.rows / G) return;                 // whole rows, which meet at no common barrier
  const int b = (int)(row / HG), h = (int)(row % HG) * G, hk = h / (a.H / a.Hkv);

  extern __shared__ __align__(128) unsigned char rings[];
  unsigned char* const mine = rings + warp * f16_warp_bytes<S, G>;
  const uint32_t ring = smem_u32(mine), queries = ring + S * 2 * F16_TILE;
#pragma unroll
  for (int i = lane; i < 16 * G; i += 32)
    cp_async16(queries + (i >> 4) * Q_ROW + 16 * (i & 15), a.q + (int64_t)b * a.q_stride + (h + (i >> 4)) * D + 8 * (i & 15), true);

  // (entries of the table beyond the length need not exist)
  const int len = a.seq_lens ? min(max(a.seq_lens[b], 0), a.L) : a.L;
  const void* const table = MODE == 1 ? (const void*)(reinterpret_cast<const int16_t*>(a.tbl) + (int64_t)b * a.tbl_stride)
                                      : (const void*)(reinterpret_cast<const int32_t*>(a.tbl) + (int64_t)b * a.tbl_stride);
  const int64_t kv0 = (MODE == 0 ? (int64_t)(b * a.Hkv + hk) * a.L : (int64_t)hk * a.P) * D + (lane & 15) * 8;
  const __half *kbase = a.k + kv0, *vbase = a.v + kv0;
  constexpr int STEP = WPR * F16_KEYS;
  // slots of the 16 keys from t0 in lanes 0 to 15 and again in 16 to 31, looked up one request ahead
  const auto slots_of = [&](int t0) { const int k = t0 + (lane & 15); return k < len ? key_slot<MODE>(a, table, k) : 0; };
  // Half a warp copies a key; keys beyond the length become zeros
  const auto request = [&](int t0, int stage, int slots) {
    const uint32_t kt = ring + stage * 2 * F16_TILE;
#pragma unroll
    for (int j = 0; j < F16_KEYS / 2; ++j) {
      const int r = 2 * j + (lane >> 4);
      const bool ok = t0 + r < len;
      const int64_t off = (int64_t)(MODE == 0 ? (ok ? t0 + r : 0) : __shfl_sync(0xffffffffu, slots, r)) * D;
      cp_async16(kt + tile_off(r, lane & 15), kbase + off, ok);
      cp_async16(kt + F16_TILE + tile_off(r, lane & 15), vbase + off, ok);
    }
  };
  int slots = MODE == 0 ? 0 : slots_of(part * F16_KEYS);
#pragma unroll
  for (int i = 0; i < S; ++i) {
    const int t0 = part * F16_KEYS + i * STEP;
    if (t0 < len) request(t0, i, slots);
    cp_async_commit();
    if (MODE != 0) slots = slots_of(t0 + STEP);
  }
  cp_async_wait<S - 1>();
  __syncwarp();

  uint32_t qb[8][2];                             // B fragments of the queries
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(qb[ks][r]) : "r"(queries + ((g >> 1) >> GL) * Q_ROW + 32 * ks + 16 * r + 4 * t));
  float m = -CUDART_INF_F, l = 0.f;              // m: WEIGHT_BITS below the largest score; l: of this lane's keys
  float acc[8][4];                               // dims 16i + g (columns: both parts of the weights) and 16i + 8 + g
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  int stage = 0;
#pragma unroll 1
  for (int t0 = part * F16_KEYS; t0 < len; t0 += STEP) {
    cp_async_wait<S - 1>();
    __syncwarp();
    const uint32_t kt = ring + stage * 2 * F16_TILE, vt = kt + F16_TILE;
    float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < 8; ks += 2) {
      uint32_t x[4], y[4];
      const int r = (lane & 7) + (mi & 1) * 8;
      ldsm_x4(kt + tile_off(r, 2 * ks + (mi >> 1)), x[0], x[1], x[2], x[3]);
      ldsm_x4(kt + tile_off(r, 2 * ks + 2 + (mi >> 1)), y[0], y[1], y[2], y[3]);
      mma_f16(c0, x[0], x[1], x[2], x[3], qb[ks][0], qb[ks][1]);
      mma_f16(c1, y[0], y[1], y[2], y[3], qb[ks + 1][0], qb[ks + 1][1]);
    }
    float s[2], mnew = m;                        // a head's columns are alike
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      s[r] = t0 + 8 * r + g < len ? (c0[2 * r] + c1[2 * r]) * a.scale_log2 : -CUDART_INF_F;
      mnew = fmaxf(mnew, s[r] - WEIGHT_BITS);
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) mnew = fmaxf(mnew, __shfl_xor_sync(0xffffffffu, mnew, o));
    if (mnew != m) {
      const float corr = ex2(m - mnew);
      l *= corr;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= corr;
      m = mnew;
    }
    __syncwarp();                                // heads differ in whether theirs has moved
    uint32_t pk[2];                              // of keys g and g + 8
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float p = ex2(s[r] - m);
      l += p;
      pk[r] = weight_parts(p);
    }
    // column g's weights of keys 2t, 2t + 1, 2t + 8 and 2t + 9
    const auto of_key = [&](int r) { return __shfl_sync(0xffffffffu, pk[r >> 1], 8 * t + 4 * (r & 1) + (g >> 1)); };
    const uint32_t sel = g & 1 ? 0x7632u : 0x5410u;                       // odd columns: the rest
    const uint32_t x0 = of_key(0), x1 = of_key(1), x2 = of_key(2), x3 = of_key(3);
    const uint32_t b0 = prmt(x0, x1, sel), b1 = prmt(x2, x3, sel);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t v[4];
      ldsm_x4_t(vt + tile_off((lane & 7) + (mi >> 1) * 8, 2 * i + (mi & 1)), v[0], v[1], v[2], v[3]);
      mma_f16(acc[i], v[0], v[1], v[2], v[3], b0, b1);
    }
    __syncwarp();
    if (t0 + S * STEP < len) request(t0 + S * STEP, stage, slots);
    cp_async_commit();
    if (MODE != 0) slots = slots_of(t0 + (S + 1) * STEP);
    if (++stage == S) stage = 0;
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);

  // the ring, which is empty, takes the warp's outputs
  __shared__ float sm_m[G][NW], sm_l[G][NW];
  constexpr int O_STRIDE = f16_warp_bytes<S, G> / 4;
  float* const out = reinterpret_cast<float*>(mine);
  __syncwarp();
  if (lane < 4 && (lane & ((1 << GL) - 1)) == 0) { sm_m[t >> GL][warp] = m; sm_l[t >> GL][warp] = l; }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (GL == 0 || (i & ((1 << GL) - 1)) == (t & ((1 << GL) - 1))) {
      out[(t >> GL) * D + 16 * i + g] = both_parts(acc[i][0], acc[i][1]);
      out[(t >> GL) * D + 16 * i + 8 + g] = both_parts(acc[i][2], acc[i][3]);
    }
  if (a.beside_prefix) asm volatile("griddepcontrol.wait;" ::: "memory");
  RowMerge<WPR, RT> merge[G];
  const int64_t bh = (int64_t)b * a.H + h;
#pragma unroll
  for (int i = 0; i < G; ++i) merge[i].load(a, a.rows, bh + i, part * 32 + lane, lane);
  if (WPR == 1) __syncwarp();
  else if (WPR == NW) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "n"(RT) : "memory");
  const float* const outs = reinterpret_cast<const float*>(rings + slot * WPR * f16_warp_bytes<S, G>);
#pragma unroll
  for (int i = 0; i < G; ++i)
    merge[i].template finish<O_STRIDE>(a, a.rows, bh + i, part * 32 + lane, lane, sm_m[i] + slot * WPR, sm_l[i] + slot * WPR, outs + i * D);
}

template <int MODE, int WPR, int S, int G>
static int launch_f16(const BranchArgs& a, cudaStream_t st) {
  static std::atomic<uint64_t> ready;
  constexpr int NW = F16Shape<WPR>::NW, BYTES = NW * f16_warp_bytes<S, G>, PER = NW / WPR * G;
  cudaError_t e = q40_allow_smem(ready, (const void*)attn_branch_f16_kernel<MODE, WPR, S, G>, BYTES);
  const unsigned grid = (unsigned)((a.rows + PER - 1) / PER);
  if (e == cudaSuccess) e = q40_launch_pdl(attn_branch_f16_kernel<MODE, WPR, S, G>, dim3(grid), dim3(NW * 32), BYTES, st, a);
  return e == cudaSuccess ? Q40_OK : (int)e;
}

// Which form a call takes: heads of a row, warps of a row, stages of a ring; heads 0: attn_branch_kernel is faster.  What fits on an SM at
// a time: one CTA of eight warps, two of four with three stages, three of four with two.
struct F16Form { int heads, warps, stages; };
// With lengths, which are on the device.  The table's width only bounds them, and the pool may be larger or shared: neither changes the result,
// so neither may change the form, whose sums have an order of their own.  By rows and prompt alone, then, for what loses least over lengths of up to 16,
// 64, 128, 256 and 500, uniform from 0, in the geometric mean (below: times as long as attn_branch_kernel, least and most of single lengths):
//   4 heads a kv head behind 200 keys, 20 / 26 / 33 branches: two heads a row, two warps 0.85 / 0.85 / 0.75 (0.67 to 1.07), four heads, four warps 0.88 /
//     0.87 / 0.75 (0.51 to 1.26); behind 850, 20 / 26 / 33: two heads, two warps 1.15 / 1.02 / 0.78, four 0.85 / 0.76 / 0.94, four heads, four 0.94 / 0.84 /
//     0.76, two 1.23 / 1.11 / 0.84; 36 branches four 0.83, two 0.83, behind 2048 0.86 and 0.84.  (A long prompt leaves the branches fewer SMs at a
//     time; two heads a kv head behind 1024, 20 / 26 branches, two warps 1.19 / 1.03, four 0.89 / 0.77; behind 100, 26 branches 0.90 and 0.99)
//   one head, 20 / 24 / 27 branches (four and a bit rows an SM), two warps: behind 200 keys 1.08 / 1.01 / 1.00 (to 1.26), behind 700 0.95 / 0.87 / 0.88
//   one head and no prompt, one warp a row: 38 / 42 / 44 / 48 branches 1.15 / 1.02 / 0.95 / 0.92
// Us for lengths up to 16 / 128 / 500: 20 branches 3.4 / 6.5 / 16.7 (four warps a row by scalar products 3.7 / 7.3 / 17.2); 48 branches 4.0 / 10.2 / 34.9
// (5.8 / 10.0 / 36.4)
static F16Form f16_form_of_rows(int64_t all, int rep, int prompt) {
  constexpr int64_t SMS = 148;
  const bool prefix = prompt > 0, far = prompt > 640;
  const int heads = rep % 4 == 0 && all > (prefix && !far ? 8 : 6) * SMS ? 4 : rep % 2 == 0 && all > SMS ? 2 : 1;
  const int64_t rows = all / heads;
  if (heads == 4 && prefix) return {4, 4 * all <= 29 * SMS ? 4 : 2, 2};
  if (heads > 1 && prefix) return {heads, rows <= (far ? 3 : 2) * SMS ? 4 : 2, 2};
  if (heads > 1) return {heads, rows <= SMS ? 8 : rows <= 3 * SMS ? 4 : 2, rows > SMS && rows <= 2 * SMS ? 3 : 2};
  if (rows <= (prefix ? 200 : SMS)) return {0, 0, 0};
  if (rows <= 3 * SMS) return {1, 4, rows <= 2 * SMS ? 3 : 2};
  if (rows <= 4 * SMS) return {0, 0, 0};
  if (rows <= 6 * SMS) return {!prefix || far, 2, 2};
  return {4 * rows > (prefix ? 56 : 37) * SMS, 1, 2};
}

static F16Form f16_form(const BranchArgs& a, int mode, int prompt) {
  constexpr int64_t SMS = 148;
  const bool prefix = a.beside_prefix;
  const int rep = a.H / a.Hkv, L = a.L;
  if (a.seq_lens) return f16_form_of_rows(a.rows, rep, prompt);
  // As many heads as leave rows for the SMs.  Us by heads (of 4 a kv head) at their best number of warps: paged, 300 keys, 96 rows of one head
  // 5.13 / 5.48 / 6.51 with 1 / 2 / 4, 224 rows 7.2 / 5.49 / 6.57, 384 rows 8.5 / 7.6 / 6.9; 20 keys, 640 rows 3.8 / 3.8 / 4.5 (contiguous 3.5 / 3.4 / 3.8, attn_branch_kernel 3.1); 40 keys behind
  // 400, 640 rows 8.2 / 7.6 / 8.6, 1600 rows 12.7 / 10.9 / 11.2
  const int64_t enough = L <= 64 ? (prefix ? 300 : 200) : prefix ? SMS : SMS / 2;
  const int heads = rep % 4 == 0 && a.rows / 4 > enough ? 4 : rep % 2 == 0 && a.rows / 2 > enough ? 2 : 1;
  const int64_t rows = a.rows / heads;
  // Several: as many warps as all rows leave room for, with short ones behind a prefix fewer.  Us, 1 / 2 / 4 / 8 warps (attn_branch_kernel): paged, 512 keys,
  // 160 rows 27.7 / 15.4 / 11.4 (three stages 11.0) / 14.0 (19.1); 100 keys, 320 rows 10.1 / 7.5 / 6.2 / 12.0 (11.0), 800 rows 11.5 / 8.6 / 10.9 / 23.6
  // (18.8); contiguous, 300 keys, 800 rows 23.2 / 21.8 / 23.7 / 35.2 (42.4); 40 keys behind 400, 448 rows 10.3 / 8.2 / 11.3 / 17.1 (10.1)
  if (heads > 1) {
    if (mode == 0 && L < 32 && a.rows <= 8 * SMS) return {0, 0, 0};
    if (prefix && L <= 64) return {heads, 2, 2};
    if (rows <= SMS && !prefix) return {heads, 8, 2};
    if (rows <= 2 * SMS) return {heads, 4, 3};
    if (rows <= 3 * SMS) return {heads, 4, 2};
    return {heads, rows <= 8 * SMS || prefix ? 2 : 1, 2};
  }
  // One, beside the prefix pass.  Us of attn_branch_kernel and here: 320 rows of up to 130 9.5, 8.6, of 40 8.2, 7.6; 480 of 250 11.6, 12.3;
  // 160 of 161 9.2, 9.5, 192 of 142 7.5, 7.1; 832 of 300 18.9, 16.2; 2048 of 138 17.0, 18.6, of 256 behind 2048 37.4, 36.5, 3200 of 250 37.9, 36.1
  if (prefix) {
    if (rep > 1 && L <= 64 && rows > SMS && rows <= 3 * SMS) return {1, 2, 2};
    if (rows <= 2 * SMS) return {rows <= SMS || L <= 150, 4, 3};
    if (rows <= 3 * SMS) return {1, 4, 2};
    return {rows > 5 * SMS && L > 240, 2, 2};
  }
  // One, without.  Us of attn_branch_kernel and here: 64 rows of 700 8.6, 7.9, of 235 4.1, 4.5; 96 of 300 5.8, 5.1; 256 of 400 11.7, 13.0;
  // paged, 320 rows of 512 12.3, 11.5; contiguous 10.6, 9.6, of 130 4.8, 5.1; paged, 480 of 300 9.9, 11.7, 832 16.6, 13.4, 1088 17.8, 22.1, 1280 of
  // 200 18.2, 16.3, 1696 of 352 36.1, 29.7, 1824 of 150 (a wave of one warp a row and a little) 16.4, 21.5, 3200 of 300 58.5, 54.9; 1792 of 52 8.9,
  // 10.9; contiguous, 1824 of 150 27.0, 25.9, 683 101.2, 99.6 (four warps 94.3), 3520 of 683 177.9, 174.0
  if (rows <= SMS) return {L > 384 || (L > 256 && rows > 64), 8, 2};
  if (rows <= 2 * SMS) return {rep > 1 && L <= 64, 4, 3};
  if (rows <= 3 * SMS) return {mode != 0 || L > 256, 4, 2};
  if (rows <= 5 * SMS) return {0, 0, 0};
  if (rows <= 6 * SMS) return {1, 2, 2};
  if (rows <= 8 * SMS || L <= 128) return {0, 0, 0};
  if (mode == 0) return {1, L > 400 ? 4 : 2, 2};
  const int64_t wave = 12 * SMS, waves = (rows + wave - 1) / wave;
  return {rows <= wave || 20 * rows > 17 * waves * wave, 1, 2};
}

template <int MODE, int G>
static int launch_f16_form(const BranchArgs& a, const F16Form& f, cudaStream_t st) {
  if (f.warps == 8) return launch_f16<MODE, 8, 2, G>(a, st);
  if (f.warps == 4) return f.stages == 3 ? launch_f16<MODE, 4, 3, G>(a, st) : launch_f16<MODE, 4, 2, G>(a, st);
  return f.warps == 2 ? launch_f16<MODE, 2, 2, G>(a, st) : launch_f16<MODE, 1, 2, G>(a, st);
}
template <int MODE>
static int launch_f16_heads(const BranchArgs& a, const F16Form& f, cudaStream_t st) {
  return f.heads == 4 ? launch_f16_form<MODE, 4>(a, f, st) : f.heads == 2 ? launch_f16_form<MODE, 2>(a, f, st) : launch_f16_form<MODE, 1>(a, f, st);
}

bool launch_branch_f16(const BranchArgs& a, int mode, int prompt, cudaStream_t st, int& rc) {
  const F16Form f = f16_form(a, mode, prompt);
  if (f.heads == 0) return false;
  rc = mode == 0 ? launch_f16_heads<0>(a, f, st) : mode == 1 ? launch_f16_heads<1>(a, f, st) : launch_f16_heads<2>(a, f, st);
  return true;
}

}  // namespace q40
