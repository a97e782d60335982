// Q4_0 dequant-matmul on the tiled weight copies (format: q40_gemv_tiled.cu) for two CTAs that work as a pair: the
// MMAs are tcgen05 cta_group::2, 256 features of a span x up to 256 batch rows, each CTA of the pair holding 128
// features (its half of the A operand and of the accumulators, both in its tensor memory) and HALF of the batch rows
// of a k block in its shared memory.
//
// Why pairs: a CTA that does 128 features x 256 rows by itself loads 32 KB of activations and 4.3 KB of weights per
// 512 tensor cycles of a k block, 72 bytes a cycle, more than an SM gets from L2 (64 at most); a pair loads 16 KB of
// activations per CTA instead.  The batch rows are the MMA's N, so that a k block is four MMAs whatever the rows.
//
// Persistent: a pair takes a contiguous share of all (tile, k block) units and runs through it without a break, weights
// and activations of the next tile on their way while the last one is finished by warps of its own, out of the second
// of two accumulators (one, if they do not fit tensor memory beside the A buffers).  Roles of a CTA's 24 warps:
//   warp 0        weights: two tensor copies per k block into a ring stage
//   warp 1        issues the MMAs (the even CTA's, for both)
//   warp 2        activations: a TMA copy per 64 k (half of the rows, 128-byte swizzle)
//   warps 4..19   dequantise: four sets of four (one warp per 32 tensor-memory lanes) that take the k blocks in turn
//                 and write fp16(code * scale), the reference's operand value (triton_kernels.py:444-445), to
//                 tensor memory (see q40_gemm_tiled_tc.cu)
//   warps 20..23  accumulators -> output
// The pair's last tile is finished by the dequantiser warps as well.  Where it is the only one, warps 20..23 are a fifth set; where finishing
// is what a pair waits for, warps 16..19 finish too (see layout).
//
// A tile whose k range is cut between pairs: all but the last leave their fp32 sums in a scratch slot (first thing,
// each has one at most) and raise flags; the pair with the last k blocks does them last and adds the slots in order.  A
// pair waits for lower-numbered pairs only, and those publish before they wait, so that no order of scheduling can make
// them wait for each other.  Results depend on nothing but operands and grid.
//
// What bounds it, per 128 k of a tile (cycles): up to 96 rows the dequantisers (430; their loop alone takes 343, of which 260 are the
// half-rate fp16 subtractions and multiplications), at 112 and 128 rows the MMAs (500 and 545 with their gaps, 450 and 512 without), above,
// with all SMs busy, loads from L2 (512 rows x 4096 x 11008: 26 bytes a cycle and SM over a launch).  A launch adds 3.4 to 5: what its CTAs do
// first (1.2, beside the launch in front where that leaves SMs free), activations 0.8, the last accumulator's way out 0.6 to 1.5, the end 0.6.
// As many A buffers as tensor memory has room for (seven up to 32 rows, with four a dequantiser waited half its time for the MMAs of the
// block before); one warp of the epilogue polls.
// Microseconds, launches in a row out of a graph, six sets of weights in turn, the power limit active above 64 rows; before these and now: 10 rows
// x 4096 x 4096 8.2 and 6.9, three of them 13.3 and 12.3, x 11008 x 4096 13.3 and 12.0; 102 rows 9.9 and 9.2, 17.3 and 15.6, 15.8 and 15.4. With the
// SiLU product: 10 rows x 4096 x 11008 17.7 and 16.2, 64 rows 24.3 and 21.2, 100 rows 31.4 and 25.6, 512 rows 94.5 and 82.5 (eight quotients in flight
// at once: see silu). 512 rows without it, whose k blocks wait for L2: 49.6 and 48.3 x 11008, 45.4 and 44.9 x 11008 x 4096.
// With pauses, off the power limit: 144 rows x 4096 x 11008 21.9 and 17.0, 256 rows 25.9 and 24.3, 400 and 512 rows with the SiLU product 73.4 and 61.3, 73.9
// and 70.2; 300 and 400 rows x 11008 x 4096 31.6 and 30.4, 34.2 and 34.3.
//
// Every wait is bounded (by seconds): on expiry an error word is set and no more copies are requested; what is still
// multiplied and stored is undefined, as is the scratch.  Copies and MMAs in flight are waited for, tensor memory is freed.
#include <algorithm>

#include "q40_tc_common.cuh"

namespace q40 {
namespace ttc {
namespace pair {

constexpr int FEATS = 128;                      // features of a CTA
constexpr int MAX_ROWS = 256;
constexpr int DSETS = 4;                        // dequantiser sets, of one warp per tensor-memory quadrant
constexpr int DQ_WARP0 = 4, EPI_WARP0 = DQ_WARP0 + 4 * DSETS;
constexpr int THREADS = (EPI_WARP0 + 4) * 32;
constexpr int BLK = 2;                          // 64-row k steps of a block: 8 MMAs per wait and commit (with 4 the issuing
                                                // thread's own latencies, 390 cycles, bound the loop)
constexpr int RAW_W = 8 * 1024, RAW_S = 8 * 64; // of a block: eight half steps (two 64-column groups each) and their scales
constexpr int RAW_BYTES = RAW_W + RAW_S;
constexpr int RAW_PAD = 9216;                   // next multiple of 1024 (the B tiles want that alignment)
constexpr int S_MAX = 16;                       // ring stages
constexpr int A_COLS = 32 * BLK;                // tensor-memory columns of an A buffer
constexpr int NA_MAX = 8;
constexpr int TMEM_COLS = 512;
constexpr int CUT = 2;                          // a k range is cut at multiples of so many blocks
constexpr int GROUPS = 1 + DSETS;               // of four warps, one per tensor-memory quadrant, that finish a pair's last tile
template <bool EARLY>
constexpr int BAR_BYTES = (EARLY ? 24 : 16) * S_MAX + 8 * NA_MAX + 64;
constexpr uint32_t FLAG_POLLS = 1u << 22;       // of one flag, before giving up: seconds, like the other waits
// Of the other waits: 10 s.  Roles that are there early wait for what the launch in front leaves, which may take the 4 s in which its flags run out; with less
// than that theirs would run out too.  (griddepcontrol.wait ahead of the first of them, by each role: three matrices of 10 rows x 4096 x 4096 11.9 us, 12.3)
constexpr uint32_t WAIT_POLLS = 4 * SPIN_LIMIT;
constexpr int OUT_LD = FEATS + 8;              // halves between rows that wait in shared memory
constexpr int MAX_PAIRS = 128;
constexpr int FLAG_BYTES = MAX_PAIRS * 64;      // at the start of the scratch, per pair: [half][quadrant] arrivals, and as many words without use

// Tensor maps: the activations, and per matrix the weights (box 1024 bytes x 8 steps, half of it with SiLU) and scales (64 bytes x
// 8 steps, or half) of a tiled copy read as rows of one step
struct Maps { CUtensorMap act, w[3], s[3]; };

struct Params {
  __half* c[3];
  int64_t ldc[3];
  int spans[3], nprob;
  int M, K, npad;          // npad: rows of a tile, a multiple of 16
  int chunks;              // row chunks; tile = span * chunks + chunk
  int ntiles, nblk;        // blocks of a tile: up to BLK 64-row k steps of one range
  int k64, range, rblk;    // k steps of a tile and of a range, and blocks of a range.  A range is summed in tensor memory;
                           // the sums of a tile's ranges are added in order
  int cut;                 // tiles may be shared between pairs along k (scratch given)
  int share, rest;         // cut: a pair has share units of CUT blocks, the first `rest` pairs one more
  int bps, own;            // SPLIT: blocks of a rank, and of the four-row groups that it finishes
  int stages, nacc, na;    // ring stages, accumulators, A buffers
  int dsets, egroups;      // sets that dequantise, and groups that finish tiles beside the main loop: four and one; all five where there is
                           // but one tile; three and two where finishing takes longer (see layout)
  int run_off, out_off, bar_off;           // byte offsets in the aligned shared memory (run: SPLIT: sums of the other ranks)
  int silu;                // c[0] = silu(A @ deq(B_0)) * (A @ deq(B_1)): a tile is 128 features of
                           // both, of which a CTA has 64 (its A rows 0..63 those of matrix 0)
  int vec;                 // outputs take 16-byte stores
  const __half* nk_s;      // NK: scales [n_cols][K / 64]
  int n_cols;
  union {                  // (NK never cuts tiles; arguments are launch time)
    float* part;           // scratch slots: [pair][half][npad][128]
    const __half* x;       // NK: activations that no tensor copy takes (8-byte boundaries), or null
  };
  union {
    int* flags;            // per pair: see FLAG_BYTES
    int64_t ldx;
  };
  int* err;
};

// A bounded wait as one instruction to the compiler, and without a way out of the loop around it: what that loop computes
// stays uniform, so that MMA operands are kept in uniform registers (an MMA issues in 15 cycles instead of 53).  `limit` is
// what remains of the polls; it is 0 once a wait has run out, and later ones then ask once.
__device__ __forceinline__ void wait_limited(uint32_t bar, uint32_t parity, uint32_t& limit) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, %3;\n\t"
      "TRY:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %4;\n\t@p bra DONE;\n\t"
      "setp.eq.u32 q, n, 0;\n\t@q bra DONE;\n\tsub.u32 n, n, 1;\n\tbra TRY;\n\t"
      "DONE:\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(limit), "r"(POLL_NS) : "memory");
  limit = ok ? limit : 0;
}
// A position in a ring of n slots and the parity of its turn
struct Slot {
  int i = 0;
  uint32_t turn = 0;
  __device__ __forceinline__ void next(int n) { if (++i == n) { i = 0; turn ^= 1; } }
  __device__ __forceinline__ void skip(int by, int n) { for (i += by; i >= n; i -= n) turn ^= 1; }
};
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// An arrival in the even CTA's shared memory.  It publishes no ordinary stores (tensor-memory accesses are ordered by the
// tcgen05 waits and fences, copies by their own barrier), so it goes without a cluster-wide release, which costs a
// dequantiser warp 1100 cycles
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Four values into the shared memory of a CTA of the cluster, counted by a barrier there
__device__ __forceinline__ void push4(uint32_t dst, const uint32_t (&v)[4], uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}
__device__ __forceinline__ void ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void wait_ld4(uint32_t (&r)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]) :: "memory");
}
// x / (1 + exp(-x)) for x that fp16 can hold.  The quotient by one Newton step for the reciprocal and the remainder of the product
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, 1990): eight of them in flight take a fifth of the
// time of eight divisions one after the other.  Rounded to fp16 it is what those give for every fp16 x, which is what the tests compare.
// Beyond 32 the divisor is 1; below -80 the result is -0 in fp16 whatever the exponential; a zero keeps its sign
// (a remainder of +0 times -r, which is -0, added to it)
__device__ __forceinline__ float silu(float x) {
  const float d = 1.0f + expf(fminf(-x, 80.0f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.0f), r, r);
  const float q = x * r;
  return x > 32.0f ? x : fmaf(fmaf(d, q, -x), -r, q);
}
__device__ __forceinline__ void commit2(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void mma2_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
}

// 16 columns of the lane's own row of tensor memory
__device__ __forceinline__ void st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// Waits for tensor-memory loads; naming the registers keeps their uses behind it
__device__ __forceinline__ void wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}

// `n` finished rows of W features from shared memory to the output, by the 128 threads t of a group
template <int W, bool RAGGED = false>
__device__ __forceinline__ void store_rows(const __half* o, __half* c, int64_t ldc, int n, int t, int vec, int cols = W) {
  if (RAGGED && (cols < W || vec == 2)) {                    // fewer features than W, or rows at any address
    for (int row = t / 32; row < n; row += 4)
      for (int col = t % 32; col < cols; col += 32) c[row * ldc + col] = o[row * OUT_LD + col];
  } else if (vec) {
    const int col = t % (W / 8) * 8;
    for (int row = t / (W / 8); row < n; row += 1024 / W)
      *reinterpret_cast<uint4*>(c + row * ldc + col) = *reinterpret_cast<const uint4*>(o + row * OUT_LD + col);
  } else {
    const int col = t % (W / 2) * 2;
    for (int row = t / (W / 2); row < n; row += 256 / W)
      *reinterpret_cast<uint32_t*>(c + row * ldc + col) = *reinterpret_cast<const uint32_t*>(o + row * OUT_LD + col);
  }
}

// First block of pair q
__device__ __forceinline__ int first_block(const Params& p, int q, int npairs) {
  if (q >= npairs) return p.ntiles * p.nblk;
  if (!p.cut) return (int)((uint32_t)p.ntiles * (uint32_t)q / (uint32_t)npairs) * p.nblk;
  return CUT * (q * p.share + min(q, p.rest));
}

// The k steps of block b of a tile, and of those behind it
struct KCursor {
  int k, end;                                  // first k step; end of the range it belongs to
  __device__ __forceinline__ KCursor(const Params& p, int b) {
    const int r = b / p.rblk;
    k = r * p.range + (b - r * p.rblk) * BLK;
    end = min(p.k64, (r + 1) * p.range);
  }
  __device__ __forceinline__ bool next(const Params& p) {      // true: the range has ended
    k = min(k + BLK, end);
    if (k < end) return false;
    end = min(p.k64, end + p.range);
    return true;
  }
};

// NK: 64 bytes of a row, 16 at a time, are 64 k of one group in their high nibbles and 64 k of the next in their low ones, and a lane's columns of
// the A buffer from ta on and from ta + 32 on: fp16(code * scale) of k pairs.  The 16-byte pieces lie swizzled (64 bytes)
__device__ __forceinline__ void dequant_row(const unsigned char* row, int swizzle, uint32_t scales, uint32_t ta) {
  constexpr uint32_t HI = 0x54805480u, LO = 0x64086408u;     // see dequant_step; both codes are two's complement here
  const __half2 sh = __low2half2(u32_as_h2(scales)), sl = __high2half2(u32_as_h2(scales));
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t hi[16], lo[16];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const uint4 v = *reinterpret_cast<const uint4*>(row + (((2 * h + c) ^ swizzle) << 4));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t p0 = prmt(w[j], w[j], 0x1100), p1 = prmt(w[j], w[j], 0x3322);       // bytes 0 and 1, 2 and 3, to 16 bits each
        hi[8 * c + 2 * j] = deq_pair<HI>(lop3_and_xor(p0, 0x00F000F0u, HI), sh);
        hi[8 * c + 2 * j + 1] = deq_pair<HI>(lop3_and_xor(p1, 0x00F000F0u, HI), sh);
        lo[8 * c + 2 * j] = deq_pair<LO>(lop3_and_xor(p0, 0x000F000Fu, LO), sl);
        lo[8 * c + 2 * j + 1] = deq_pair<LO>(lop3_and_xor(p1, 0x000F000Fu, LO), sl);
      }
    }
    st_32x32b_x16(ta + 16 * h, hi);
    st_32x32b_x16(ta + 32 + 16 * h, lo);
  }
}

// The pieces of tiles that a pair works on, in the order it takes them: the one it publishes first (the last tile, if its
// k range goes on beyond the pair's share), the one it may have to wait for last (the first tile)
struct Work {
  int u0, u1, nblk, t0, t1, np;
  bool pub;
  __device__ __forceinline__ Work(int4 w, int n) : u0(w.x), u1(w.y), nblk(n), t0(w.z), t1(w.w) {
    np = u1 > u0 ? t1 - t0 + 1 : 0;
    pub = u1 > u0 && u1 < (t1 + 1) * n;
  }
  // First and last block (exclusive) of the pair, and their tiles
  static __device__ __forceinline__ int4 share(int a, int b, int n) { return make_int4(a, b, a / n, (max(b, a + 1) - 1) / n); }
  __device__ __forceinline__ void piece(int k, int& tile, int& b0, int& b1) const {
    tile = k == np - 1 ? t0 : (pub ? (k == 0 ? t1 : t0 + k) : t0 + 1 + k);
    b0 = tile == t0 ? u0 - tile * nblk : 0;
    b1 = tile == t1 ? u1 - tile * nblk : nblk;
  }
};

// SPLIT: the k range of one tile is spread over the pairs of a cluster (grid y), whose fp32 sums meet through
// distributed shared memory.  Otherwise a cluster is a pair.
// CUT: tiles may be shared between pairs along k; SILU: see Params (compiled for each, to keep the registers of all roles
// below the 80 that 24 warps leave)
// NK: one matrix [n_cols, K] with groups along K, as quantised in memory (not a tiled copy): a lane expands its own feature's row
// EARLY: weights are expanded before their block's activations have landed, which the launch in front may still write.  Where a pair has one tile:
// 10 rows x 4096 x 4096 6.9 us, 7.2 without; 100 rows 9.2 and 9.6.  Where it has several the wait of its own costs more: 512 rows x 4096 x 11008 46.4
// without and 49.6, x 11008 x 4096 43.2 and 44.4, 100 x 11008 x 11008 33.1 and 34.1 (for a pair's first blocks alone: 48.4, 44.3, 33.3)
template <bool EARLY, bool SPLIT, bool CUT_K, bool SILU, bool NK = false>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const Params p, const __grid_constant__ Maps maps) {
  extern __shared__ unsigned char smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = blockIdx.x & 1, me = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const uint32_t lead = SPLIT ? 2 * blockIdx.y : 0;          // rank of the pair's even CTA in the cluster
  const int S = p.stages, NA = p.na;                         // at least as many stages as A buffers, and four
  const uint32_t b_bytes = (uint32_t)p.npad * 64u;           // B tile of a k step: npad / 2 rows x 64 k x 2 B
  const uint32_t stage_bytes = RAW_PAD + BLK * b_bytes;

  const uint32_t raw0 = smem_u32(smem_raw);
  const uint32_t ring = (raw0 + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (ring - raw0);
  // Block i has stage and barriers i % S and A buffer i % NA.  full: its weights and activations have landed in this
  // CTA (EARLY: its weights; act: its activations); mdone: its MMAs are complete, in both CTAs; accfull[b]: an accumulator is complete.  In the even CTA, for
  // both: afull: the A operand is written (and the activations have landed); accfree[b]: an accumulator has been read.
  const uint32_t bar_full = ring + (uint32_t)p.bar_off, bar_act = EARLY ? bar_full + 8 * S_MAX : bar_full, bar_mdone = bar_act + 8 * S_MAX,
                 bar_afull = bar_mdone + 8 * S_MAX, bar_accfull = bar_afull + 8 * NA_MAX, bar_accfree = bar_accfull + 16,
                 bar_done = bar_accfree + 16, bar_last = bar_done + 8, bar_flags = bar_last + 8, bar_recv = bar_flags + 8;
  unsigned char* tail = gbase + p.bar_off + BAR_BYTES<EARLY>;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail);
  volatile int* s_failed = reinterpret_cast<volatile int*>(tail + 8);
  volatile int* s_acc = reinterpret_cast<volatile int*>(tail + 24);        // accumulator of a pair's last tile
  volatile int* s_copied = reinterpret_cast<volatile int*>(tail + 16);     // blocks requested: [0] weights, [1] activations, [3] copy_rows' second warp
  int4* s_share = reinterpret_cast<int4*>(tail + 32);                      // see Work::share
  float* run = reinterpret_cast<float*>(gbase + p.run_off);                // [npad][128] sums of earlier ranges
  __half* out_s = reinterpret_cast<__half*>(gbase + p.out_off);            // [2][16][OUT_LD] finished rows on their way out

  // matrix, span, 128-feature half of this CTA (SiLU: of the tile, in both matrices) and first row of a tile
  auto decode = [&](int tile, int& pi, int& span, int& fh, int& m0) {
    span = tile / p.chunks;
    m0 = (tile - span * p.chunks) * p.npad;
    if (SILU) {
      pi = 0;
      fh = span & 1;
      span >>= 1;
      return;
    }
    pi = 0;
    fh = half;
    while (pi < p.nprob - 1 && span >= p.spans[pi]) { span -= p.spans[pi]; ++pi; }
  };
  bool failed = false;
  uint32_t limit = WAIT_POLLS;                               // see wait_limited

  // ---- copies of blocks first .. last - 1 of the pair, weights or activations.  `first`: 0, or S where the first S have been requested:
  // weights do not depend on the previous launch, so their first stages are, before anything else ----
  int requested = 0;
  auto copy_blocks = [&](const Work& wk, int first, int last, bool weights) {
    int i = 0;                                               // first block of a piece
    Slot sl;
    sl.turn = first > 0;
    requested = first;
    for (int k = 0; k < wk.np && i < last; ++k) {
      int tile, b0, b1, pi, span, fh, m0;
      wk.piece(k, tile, b0, b1);
      const int from = max(first - i, 0), to = min(b1 - b0, last - i);
      i += b1 - b0;
      if (from >= to) continue;
      decode(tile, pi, span, fh, m0);
      KCursor kc(p, b0 + from);
      for (int b = from; b < to; ++b, kc.next(p)) {
        const int s = sl.i;
        if (requested >= S) wait_limited(bar_mdone + 8 * s, sl.turn ^ 1, limit);
        if (limit == 0) return;
        const uint32_t dst = ring + s * stage_bytes;
        if (weights) {
          const int step = (span * p.k64 + kc.k) * 4;
          mbar_expect_tx(bar_full + 8 * s, NK ? RAW_W : RAW_BYTES);
          if constexpr (NK) {
            tma_2d(dst, &maps.w[0], kc.k * 32, span * SPAN + half * FEATS, bar_full + 8 * s);                  // x in bytes
          } else if constexpr (SILU) {                                                  // a 64-column group of each matrix
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              tma_2d(dst + m * (RAW_W / 2), &maps.w[m], fh * 256 + half * 128, step, bar_full + 8 * s);    // x in words of four bytes
              tma_2d(dst + RAW_W + m * (RAW_S / 2), &maps.s[m], 512 + fh * 16 + half * 8, step, bar_full + 8 * s);
            }
          } else {
            tma_2d(dst, &maps.w[pi], fh * 256, step, bar_full + 8 * s);
            tma_2d(dst + RAW_W, &maps.s[pi], 512 + fh * 16, step, bar_full + 8 * s);
          }
        } else {
          // the second k step of a range's last block may be the next range's or beyond K (zeros): not multiplied
          mbar_expect_tx(bar_act + 8 * s, BLK * b_bytes);
#pragma unroll
          for (int h = 0; h < BLK; ++h)
            tma_2d(dst + RAW_PAD + h * b_bytes, &maps.act, (kc.k + h) * BK, m0 + half * (p.npad / 2), bar_act + 8 * s);
        }
        ++requested;
        sl.next(S);
      }
    }
  };
  // The activations of all blocks, eight bytes a lane, one k step of each by this warp; four blocks on their way.  Rows of the tile behind the last
  // keep what was there: nothing is stored of their products.  Here, and by tensor copies behind a launch that copies the rows to 16 bytes: 10 rows
  // x 11008 x 4096 15.4 and 15.9 us, 40 x 4096 x 11008 20.3 and 16.7, 100 rows 28.9 and 18.2 (by one warp 81, with rows of zeros; copies of eight
  // bytes are what it waits for).  In place all the same: two threads on a stream may have their copies and products in any order
  auto copy_rows = [&](const Work& wk, int h) {
    constexpr int AHEAD = 3;                                 // below the number of stages
    const int at = lane & 15, r0 = lane >> 4;
    uint32_t to[4];                                          // rows r0, r0 + 2, .. + 6 of every eight
#pragma unroll
    for (int j = 0; j < 4; ++j) to[j] = RAW_PAD + h * b_bytes + (r0 + 2 * j) * 128 + (((at >> 1) ^ (r0 + 2 * j)) << 4) + 8 * (at & 1);
    Slot sl, landed;
    int n = 0, arrived = 0;
    const auto arrive = [&]() {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the products read them through another proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_act + 8 * landed.i);
      landed.next(S);
      ++arrived;
    };
    for (int k = 0; k < wk.np && limit; ++k) {
      int tile, b0, b1, pi, span, fh, m0;
      wk.piece(k, tile, b0, b1);
      decode(tile, pi, span, fh, m0);
      m0 += half * (p.npad / 2);
      const int rows = min(p.npad / 2, p.M - m0) - r0;
      const __half* src = p.x + (m0 + r0) * p.ldx + (b0 * BLK + h) * BK + 4 * at;
      for (int b = b0; b < b1; ++b, src += BLK * BK) {
        if (n >= S) wait_limited(bar_mdone + 8 * sl.i, sl.turn ^ 1, limit);
        limit = __all_sync(0xffffffffu, limit != 0) ? limit : 0;
        if (limit == 0) break;
        uint32_t dst = ring + sl.i * stage_bytes;
        const __half* from = src;
        for (int r = 0; r < rows; r += 8, dst += 1024, from += 8 * p.ldx) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (r + 2 * j < rows)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + to[j]), "l"(from + 2 * j * p.ldx) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        sl.next(S);
        if (++n > AHEAD) {
          asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
          arrive();
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    while (arrived < n) arrive();
    s_copied[h ? 3 : 1] = n;
    failed = limit == 0;
  };
  // Until then, only the warps that have something to do run: with all 24 finding out their share (five divisions) first, the first
  // weights were requested 1.4 to 1.9 us after the start of a CTA
  if (warp == 0) {
    if (lane == 0) {
      *s_failed = 0;
      mbar_init(bar_done, 1);
      mbar_init(bar_last, 4);
      mbar_init(bar_flags, 4);
      mbar_init(bar_recv, 1);
      if (SPLIT) {
        const int own = min(p.own, (p.M + 3) / 4 - (int)blockIdx.y * p.own);
        if (own > 0) mbar_expect_tx(bar_recv, (gridDim.y - 1) * own * FEATS * 16);
      }
    }
    if (lane < S) {
      const int acts = NK && p.x ? BLK : 1;                  // arrivals of a block's activations
      mbar_init(bar_full + 8 * lane, EARLY ? 1 : 1 + acts);
      if (EARLY) mbar_init(bar_act + 8 * lane, acts);
      mbar_init(bar_mdone + 8 * lane, 1);
    }
    if (lane < NA) mbar_init(bar_afull + 8 * lane, 8);
    if (lane < 2) { mbar_init(bar_accfull + 8 * lane, 1); mbar_init(bar_accfree + 8 * lane, 8 * p.egroups); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const int sb0 = SPLIT ? blockIdx.y * p.bps : 0, sb1 = SPLIT ? min(p.nblk, sb0 + p.bps) : 0;
    const int4 share = Work::share(SPLIT ? me * p.nblk + sb0 : first_block(p, me, npairs),
                                   SPLIT ? me * p.nblk + sb1 : first_block(p, me + 1, npairs), p.nblk);
    if (lane == 0) *s_share = share;
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (elect_one()) {
      if (NK) asm volatile("griddepcontrol.wait;" ::: "memory");       // the launch in front may be the one that writes the weights
      copy_blocks(Work(share, p.nblk), 0, S, true);
    }
    __syncwarp();
  } else {
    if (warp == 1) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TMEM_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp == 3 && lane <= (NK ? 1 : 2 * p.nprob) && !(NK && lane == 0 && p.x)) {
      const CUtensorMap* m = lane == 0 ? &maps.act : lane <= p.nprob ? &maps.w[lane - 1] : &maps.s[lane - 1 - p.nprob];
      asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // both CTAs' barriers and tensor memory are there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const Work wk(*s_share, p.nblk);
  const int total = wk.u1 - wk.u0;                    // blocks of this pair
  const uint32_t A_COL0 = TMEM_COLS - A_COLS * NA;
  asm volatile("griddepcontrol.launch_dependents;");

  if (NK && p.x && (warp == 2 || warp == 3)) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    copy_rows(wk, warp - 2);
  } else if (warp == 0 || warp == 2) {
    if (elect_one()) {
      if (warp == 0) {
        if (total > S) copy_blocks(wk, S, total, true);
      } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        copy_blocks(wk, 0, total, false);
      }
      failed = limit == 0;
      s_copied[warp >> 1] = requested;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (half == 0) {
      // instruction descriptor: D fp32, A and B fp16 and K-major, N = npad, M = 256 over the two CTAs
      const uint32_t idesc = (1u << 4) | ((uint32_t)(p.npad >> 3) << 17) | ((uint32_t)(2 * FEATS >> 4) << 24);
      const uint16_t both = (uint16_t)(3u << lead);
      const uint64_t bdesc = kmajor_desc(ring + RAW_PAD);
      const uint32_t b_step = b_bytes >> 4, stage_step = stage_bytes >> 4;
      if (elect_one()) {
        Slot sl, sa, sc;                                     // stage, A buffer, accumulator
        uint32_t bofs = 0;                                   // of the stage, in the operand descriptor's unit
        int g = 0;
        for (int k = 0; k < wk.np; ++k) {
          int tile, b, b1;
          wk.piece(k, tile, b, b1);
          while (b < b1) {                                   // a range, or the pair's share of it
            const int r = b / p.rblk, e = min(b1, (r + 1) * p.rblk);
            // its last block may be one k step
            const int odd = min(p.k64, (r + 1) * p.range) - (r * p.range + (e - 1 - r * p.rblk) * BLK) < BLK ? e - 1 : -1;
            if (g >= p.nacc) wait_limited(bar_accfree + 8 * sc.i, sc.turn ^ 1, limit);
            const uint32_t acc = tmem + sc.i * p.npad;
            uint32_t accum = 0;
            for (; b < e; ++b) {
              wait_limited(bar_afull + 8 * sa.i, sa.turn, limit);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint64_t bd0 = bdesc + bofs, bd1 = bd0 + b_step;
              const uint32_t ta = tmem + A_COL0 + sa.i * A_COLS, done = bar_mdone + 8 * sl.i;
              sl.next(S);
              sa.next(NA);
              bofs = sl.i ? bofs + stage_step : 0;
#pragma unroll
              for (int ks = 0; ks < BK / 16; ++ks) mma2_ts(acc, ta + ks * 8, bd0 + (uint64_t)(ks * 2), idesc, ks ? 1u : accum);
              if (b != odd) {
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks) mma2_ts(acc, ta + 32 + ks * 8, bd1 + (uint64_t)(ks * 2), idesc, 1);
              }
              commit2(done, both);
              accum = 1;
            }
            commit2(bar_accfull + 8 * sc.i, both);
            sc.next(p.nacc);
            ++g;
          }
        }
        failed = limit == 0;
        commit2(bar_done, both);
      }
      __syncwarp();
    }
  } else if (warp >= DQ_WARP0 && (warp - DQ_WARP0) >> 2 < p.dsets) {
    // warp = (set, quadrant): 32 feature rows = two 16-row tiles of one 64-column group, all k of a block.  Lane (g, t) holds, per
    // 16-row tile and 16 k, rows g and g + 8 at k = 4t .. 4t + 3
    const int quad = warp & 3, dset = (warp - DQ_WARP0) >> 2, dsets = p.dsets;
    const int q = quad >> 1, t = lane & 3;
    // bytes between half steps of a group, and between groups: of one matrix, side by side; with SiLU each of its own
    constexpr int WSTEP = SILU ? 512 : 1024, SSTEP = SILU ? 32 : 64, WGRP = SILU ? RAW_W / 2 : 512, SGRP = SILU ? RAW_S / 2 : 32;
    const unsigned char* lane_w = gbase + q * WGRP + lane * 16 + (quad & 1) * 8;
    const unsigned char* lane_s = gbase + RAW_W + q * SGRP + t * 8;
    const uint32_t afull_lead = mapa(bar_afull, lead), ta0 = tmem + ((uint32_t)(32 * quad) << 16) + A_COL0;
    Slot sl, sa, sw;                             // stage and A buffer of this block, and stage of the one that used the buffer before
    for (sl.i = dset, sa.i = dset; sa.i >= NA; sa.i -= NA) sa.turn ^= 1;
    for (sw.i = dset; sw.i < NA;) sw.i += dsets;
    sw.i -= NA;                                  // of the first block that waits for one; below dsets, and so below S
    // NK: the lane's row, where this block's scales are, and how many blocks of the piece begin there; scales are read a block ahead
    const __half* sc = nullptr;
    int piece = 0, kb = dset, len = 1;
    uint32_t scales = 0;
    auto next_scales = [&]() {
      if (sc == nullptr || kb >= len) {
        if (sc != nullptr) { kb -= len; ++piece; }
        for (;; ++piece) {
          int tile, b0, b1, pi, span, fh, m0;
          wk.piece(piece, tile, b0, b1);
          decode(tile, pi, span, fh, m0);
          len = b1 - b0;
          sc = p.nk_s + (int64_t)min(span * SPAN + fh * FEATS + 32 * quad + lane, p.n_cols - 1) * (p.K / 64) + 2 * b0;
          if (kb < len) break;
          kb -= len;
        }
      }
      scales = __ldg(reinterpret_cast<const uint32_t*>(sc + 2 * kb));
      kb += dsets;
    };
    const int frow = 32 * quad + lane;
    if constexpr (NK) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (dset < total) next_scales();
    }
    for (int i = dset; i < total; i += dsets) {
      // The MMAs of the block that last used this A buffer are complete.  As the ring has at least NA stages, the block that
      // last used this stage is through as well, and the stage's barriers, which tell only odd from even phases, are in one
      // of the two phases that they can tell apart
      if (i >= NA) {
        wait_limited(bar_mdone + 8 * sw.i, sw.turn, limit);
        sw.skip(dsets, S);
      }
      wait_limited(bar_full + 8 * sl.i, sl.turn, limit);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t so = sl.i * stage_bytes, ta = ta0 + sa.i * A_COLS;
      if constexpr (NK) {
        const uint32_t now = scales;
        if (i + dsets < total) next_scales();
        dequant_row(gbase + so + frow * 64, (frow >> 1) & 3, now, ta);
      } else
#pragma unroll
      for (int h = 0; h < BLK; ++h) {
        uint32_t r[2][16];
#pragma unroll
        for (int st = 0; st < 4; ++st) dequant_step(lane_w + so + (4 * h + st) * WSTEP, lane_s + so + (4 * h + st) * SSTEP, r, st);
        st_16x256b_x4(ta + 32 * h, r[0]);
        st_16x256b_x4(ta + 32 * h + (16u << 16), r[1]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      if constexpr (EARLY) wait_limited(bar_act + 8 * sl.i, sl.turn, limit);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(afull_lead + 8 * sa.i);
      sl.skip(dsets, S);
      sa.skip(dsets, NA);
    }
    failed = limit == 0;
  }
  if (!SPLIT && warp >= DQ_WARP0) {
    // ================= accumulators -> output =================
    // Group 0 (warps 20..23; with it group 1, of warps 16..19, if p.egroups is 2) finishes every tile but the pair's last beside the main
    // loop; the last one (the last range of it) falls to all groups, the dequantisers having come to their end: 16-row chunks group,
    // group + GROUPS, ...
    // No wait leaves these loops early, so that the warps of a group always meet at its (plain) barrier.
    const int group = DSETS - ((warp - DQ_WARP0) >> 2), E = SILU && !CUT_K ? 1 : p.egroups;
    const int quad = warp & 3, feat = 32 * quad + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * quad) << 16);
    // two buffers of 16 finished rows per group; those of groups E.. over the ring, which is idle by then
    __half* out_g = (group < E ? out_s + group * 2 * 16 * OUT_LD : reinterpret_cast<__half*>(gbase) + (group - E) * 2 * 16 * OUT_LD);
    const int nchunk = p.npad / 16;
    Slot sc;                                                 // accumulator
    int turn = 0;                                            // output buffer
    const int ranges = CUT_K ? wk.np : wk.np * ((p.nblk + p.rblk - 1) / p.rblk);
    int gr = 0;                                              // ranges that this group has read
    // outputs, scratch and flags may still be in use by the launch in front of this one
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int k = group < E ? 0 : max(0, wk.np - 1); k < wk.np; ++k) {
      int tile, b0, b1, pi, span, fh, m0;
      wk.piece(k, tile, b0, b1);
      decode(tile, pi, span, fh, m0);
      const bool whole = !CUT_K || b1 == p.nblk;                       // this pair has the tile's last blocks and finishes it
      const int rows = min(p.npad, p.M - m0), cols = NK ? min(FEATS, p.n_cols - span * SPAN - fh * FEATS) : FEATS;
      const int64_t ldc = p.ldc[pi];
      __half* c = p.c[pi] + (int64_t)m0 * ldc + span * SPAN + fh * FEATS + (SILU ? half * (FEATS / 2) : 0);
      // the pairs with its first blocks, whose sums are added in k order
      int q0 = me;
      if (CUT_K && whole && b0 > 0) {
        --q0;
        while (q0 > 0 && first_block(p, q0, npairs) > wk.u0 - b0) --q0;
      }
      bool all = false;
      for (int b = b0; b < b1;) {
        const int e = CUT_K ? b1 : min(b1, (b / p.rblk + 1) * p.rblk);    // a range, or the pair's share of it
        const bool add_run = b > b0;
        b = e;
        all = e == b1 && k == wk.np - 1;
        if (group >= E && !all) continue;
        const int ch0 = group, step = all ? GROUPS : E;
        const float* first = p.part + ((int64_t)(q0 * 2 + half) * p.npad) * FEATS + feat;
        float v[16];
        if (CUT_K && e == b1 && q0 < me) {
          // group 0 looks at the flags, makes them ready for the next launch and tells the others
          if (group == 0) {
            for (int q = q0; q < me; ++q) {
              int* flag = p.flags + q * 16 + half * 4 + quad;
              int arrived;
              uint32_t polls = FLAG_POLLS;
              do {
                asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(arrived) : "l"(flag) : "memory");
                if (arrived < GROUPS) { __nanosleep(64); --polls; }
              } while (arrived < GROUPS && polls && limit);
              if (arrived < GROUPS) limit = 0;
              __syncwarp();
              if (lane == 0) *flag = 0;
            }
            if (lane == 0) mbar_arrive(bar_flags);
          } else {
            wait_limited(bar_flags, 0, limit);
          }
          if (ch0 < nchunk) {                                // while the last MMAs run
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __ldcg(first + (ch0 * 16 + j) * FEATS);
          }
        }
        // (a barrier's parity tells a phase from its neighbours only: the other groups, which have not followed accfull,
        // wait for the end of all MMAs and for group 0, which has)
        if (group < E) {
          // one warp polls for the four (polls are issue slots: with all of them, and three more warps that had nothing else to do, a
          // third of all instructions)
          if (quad == 2) wait_limited(bar_accfull + 8 * sc.i, sc.turn, limit);
          asm volatile("bar.sync %0, 128;" ::"r"(1 + GROUPS + group) : "memory");
          if (all && group == 0 && lane == 0) {
            *s_acc = sc.i;
            mbar_arrive(bar_last);
          }
        } else {
          wait_limited(bar_done, 0, limit);
          wait_limited(bar_last, 0, limit);
          sc.i = *s_acc;
        }
        limit = __all_sync(0xffffffffu, limit != 0) ? limit : 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = lane_base + sc.i * p.npad;
        constexpr bool AHEAD = !CUT_K && !SILU;              // the others have no registers for it
        uint32_t nx[16];                                     // the next chunk
        if (AHEAD && ch0 < nchunk) ld16(acc + ch0 * 16, nx);
#pragma unroll 1
        for (int ch = ch0; ch < nchunk; ch += step) {
          uint32_t r[16];
          if constexpr (!AHEAD) {
            ld16(acc + ch * 16, r);
            wait_ld16(r);
          } else {
            wait_ld16(nx);
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = nx[j];
            if (ch + step < nchunk) ld16(acc + (ch + step) * 16, nx);
          }
          if (CUT_K && q0 < me) {
            for (int q = q0 + 1; q < me; ++q) {
              const float* src = first + ((int64_t)(q - q0) * 2 * p.npad + ch * 16) * FEATS;
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += __ldcg(src + j * FEATS);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(v[j] + __uint_as_float(r[j]));
            if (ch + step < nchunk) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __ldcg(first + ((ch + step) * 16 + j) * FEATS);
            }
          }
          if (!CUT_K && add_run) {
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(run[(ch * 16 + j) * FEATS + feat] + __uint_as_float(r[j]));
          }
          if (!CUT_K && e < b1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) run[(ch * 16 + j) * FEATS + feat] = __uint_as_float(r[j]);
          } else if (CUT_K && !whole) {
            float* dst = p.part + ((int64_t)(me * 2 + half) * p.npad + ch * 16) * FEATS + feat;
#pragma unroll
            for (int j = 0; j < 16; ++j) __stcg(dst + j * FEATS, __uint_as_float(r[j]));
          } else if (SILU) {
            // warps 0 and 1 of a group have silu's argument (matrix 0), 2 and 3 the factor of the same features; each finish eight
            // of the 16 rows and give the others, through the unused half of the output buffer, what they need for theirs
            const int hi = quad >> 1, f64 = feat & 63;
            union { uint4 v; __half2 h[4]; } mine, x;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __half2 r_lo = __floats2half2_rn(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
              const __half2 r_hi = __floats2half2_rn(__uint_as_float(r[8 + 2 * j]), __uint_as_float(r[9 + 2 * j]));
              mine.h[j] = hi ? r_hi : r_lo;
              x.h[j] = hi ? r_lo : r_hi;
            }
            __half* o = out_g + (turn ^= 1) * 16 * OUT_LD;
            const auto xchg = [&](int i) { return reinterpret_cast<uint4*>(o + (i >> 3) * OUT_LD + FEATS / 2 + (i & 7) * 8); };
            *xchg(feat ^ 64) = x.v;
            asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
            x.v = *xchg(feat);
            // (Also where all eight are padding.  With a branch around these the whole takes longer: 8 rows x 4096 x 11008 15.5 and 15.9 us, 64
            // 17.6 and 19.2, 100 23.1 and 24.0)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __half22float2(hi ? x.h[j] : mine.h[j]);
              const __half2 y = __hmul2(__floats2half2_rn(silu(f.x), silu(f.y)), hi ? mine.h[j] : x.h[j]);
              o[(8 * hi + 2 * j) * OUT_LD + f64] = __low2half(y);
              o[(8 * hi + 2 * j + 1) * OUT_LD + f64] = __high2half(y);
            }
            asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
            store_rows<FEATS / 2>(o, c + (int64_t)ch * 16 * ldc, ldc, min(16, rows - ch * 16), feat, p.vec);
          } else {
            // 16 rows x 128 features meet in shared memory, so that rows leave in 16-byte stores of 16 lanes (a warp's own
            // 64 bytes of a row at a time: 85 cycles each, 11000 for a tile of 128 rows)
            __half* o = out_g + (turn ^= 1) * 16 * OUT_LD;
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j * OUT_LD + feat] = __float2half_rn(__uint_as_float(r[j]));
            asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
            store_rows<FEATS, NK>(o, c + (int64_t)ch * 16 * ldc, ldc, min(16, rows - ch * 16), feat, p.vec, cols);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        // an arrival that nobody waits for could find the even CTA gone
        if (!all && ++gr + p.nacc <= ranges && lane == 0) mbar_arrive_cluster(mapa(bar_accfree, lead) + 8 * sc.i);
        sc.next(p.nacc);
      }
      if (CUT_K && !whole) {
        // published: GROUPS arrivals per flag, whoever drained the accumulator
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicAdd(p.flags + me * 16 + half * 4 + quad, all || group > 0 ? 1 : GROUPS - (E - 1));
      }
    }
    failed = failed || limit == 0;
  }
  if (warp >= DQ_WARP0) wait_limited(bar_done, 0, limit);
  if (failed || limit == 0) *s_failed = 1;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  failed = *s_failed != 0;
  if (failed && tid == 0) {
    // the copies still on their way, those of the last S blocks at most: none may land in shared memory that has been given back
    q40_set_error(p.err);
    mbar_wait(bar_done, 0);                                  // MMAs, too: a wait that is over asked for them only once
    if constexpr (EARLY) {
      for (int h = 0; h < 2; ++h)
        for (int n = h && NK && p.x ? min(s_copied[1], s_copied[3]) : s_copied[h], i = max(0, n - S); i < n; ++i)
          mbar_wait((h ? bar_act : bar_full) + 8 * (i % S), (uint32_t)((i / S) & 1));
    } else {
      // (first in the place of those that gave up before they requested a block that another did)
      for (int h = 0, n = max(s_copied[0], s_copied[1]); h < (NK && p.x ? 3 : 2); ++h)
        for (int i = s_copied[h == 2 ? 3 : h]; i < n; ++i) mbar_arrive(bar_full + 8 * (i % S));
      for (int n = max(s_copied[0], s_copied[1]), i = max(0, n - S); i < n; ++i) mbar_wait(bar_full + 8 * (i % S), (uint32_t)((i / S) & 1));
    }
  }

  if (SPLIT && warp >= DQ_WARP0) {
    // The ranks of a cluster have the sums of a k range each.  Of the groups of four rows, rank r finishes p.own: it gets the others' from
    // them, as they come to their end, and adds all in k order
    const int quad = warp & 3, group = (warp - DQ_WARP0) >> 2, feat = 32 * quad + lane;
    const int nranks = (int)gridDim.y, rank = (int)blockIdx.y;
    int pi, span, fh, m0;
    decode(me, pi, span, fh, m0);
    const int rows = min(p.npad, p.M - m0), ngroups = (rows + 3) / 4;
    const int g0 = min(ngroups, rank * p.own), g1 = min(ngroups, g0 + p.own);
    const uint32_t acc = tmem + ((uint32_t)(32 * quad) << 16);
    const uint32_t recv = ring + (uint32_t)p.run_off;        // [rank, without this one's][group][feature][row]
    if (!failed) {
      for (int g = group; g < ngroups; g += GROUPS) {
        const int to = g / p.own;
        if (to == rank) continue;
        uint32_t r[4];
        ld4(acc + 4 * g, r);
        wait_ld4(r);
        const int slot = rank < to ? rank : rank - 1;
        push4(mapa(recv, 2 * to + half) + (uint32_t)(((slot * p.own + g - to * p.own) * FEATS + feat) * 16), r, mapa(bar_recv, 2 * to + half));
      }
    }
    if (g0 < g1 && !failed) {
      wait_limited(bar_recv, 0, limit);
      __half* o = reinterpret_cast<__half*>(gbase) + group * 4 * OUT_LD;     // over the ring, which is idle
      const float4* in = reinterpret_cast<const float4*>(gbase + p.run_off) + feat;
      __half* c = p.c[pi] + (int64_t)m0 * p.ldc[pi] + span * SPAN + fh * FEATS;
      for (int g = g0 + group; g < g1; g += GROUPS) {
        uint32_t r[4];
        ld4(acc + 4 * g, r);
        wait_ld4(r);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < nranks; ++k) {
          float4 t = make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
          if (k != rank) t = in[((k < rank ? k : k - 1) * p.own + g - g0) * FEATS];
          v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        o[feat] = __float2half_rn(v.x);
        o[OUT_LD + feat] = __float2half_rn(v.y);
        o[2 * OUT_LD + feat] = __float2half_rn(v.z);
        o[3 * OUT_LD + feat] = __float2half_rn(v.w);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
        store_rows<FEATS, NK>(o, c + (int64_t)(4 * g) * p.ldc[pi], p.ldc[pi], min(4, rows - 4 * g), feat, p.vec,
                              NK ? min(FEATS, p.n_cols - span * SPAN - fh * FEATS) : FEATS);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
      }
      if (limit == 0) q40_set_error(p.err);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  // No ordinary store is meant for another CTA, and what a CTA still sends another is waited for there: execution alone meets here (with the
  // default release, for the stores of the output: half a microsecond more)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS));
  }
}

}  // namespace pair
}  // namespace ttc
}  // namespace q40

using PairKernel = void (*)(const q40::ttc::pair::Params, const q40::ttc::pair::Maps);

// [0] SPLIT; [1] EARLY; else 2 + 1 SiLU + 2 cut; [6] .. [8] with groups along K: SPLIT, EARLY, neither
static PairKernel pair_kernel(int which) {
  using namespace q40::ttc::pair;
  switch (which) {
    case 0: return gemm_pair_kernel<true, true, false, false>;
    case 1: return gemm_pair_kernel<true, false, false, false>;
    case 2: return gemm_pair_kernel<false, false, false, false>;
    case 3: return gemm_pair_kernel<false, false, false, true>;
    case 4: return gemm_pair_kernel<false, false, true, false>;
    case 5: return gemm_pair_kernel<false, false, true, true>;
    case 6: return gemm_pair_kernel<true, true, false, false, true>;
    case 7: return gemm_pair_kernel<true, false, false, false, true>;
    default: return gemm_pair_kernel<false, false, false, false, true>;
  }
}

// How many clusters of (2, nsplit) CTAs run at once, one CTA per SM (an answer is kept per device and split; 0, not kept,
// when the runtime cannot tell)
static int pair_max_clusters(PairKernel kern, int nsplit) {
  using namespace q40::ttc;
  static std::atomic<int> cache[16][5];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* kept = dev < 16 ? &cache[dev][nsplit] : nullptr;
  if (kept && kept->load(std::memory_order_relaxed)) return kept->load(std::memory_order_relaxed) - 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2048, nsplit, 1);
  cfg.blockDim = dim3(pair::THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM_MAX;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = nsplit;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  if (kept) kept->store(n + 1, std::memory_order_relaxed);
  return n;
}

namespace q40 {
namespace ttc {
namespace pair {

// Rows of a tile
static void tile_rows(Params& p, int npad) {
  p.npad = npad;
  p.chunks = (p.M + npad - 1) / npad;
}

// Shared memory of a launch, or 0 if it does not fit: [ring][run][rows on their way out][barriers]; ring stages, accumulators and A
// buffers.  `single`: no pair has more than one tile, of one range, and a second accumulator would be for nothing.  Else two where
// they fit tensor memory beside at least two A buffers.
// Two groups finish tiles where that is what a pair waits for: the sums of ranges of few blocks (three matrices of 512 rows x 4096 x 4096, eight
// blocks: 54.4 us with one, 52.4; 300 rows 39.0 and 34.9; but 22 blocks, x 11008 x 4096, 43.3 and 46.4), and many rows of a SiLU product
// with shared tiles (x 4096 x 11008, 100 rows 26.2 and 24.5, 128 28.8 and 26.2; 77 21.7 and 22.0).  Where there is one tile a pair, its warps
// dequantise too (10 rows x 4096 x 12288 12.1 and 11.8, x 11008 x 4096 11.6 and 11.4, 64 rows 12.7 and 12.3, 100 the same).
// `alone`: no pair has more than one tile.  Then one group, where the output rows of two leave no room for the ring (three x 4096 x 4096 in tiles of
// 176 rows: 171 rows 25.2 us, in tiles of 96 with two groups 26.7); where pairs have more, smaller tiles are the faster ones (512 rows 55.8 and 52.8)
static size_t layout(Params& p, int split, bool single, bool alone) {
  const size_t tile = (size_t)p.npad * FEATS * 4, stage = RAW_PAD + (size_t)p.npad * 64 * BLK;
  p.own = ((p.M + 3) / 4 + split - 1) / split;
  const size_t run = split > 1 ? (size_t)(split - 1) * p.own * FEATS * 16 : p.range < p.k64 ? tile : 0;
  const bool early = single && !p.silu;
  p.egroups = !single && (p.silu ? p.cut && p.npad >= 96 : 8 * p.rblk <= p.npad) ? 2 : 1;
  const auto out_bytes = [&]() { return split > 1 ? (size_t)0 : (size_t)p.egroups * 2 * 16 * OUT_LD * 2; };
  const size_t rest = 1024 /* alignment */ + (early ? BAR_BYTES<true> : BAR_BYTES<false>) + 64 /* tail */ + run;
  if (alone && rest + out_bytes() + DSETS * stage > (size_t)SMEM_MAX) p.egroups = 1;
  const size_t out = out_bytes(), fixed = rest + out;
  if (fixed + DSETS * stage > (size_t)SMEM_MAX) return 0;
  p.stages = std::min(S_MAX, (int)((SMEM_MAX - fixed) / stage));
  p.nacc = !single && 2 * p.npad + 2 * A_COLS <= TMEM_COLS ? 2 : 1;
  p.na = std::min({NA_MAX, p.stages, (TMEM_COLS - p.nacc * p.npad) / A_COLS});
  p.dsets = single && p.stages > DSETS ? GROUPS : GROUPS - p.egroups;
  const size_t off = p.stages * stage;
  p.run_off = (int)off;
  p.out_off = (int)(off + run);
  p.bar_off = (int)(off + run + out);
  // more than half of an SM's: two pairs of different launches that each got one SM's tensor memory would wait for the other's
  const size_t smem = off + fixed;
  return smem < 116 * 1024 ? 116 * 1024 : smem;
}

// k steps -> blocks; `range` k steps are summed in tensor memory
static void k_blocks(Params& p, int range) {
  p.range = range;
  p.rblk = (range + BLK - 1) / BLK;
  const int nr = (p.k64 + range - 1) / range;
  p.nblk = (nr - 1) * p.rblk + (p.k64 - (nr - 1) * range + BLK - 1) / BLK;
}

}  // namespace pair
}  // namespace ttc
}  // namespace q40

// Which launch: the one of least estimated time.  Nanoseconds on a B200, weights from HBM, launches in a row; npad = rows
// of a tile, a block = 128 k of 256 features:
//   a block           232 + npad / 4, or the MMAs' 2.2 npad (one tile per pair; 16 rows 236, 112 rows 258, 128 rows 283);
//                     165 + 1.8 npad, 2.8 npad beyond 128, while all SMs draw activations from L2 (64 rows 287, 128 rows 390, 256 rows 710)
//   a launch          3900 + 12 npad; with shared tiles 3800 + 28 npad more; with k split over the pairs of a cluster 700 more per
//                     pair, and all of it once per wave of clusters (they are not persistent); a range after the first 16 npad for its sums where the next one's MMAs do not hide it
// 10 rows x 4096 x 11008, two matrices: 16.8 us shared, 21.9 not, 29.3 split in two; 100 rows x 11008 x 4096: 15.7 split in
// three, 17.6 in two, 27.5 not; 512 rows x 4096 x 11008: 128-row tiles 41.3, 112 39.5, 176 45.4, 256 57.2: there the
// estimate, 39.9 for 176 rows and 40.4 for 112, takes the slower one.
// The launch of p's matmul (matrices, sizes and k blocks are in it) as the variant of least estimated time, if that is below beat_ns
template <typename EncodeWeights>
static int pair_run(q40::ttc::pair::Params& p, bool nk, int spans, const void* a, int64_t lda, void* workspace, size_t workspace_bytes, double beat_ns,
                    int use_pdl, void* stream, EncodeWeights encode_weights) {
  using namespace q40;
  using namespace q40::ttc;
  const int M = p.M, K = p.K, silu = p.silu;
  EncodeTiledFn encode = ttc_encode_fn();
  if (!encode) return Q40_E_UNSUPPORTED;
  if ((int64_t)spans * ((M + 63) / 64) * std::max(p.nblk, pair::MAX_PAIRS) > 0x7fffffffLL) return Q40_E_UNSUPPORTED;
  // the kernels' attributes come first: the runtime is asked how many fit with the shared memory that they allow
  static std::atomic<uint64_t> ready[9];
  auto kernel = [&](int which) -> PairKernel {
    PairKernel k = pair_kernel(which);
    if (q40_allow_smem(ready[which], (const void*)k, SMEM_MAX) == cudaSuccess) return k;
    (void)cudaGetLastError();
    return nullptr;
  };
  PairKernel plain = kernel(nk ? 8 : 2), in_clusters = kernel(nk ? 6 : 0);
  if (!plain || !in_clusters) return Q40_E_UNSUPPORTED;
  const int fit = pair_max_clusters(plain, 1) < pair::MAX_PAIRS ? pair_max_clusters(plain, 1) : pair::MAX_PAIRS;
  if (fit < 1) return Q40_E_UNSUPPORTED;

  double best = beat_ns;
  int npad = 0, split = 1, cut = 0;
  if (M <= 128) {
    const int n = (M + 15) / 16 * 16;
    const double block = std::max(232.0 + 0.25 * n, 2.21 * n), launch = 3900 + 12.0 * n;
    auto consider = [&](double ns, int sp, int ct) { if (ns < best) { best = ns; npad = n; split = sp; cut = ct; } };
    consider(launch + (double)((spans + fit - 1) / fit) * p.nblk * block, 1, 0);
    const int64_t units = (int64_t)spans * p.nblk / pair::CUT;
    if (workspace && workspace_bytes >= q40_gemm_tiled_tc_ws_bytes(M) && units * 2 * pair::CUT >= (int64_t)fit * p.nblk)
      consider(launch + 3800 + 28.0 * n + (double)spans * p.nblk / fit * block, 1, 1);
    for (int sp = 2; sp <= 4 && !silu; ++sp) {
      const int bps = (p.nblk + sp - 1) / sp, f = (sp - 1) * bps < p.nblk ? pair_max_clusters(in_clusters, sp) : 0;
      if (f > 0) consider((double)((spans + f - 1) / f) * (launch + 700.0 * (sp - 1) + bps * block), sp, 0);
    }
  } else {
    for (int n = 64; n <= pair::MAX_ROWS; n += 16) {
      const int chunks = (M + n - 1) / n;
      if (((M + chunks - 1) / chunks + 15) / 16 * 16 != n) continue;           // the same chunks with fewer rows of padding
      pair::tile_rows(p, n);
      if (pair::layout(p, 1, false, (int64_t)spans * chunks <= fit) == 0) continue;
      const double waves = (double)(((int64_t)spans * chunks + fit - 1) / fit);
      const double block = n <= 128 ? 165 + 1.8 * n : 395 + 2.8 * (n - 128);
      const int nr = (p.k64 + p.range - 1) / p.range;
      const double tile = nr > 1 ? nr * std::max(p.rblk * block + 1000, 16.5 * n) : p.nblk * block;
      const double ns = 3900 + 12.0 * n + waves * tile;
      if (ns < best) { best = ns; npad = n; }
    }
  }
  if (npad == 0) return Q40_E_UNSUPPORTED;

  pair::tile_rows(p, npad);
  p.ntiles = spans * p.chunks;                   // SiLU: as many, of half a span of both matrices
  p.cut = cut;
  if (cut) {
    p.flags = (int*)workspace;
    p.part = (float*)((char*)workspace + pair::FLAG_BYTES);
  }
  int npairs = p.ntiles;
  if (split > 1) {
    p.bps = (p.nblk + split - 1) / split;
  } else {
    const int units = cut ? p.ntiles * p.nblk / pair::CUT : p.ntiles;
    npairs = units < fit ? (units < 1 ? 1 : units) : fit;
    p.share = units / npairs;
    p.rest = units % npairs;
  }
  const bool single = split > 1 || (!cut && p.ntiles <= npairs && p.range == p.k64);
  const size_t smem = pair::layout(p, split, single, p.ntiles <= npairs);
  if (smem == 0 || smem > (size_t)SMEM_MAX) return Q40_E_UNSUPPORTED;
  PairKernel kern = split > 1 ? in_clusters : single && !silu ? kernel(nk ? 7 : 1) : nk ? plain : kernel(2 + silu + 2 * cut);
  if (!kern) return Q40_E_UNSUPPORTED;
  pair::Maps maps{};
  const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t gstride[1] = {(cuuint64_t)lda * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)p.npad / 2};
  const cuuint32_t estr[2] = {1, 1};
  if (!(nk && p.x) && ttc_encode(encode, &maps.act, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)a, gdim, gstride, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q40_E_UNSUPPORTED;
  if (!encode_weights(encode, maps)) return Q40_E_UNSUPPORTED;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * npairs, split, 1);
  cfg.blockDim = dim3(pair::THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = split;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, maps);
  if (e != cudaSuccess) return (int)e;
  return Q40_OK;
}

// The launch that q40_gemm_tiled_tc_multi and q40_gemm_tiled_tc_ws make: see q40_tc_common.cuh.  Arguments are checked.
int q40_pair_gemm(int nmat, const void* a, int64_t lda, const void* const* bw_tiled, void* const* c, const int64_t* ldc,
                  const int* n_cols, int M, int K, int ranges, int silu, void* workspace, size_t workspace_bytes, double beat_ns,
                  int* err, int use_pdl, void* stream) {
  using namespace q40;
  using namespace q40::ttc;
  pair::Params p{};
  int spans = 0;
  p.vec = 1;
  for (int i = 0; i < nmat; ++i) {
    p.c[i] = (__half*)c[i]; p.ldc[i] = ldc[i];
    p.spans[i] = n_cols[i] / SPAN;
    p.vec &= q40_aligned(c[i], 16) && ldc[i] % 8 == 0;
    spans += p.spans[i];
  }
  p.nprob = nmat; p.M = M; p.K = K; p.err = err; p.silu = silu;
  p.k64 = K / BK;
  pair::k_blocks(p, ranges > 1 ? (p.k64 + ranges - 1) / ranges : p.k64);
  return pair_run(p, false, spans, a, lda, workspace, workspace_bytes, beat_ns, use_pdl, stream, [&](EncodeTiledFn encode, pair::Maps& maps) {
    const cuuint32_t estr[2] = {1, 1};
    for (int i = 0; i < nmat; ++i) {
      const cuuint64_t wdim[2] = {STEP_BYTES / 4, (cuuint64_t)p.spans[i] * (K / 16)};
      const cuuint64_t wstride[1] = {STEP_BYTES};
      const cuuint32_t wbox[2] = {silu ? 128u : 256u, 4 * pair::BLK}, sbox[2] = {silu ? 8u : 16u, 4 * pair::BLK};
      for (int j = 0; j < 2; ++j)
        if (ttc_encode(encode, j ? &maps.s[i] : &maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)bw_tiled[i], wdim, wstride, j ? sbox : wbox,
                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
          return false;
    }
    return true;
  });
}

// Y[M, N] = X[M, K] @ deq(W)^T for W [N, K] with groups of 64 along K: see q40_gemm_nk, whose arguments are checked.  K % 128 == 0; x on 8-byte
// boundaries, rows too.  Weights may be what the launch in front writes: they are requested behind the wait for it
int q40_pair_linear(const void* x, int64_t ldx, const void* wq, const void* ws, void* y, int64_t ldy, int M, int N, int K, double beat_ns,
                    int* err, void* stream) {
  using namespace q40;
  using namespace q40::ttc;
  pair::Params p{};
  p.c[0] = (__half*)y; p.ldc[0] = ldy;
  p.spans[0] = (N + SPAN - 1) / SPAN;
  p.vec = q40_aligned(y, 16) && ldy % 8 == 0 ? 1 : q40_aligned(y, 4) && ldy % 2 == 0 ? 0 : 2;
  p.nprob = 1; p.M = M; p.K = K; p.err = err;
  p.nk_s = (const __half*)ws; p.n_cols = N;
  if (!q40_aligned(x, 16) || ldx % 8 != 0) { p.x = (const __half*)x; p.ldx = ldx; }
  p.k64 = K / BK;
  pair::k_blocks(p, p.k64);
  return pair_run(p, true, p.spans[0], x, ldx, nullptr, 0, beat_ns, 1, stream, [&](EncodeTiledFn encode, pair::Maps& maps) {
    const cuuint64_t dim[2] = {(cuuint64_t)K / 2, (cuuint64_t)N}, pitch[1] = {(cuuint64_t)K / 2};
    const cuuint32_t box[2] = {64, pair::FEATS}, estr[2] = {1, 1};
    return ttc_encode(encode, &maps.w[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)wq, dim, pitch, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  });
}

// Scratch of q40_gemm_tiled_tc_ws: flags and one slot of sums per pair (0: none is used for so many rows)
extern "C" size_t q40_gemm_tiled_tc_ws_bytes(int M) {
  using namespace q40::ttc::pair;
  if (M < 1 || M > 128) return 0;
  return (size_t)FLAG_BYTES + (size_t)MAX_PAIRS * 2 * ((M + 15) / 16 * 16) * FEATS * 4;
}
