// Causal attention of the prompt pass: out[i] = softmax_{j <= i}(q_i . k_j / sqrt(D)) v_j per head, for S
// positions processed at once (hf_model_q40_kv_shared.py:324-329 builds the prompt's K/V, :499-504 the
// triangular mask, :405 calls scaled_dot_product_attention with it).
//
// One CTA per (block of 64 query positions, query head), the blocks with most keys first: the query rows are the M dimension of
// mma.m16n8k16 (16 rows per warp, A fragments kept in registers), keys and values of the head's kv head
// (grouped-query attention reads the shared kv head directly, no repeat_interleave) stream through shared
// memory in 64-key tiles (cp.async, double buffered), S = Q K^T and O += P V on the tensor cores with an
// fp32 online softmax in the log2 domain.  Only tiles that reach the diagonal are masked; tiles beyond the
// block's last row are never loaded.  Output is normalised and written as fp16.
// What bounds it: a warp's chain of MMAs and softmax, tile after tile, and the last block, which has all the keys.  512
// positions x 32 heads: 25 us with 128 rows per CTA (128 CTAs, the longest 8 tiles with two warps per SM
// sub-partition), 18.4 us with 64 (256 CTAs that share the SMs, long ones first), an
// unmasked path for the tiles before the diagonal and less arithmetic per tile (attn_tile.cuh).
#include "attn_tile.cuh"

namespace q40 {
namespace causal {

constexpr int NWARPS = 4;
constexpr int RB = NWARPS * 16;              // query rows per CTA

struct Args {
  const __half* q;    // position i, head h at q + i * ldq + h * D
  const __half* k;    // position j, kv head g at k + j * ldk + g * D
  const __half* v;
  __half* o;          // position i, head h at o + i * ldo + h * D
  int64_t ldq, ldk, ldv, ldo;
  int S, H, Hkv;
  float scale_log2;
};

// grid: H x query blocks, the last block of every head first; block: 128 threads
__global__ void __launch_bounds__(NWARPS * 32)
attn_causal_kernel(const Args a) {
  constexpr int D = ATTN_D;
  constexpr int NT = NWARPS * 32;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);     // [Q rows][stage][K tile | V tile]
  asm volatile("griddepcontrol.launch_dependents;");   // a dependent may start prefetching its weights
  asm volatile("griddepcontrol.wait;" ::: "memory");               // ... but nothing of the previous launch is read before it is done
  const int rblk = (int)((gridDim.x - 1 - blockIdx.x) / a.H), h = (int)(blockIdx.x % a.H), hk = h / (a.H / a.Hkv);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row0 = rblk * RB;
  const int k_end = min(a.S, row0 + RB);     // keys this block can see
  const int ntiles = (k_end + TILE_KEYS - 1) / TILE_KEYS;
  const uint32_t stages = sbase + RB * TILE_ROW_BYTES;

  auto load = [&](int tile, int stage) {
    const int64_t key0 = (int64_t)tile * TILE_KEYS;
    const uint32_t kdst = stages + stage * 2 * TILE_BYTES;
    load_tile<NT>(kdst, kdst + TILE_BYTES, a.k + key0 * a.ldk + hk * D, a.v + key0 * a.ldv + hk * D, a.ldk, a.ldv, k_end - tile * TILE_KEYS, tid);
  };
  // ---- Q rows -> shared (swizzled) -> A fragments in registers, with the first tile on its way ----
  for (int idx = tid; idx < RB * 16; idx += NT) {
    const int r = idx >> 4, ch = idx & 15;
    const int qi = row0 + r;
    const bool ok = qi < a.S;
    cp_async16(sbase + tile_off(r, ch), a.q + (int64_t)(ok ? qi : 0) * a.ldq + h * D + ch * 8, ok);
  }
  cp_async_commit();
  load(0, 0);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  WarpRows w;
  w.init();
  w.load_q(sbase, warp * 16, lane);

  // query positions of this lane's two rows
  const int qi0 = row0 + warp * 16 + g, qi1 = qi0 + 8;
  const int warp_first = row0 + warp * 16, warp_last = warp_first + 15;
  for (int tile = 0; tile < ntiles; ++tile) {
    const int stage = tile & 1;
    if (tile + 1 < ntiles) load(tile + 1, stage ^ 1);
    cp_async_commit();
    cp_async_wait<1>();   // the tile for this iteration has landed
    __syncthreads();
    const int key0 = tile * TILE_KEYS;
    const uint32_t kt = stages + stage * 2 * TILE_BYTES, vt = kt + TILE_BYTES;
    // a warp whose rows all lie before this tile has nothing to add (the barriers are still shared); one whose rows all
    // lie behind it masks nothing
    if (key0 + TILE_KEYS <= min(warp_first + 1, a.S)) w.step<false>(kt, vt, a.scale_log2, 0, 0, lane);
    else if (key0 <= warp_last) w.step<true>(kt, vt, a.scale_log2, min(qi0 + 1, a.S) - key0, min(qi1 + 1, a.S) - key0, lane);
    __syncthreads();  // all warps are done with this stage before it is refilled
  }
  cp_async_wait<0>();

  // ---- normalise and write rows g and g+8 ----
  w.finish();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int qi = r ? qi1 : qi0;
    if (qi >= a.S) continue;
    const float inv = w.l[r] > 0.f ? 1.f / w.l[r] : 0.f;
    __half* dst = a.o + (int64_t)qi * a.ldo + h * D;
#pragma unroll
    for (int dt = 0; dt < 16; ++dt)
      *reinterpret_cast<__half2*>(dst + dt * 8 + 2 * t) = __floats2half2_rn(w.o[dt][2 * r] * inv, w.o[dt][2 * r + 1] * inv);
  }
}

}  // namespace causal
}  // namespace q40

// o[S, H*128] = causal attention of q[S, H*128] over k, v[S, Hkv*128] (position-major rows with the given
// row strides in elements; H % Hkv == 0).  Replaces the masked scaled_dot_product_attention of the
// reference's prompt pass (hf_model_q40_kv_shared.py:375-405, mask :499-504).
extern "C" int q40_attn_causal(const void* q, int64_t ldq, const void* k, int64_t ldk, const void* v, int64_t ldv,
                               void* o, int64_t ldo, int S, int H, int Hkv, int D, void* stream) {
  using namespace q40;
  using namespace q40::causal;
  if (!q || !k || !v || !o) return Q40_E_NULL;
  if (D != ATTN_D) return Q40_E_UNSUPPORTED;
  if (S < 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0) return Q40_E_SHAPE;
  if (ldq < (int64_t)H * D || ldo < (int64_t)H * D || ldk < (int64_t)Hkv * D || ldv < (int64_t)Hkv * D)
    return Q40_E_SHAPE;
  if (ldq % 8 != 0 || ldk % 8 != 0 || ldv % 8 != 0 || ldo % 2 != 0) return Q40_E_ALIGN;
  if (!q40_aligned(q, 16) || !q40_aligned(k, 16) || !q40_aligned(v, 16) || !q40_aligned(o, 4)) return Q40_E_ALIGN;
  if (S == 0) return Q40_OK;
  Args a{};
  a.q = (const __half*)q; a.k = (const __half*)k; a.v = (const __half*)v; a.o = (__half*)o;
  a.ldq = ldq; a.ldk = ldk; a.ldv = ldv; a.ldo = ldo; a.S = S; a.H = H; a.Hkv = Hkv;
  a.scale_log2 = attn_scale_log2(D);
  const size_t smem = RB * TILE_ROW_BYTES + 4 * TILE_BYTES;      // the Q rows, two stages of K and V
  static std::atomic<uint64_t> ready;
  cudaError_t e = q40_allow_smem(ready, (const void*)attn_causal_kernel, (int)smem);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return Q40_E_UNSUPPORTED; }
  const int64_t blocks = (int64_t)H * ((S + RB - 1) / RB);
  if (blocks > 0x7fffffffLL) return Q40_E_SHAPE;
  e = q40_launch_pdl(attn_causal_kernel, dim3((unsigned)blocks), dim3(NWARPS * 32), smem, (cudaStream_t)stream, a);
  if (e != cudaSuccess) return (int)e;
  return Q40_OK;
}
