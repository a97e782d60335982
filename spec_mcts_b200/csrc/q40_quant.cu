// Q4_0 packer and unpacker (bit-exact with the reference's torch functions).
//
// Format, restated from the reference's quantize_q40 / dequantize_q40
// (triton_kernels.py:12-56): the tensor is read row-major as groups of G elements;
// scale[g] = fp16(absmax/7) ; code = int8(rint(fp16(w/scale))) ; groups (2j, 2j+1) share a
// packed row of G bytes: byte i = code[2j][i] << 4 | code[2j+1][i] & 0xF.
//
// Both kernels are streaming kernels (HBM-bound): one thread handles 8 consecutive elements of an even
// group and the matching 8 of the odd group, so that every load and store of values is 16 bytes per lane
// and contiguous over the lanes of a pair, and it keeps ITEMS such pieces in flight.
#include "q40_common.cuh"

namespace q40 {

constexpr int QUANT_THREADS = 256;
constexpr int QUANT_ITEMS = 2;     // pieces per thread, QUANT_THREADS apart

// ---------------------------------------------------------------------------------------
// quantise: rows of `row_len` elements; a "pair" is 2*G consecutive elements of a row.
// G/8 threads cooperate on one pair (absmax via shuffles inside that lane group).  FLAT: a row is one
// pair (contiguous input and output), which saves the index division.
// 4096 x 11008, group 64: 54.5 us with two IEEE divisions per byte and one piece per thread (its
// arithmetic was the bound); packing and expanding that matrix took 80.1 us together, now 42.5 us = 4.8 TB/s.
// ---------------------------------------------------------------------------------------
template <int G, bool FLAT>
__global__ void __launch_bounds__(QUANT_THREADS)
quantize_rows_kernel(const __half* __restrict__ w, int64_t w_row_stride, uint8_t* __restrict__ q,
                     int64_t q_row_stride, __half* __restrict__ s, int64_t s_row_stride,
                     int64_t n_rows, int pairs_per_row) {
  asm volatile("griddepcontrol.wait;" ::: "memory");   // see launch_stream
  constexpr int TPP = G / 8;  // threads per pair
  const int64_t total_pairs = n_rows * (int64_t)pairs_per_row;
  const int sub = threadIdx.x % TPP;
  uint4 e[QUANT_ITEMS], o[QUANT_ITEMS];
  int64_t row[QUANT_ITEMS];
  int pj[QUANT_ITEMS];
  bool live[QUANT_ITEMS];
#pragma unroll
  for (int it = 0; it < QUANT_ITEMS; ++it) {
    const int64_t pair = ((int64_t)blockIdx.x * QUANT_ITEMS + it) * (QUANT_THREADS / TPP) + threadIdx.x / TPP;
    live[it] = pair < total_pairs;
    row[it] = FLAT ? pair : live[it] ? pair / pairs_per_row : 0;
    pj[it] = FLAT ? 0 : (int)(pair - row[it] * pairs_per_row);
    e[it] = o[it] = make_uint4(0, 0, 0, 0);
    if (live[it]) {
      const __half* src = w + row[it] * w_row_stride + (int64_t)pj[it] * 2 * G + sub * 8;
      e[it] = *reinterpret_cast<const uint4*>(src);      // 8 elements of the even group
      o[it] = *reinterpret_cast<const uint4*>(src + G);  // the same positions of the odd group
    }
  }
#pragma unroll
  for (int it = 0; it < QUANT_ITEMS; ++it) {
    const uint32_t ew[4] = {e[it].x, e[it].y, e[it].z, e[it].w}, ow[4] = {o[it].x, o[it].y, o[it].z, o[it].w};
    __half2 m = quant_max(ew, ow);      // (even, odd) maxima in one word for the shuffles
#pragma unroll
    for (int off = TPP / 2; off > 0; off >>= 1)
      m = __hmax2(m, u32_as_h2(__shfl_xor_sync(0xffffffffu, h2_as_u32(m), off)));
    __half2 sc;
    const uint2 out = quant_codes(ew, ow, m, sc);
    if (live[it]) {
      uint8_t* dst = q + row[it] * q_row_stride + (int64_t)pj[it] * G + sub * 8;
      *reinterpret_cast<uint2*>(dst) = out;
      if (sub == 0) {
        __half* sd = s + row[it] * s_row_stride + (int64_t)pj[it] * 2;
        *reinterpret_cast<__half2*>(sd) = sc;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// dequantise: a piece is 8 packed bytes -> 8 values of the even group + 8 of the odd, so that the lanes of
// a packed row write whole 32-byte sectors with every store (16 bytes per piece left each store with half
// of its sectors: 25.3 us for 4096 x 11008, group 64).
// ---------------------------------------------------------------------------------------
template <int G>
__global__ void __launch_bounds__(QUANT_THREADS)
dequantize_kernel(const uint8_t* __restrict__ q, const __half* __restrict__ s,
                  __half* __restrict__ out, int64_t n_bytes) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint2 p[QUANT_ITEMS];
  __half2 sc[QUANT_ITEMS];
#pragma unroll
  for (int it = 0; it < QUANT_ITEMS; ++it) {
    const int64_t byte0 = (((int64_t)blockIdx.x * QUANT_ITEMS + it) * QUANT_THREADS + threadIdx.x) * 8;
    p[it] = make_uint2(0, 0);
    sc[it] = u32_as_h2(0u);
    if (byte0 < n_bytes) {
      p[it] = *reinterpret_cast<const uint2*>(q + byte0);
      sc[it] = *reinterpret_cast<const __half2*>(s + 2 * (byte0 / G));
    }
  }
#pragma unroll
  for (int it = 0; it < QUANT_ITEMS; ++it) {
    const int64_t byte0 = (((int64_t)blockIdx.x * QUANT_ITEMS + it) * QUANT_THREADS + threadIdx.x) * 8;
    if (byte0 >= n_bytes) return;
    const int64_t prow = byte0 / G;      // packed row = pair index
    const int i0 = (int)(byte0 % G);
    const __half2 s_hi = __half2half2(__low2half(sc[it]));
    const __half2 s_lo = __half2half2(__high2half(sc[it]));
    const uint32_t wds[2] = {p[it].x, p[it].y};
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int wi = 0; wi < 2; ++wi) {
      const uint32_t w0 = wds[wi];       // bytes b0 b1 b2 b3
      const uint32_t w1 = w0 >> 8;       // bytes b1 b2 b3 -
      // half2 results hold (b0,b2) and (b1,b3); put them back in byte order with prmt
      const __half2 l02 = __hmul2(codes_lo_to_h2(w0), s_lo);
      const __half2 l13 = __hmul2(codes_lo_to_h2(w1), s_lo);
      const __half2 h02 = __hmul2(codes_hi_to_h2(w0), s_hi);
      const __half2 h13 = __hmul2(codes_hi_to_h2(w1), s_hi);
      lo[wi * 2 + 0] = prmt(h2_as_u32(l02), h2_as_u32(l13), 0x5410);  // (b0, b1)
      lo[wi * 2 + 1] = prmt(h2_as_u32(l02), h2_as_u32(l13), 0x7632);  // (b2, b3)
      hi[wi * 2 + 0] = prmt(h2_as_u32(h02), h2_as_u32(h13), 0x5410);
      hi[wi * 2 + 1] = prmt(h2_as_u32(h02), h2_as_u32(h13), 0x7632);
    }
    __half* oe = out + prow * 2 * G + i0;  // even group; the odd group is G further
    *reinterpret_cast<uint4*>(oe) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(oe + G) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

}  // namespace q40

// Launched while the launch in front drains: pack and expand of 4096 x 11008 in turn 39.6 us, with plain launches 42.7 (4096 x
// 4096 in a graph: 14.5 and 15.5).  Neither kernel lets the
// next one start early: a matmul behind it would read weights that are still being written.
template <typename... KArgs, typename... Args>
static int launch_stream(void (*kern)(KArgs...), int64_t grid, cudaStream_t st, Args... args) {
  return (int)q40_launch_pdl(kern, dim3((unsigned)grid), dim3(q40::QUANT_THREADS), 0, st, args...);
}

extern "C" int q40_quantize_rows(const void* w, int64_t w_row_stride, void* q, int64_t q_row_stride,
                                 void* s, int64_t s_row_stride, int64_t n_rows, int row_len,
                                 int group, void* stream) {
  if (!w || !q || !s) return Q40_E_NULL;
  if (group != 64 && group != 32) return Q40_E_UNSUPPORTED;
  if (n_rows < 0 || row_len < 0 || row_len % (2 * group) != 0) return Q40_E_SHAPE;
  if (n_rows == 0 || row_len == 0) return Q40_OK;
  if (!q40_aligned(w, 16) || !q40_aligned(q, 8) || !q40_aligned(s, 4)) return Q40_E_ALIGN;
  if (w_row_stride % 8 != 0 || q_row_stride % 8 != 0 || s_row_stride % 2 != 0) return Q40_E_ALIGN;
  const int pairs_per_row = row_len / (2 * group);
  const int64_t threads = n_rows * (int64_t)pairs_per_row * (group / 8);
  const int per_block = q40::QUANT_THREADS * q40::QUANT_ITEMS;
  const int64_t grid = (threads + per_block - 1) / per_block;
  if (grid > 0x7fffffffLL) return Q40_E_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  auto kern = group == 64 ? (pairs_per_row == 1 ? q40::quantize_rows_kernel<64, true> : q40::quantize_rows_kernel<64, false>)
                          : (pairs_per_row == 1 ? q40::quantize_rows_kernel<32, true> : q40::quantize_rows_kernel<32, false>);
  return launch_stream(kern, grid, st, (const __half*)w, w_row_stride, (uint8_t*)q, q_row_stride, (__half*)s, s_row_stride,
                       n_rows, pairs_per_row);
}

extern "C" int q40_quantize(const void* w, void* q, void* s, int64_t n, int group, void* stream) {
  if (group != 64 && group != 32) return Q40_E_UNSUPPORTED;
  if (n < 0 || n % (2 * group) != 0) return Q40_E_SHAPE;
  // one "row" per pair of groups keeps every index within int range
  return q40_quantize_rows(w, 2 * group, q, group, s, 2, n / (2 * group), 2 * group, group, stream);
}

extern "C" int q40_dequantize(const void* q, const void* s, void* out, int64_t n, int group,
                              void* stream) {
  if (!q || !s || !out) return Q40_E_NULL;
  if (group != 64 && group != 32) return Q40_E_UNSUPPORTED;
  if (n < 0 || n % (2 * group) != 0) return Q40_E_SHAPE;
  if (n == 0) return Q40_OK;
  if (!q40_aligned(q, 16) || !q40_aligned(out, 16) || !q40_aligned(s, 4)) return Q40_E_ALIGN;
  const int64_t n_bytes = n / 2;
  const int64_t threads = n_bytes / 8;
  const int per_block = q40::QUANT_THREADS * q40::QUANT_ITEMS;
  const int64_t grid = (threads + per_block - 1) / per_block;
  if (grid > 0x7fffffffLL) return Q40_E_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  auto kern = group == 64 ? q40::dequantize_kernel<64> : q40::dequantize_kernel<32>;
  return launch_stream(kern, grid, st, (const uint8_t*)q, (const __half*)s, (__half*)out, n_bytes);
}
