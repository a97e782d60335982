// Element-wise pieces of a decode step, with the reference model's rounding points
// (hf_model_q40_kv_shared.py:123-134 RMSNorm, :166-203 rotary embedding, :434 SiLU-mul,
// :463-466 residual adds).  All HBM/L2-bound and tiny at decode batch sizes.
#include "q40_common.cuh"

namespace q40 {

// The same sums in the same order as rmsnorm_kernel below, for rows of up to NV vectors of eight per thread: a row stays in
// registers and all of it is requested at once, with its weights: one trip to L2 instead of one per vector.  4096 wide, what
// a pass waits for it: 10 rows 2.8 and 3.7 us before, 1.8 and 1.7 now; 512 rows 6.8 and 5.2.
template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_reg_kernel(const __half* __restrict__ x, const __half* __restrict__ residual, const __half* __restrict__ w,
                   __half* __restrict__ y, __half* __restrict__ h_out, int dim, float eps) {
  __shared__ float red[8];
  const int tid = threadIdx.x;
  uint4 wv[NV], v[NV], u[NV];
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");     // the weights, too, may be the previous launch's
  const int64_t at = (int64_t)blockIdx.x * dim + tid * 8;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const bool in = (n * 256 + tid) * 8 < dim;
    v[n] = in ? *reinterpret_cast<const uint4*>(x + at + n * 2048) : make_uint4(0, 0, 0, 0);
    if (residual) u[n] = in ? *reinterpret_cast<const uint4*>(residual + at + n * 2048) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int i = (n * 256 + tid) * 8;
    wv[n] = i < dim ? *reinterpret_cast<const uint4*>(w + i) : make_uint4(0, 0, 0, 0);
  }
  float ss = 0.f;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    __half2* vh = reinterpret_cast<__half2*>(&v[n]);
    const __half2* uh = reinterpret_cast<const __half2*>(&u[n]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (residual) vh[j] = __hadd2(vh[j], uh[j]);           // fp16 add, one rounding
      const float2 f = __half22float2(vh[j]);
      ss = fmaf(f.x, f.x, ss);
      ss = fmaf(f.y, f.y, ss);
    }
  }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)dim + eps);
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    if ((n * 256 + tid) * 8 >= dim) break;
    if (residual && h_out) *reinterpret_cast<uint4*>(h_out + at + n * 2048) = v[n];
    __half2* vh = reinterpret_cast<__half2*>(&v[n]);
    const __half2* wh = reinterpret_cast<const __half2*>(&wv[n]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(vh[j]);
      const __half2 nn = __floats2half2_rn(f.x * inv, f.y * inv);   // round to fp16 first
      vh[j] = __hmul2(nn, wh[j]);                                   // then * weight in fp16
    }
    *reinterpret_cast<uint4*>(y + at + n * 2048) = v[n];
  }
}

// Rows of any width.  One CTA per row.  h = fp16(x + residual) (optional), y = fp16(fp16(h32 * rsqrt(mean(h32^2)+eps)) * w)
__global__ void __launch_bounds__(256)
rmsnorm_kernel(const __half* __restrict__ x, const __half* __restrict__ residual,
               const __half* __restrict__ w, __half* __restrict__ y, __half* __restrict__ h_out,
               int dim, float eps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* row = reinterpret_cast<__half*>(smem_raw);  // [dim]
  __shared__ float red[8];
  asm volatile("griddepcontrol.launch_dependents;");   // a dependent may start prefetching its weights
  asm volatile("griddepcontrol.wait;" ::: "memory");               // ... but nothing of the previous launch is read before it is done
  const int r = blockIdx.x, tid = threadIdx.x;
  const __half* xr = x + (int64_t)r * dim;
  const __half* rr = residual ? residual + (int64_t)r * dim : nullptr;
  float ss = 0.f;
  for (int i = tid * 8; i < dim; i += blockDim.x * 8) {
    uint4 v = *reinterpret_cast<const uint4*>(xr + i);
    __half2* vh = reinterpret_cast<__half2*>(&v);
    if (rr) {
      uint4 u = *reinterpret_cast<const uint4*>(rr + i);
      const __half2* uh = reinterpret_cast<const __half2*>(&u);
#pragma unroll
      for (int j = 0; j < 4; ++j) vh[j] = __hadd2(vh[j], uh[j]);  // fp16 add, one rounding
      if (h_out) *reinterpret_cast<uint4*>(h_out + (int64_t)r * dim + i) = v;
    }
    *reinterpret_cast<uint4*>(row + i) = v;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(vh[j]);
      ss = fmaf(f.x, f.x, ss);
      ss = fmaf(f.y, f.y, ss);
    }
  }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)dim + eps);
  for (int i = tid * 8; i < dim; i += blockDim.x * 8) {
    uint4 v = *reinterpret_cast<const uint4*>(row + i);
    const uint4 wv = *reinterpret_cast<const uint4*>(w + i);
    __half2* vh = reinterpret_cast<__half2*>(&v);
    const __half2* wh = reinterpret_cast<const __half2*>(&wv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(vh[j]);
      const __half2 n = __floats2half2_rn(f.x * inv, f.y * inv);  // round to fp16 first
      vh[j] = __hmul2(n, wh[j]);                                   // then * weight in fp16
    }
    *reinterpret_cast<uint4*>(y + (int64_t)r * dim + i) = v;
  }
}

// One thread per (row, head, d < D/2): handles the pair (d, d + D/2).
__global__ void __launch_bounds__(256)
rope_kernel(__half* __restrict__ x, const int32_t* __restrict__ pos, const __half* __restrict__ cos_tbl,
            const __half* __restrict__ sin_tbl, int rows, int n_heads, int D, int64_t row_stride) {
  const int half_d = D / 2;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = (int64_t)rows * n_heads * half_d;
  if (idx >= total) return;
  const int d = (int)(idx % half_d);
  const int h = (int)((idx / half_d) % n_heads);
  const int r = (int)(idx / ((int64_t)half_d * n_heads));
  const int p = pos[r];
  const __half c = cos_tbl[(int64_t)p * half_d + d];
  const __half s = sin_tbl[(int64_t)p * half_d + d];
  __half* px = x + (int64_t)r * row_stride + (int64_t)h * D + d;
  const __half x1 = px[0], x2 = px[half_d];
  // q*cos + rotate_half(q)*sin, every operation rounded to fp16 (the _rn forms are never
  // contracted into a fused multiply-add)
  px[0] = __hadd_rn(__hmul_rn(x1, c), __hmul_rn(__hneg(x2), s));
  px[half_d] = __hadd_rn(__hmul_rn(x2, c), __hmul_rn(x1, s));
}

// One of the tensors that a launch rotates
struct RopeTensor {
  __half* x;
  int64_t row_stride;
  int rows, heads;
  unsigned blocks;         // of 256 threads
};

// The same for rows, heads and tables that are 16-byte aligned: a thread turns eight neighbouring pairs
// with 16-byte loads and stores (512 rows x 32 heads of 128: 9.4 us one pair per thread).  Queries and keys of a prompt
// pass go in one launch: 512 rows 4.3 us (4.1 and 3.1 in two), 77 rows 2.4 (2.7 and 2.2).
__global__ void __launch_bounds__(256)
rope_vec_kernel(RopeTensor t0, RopeTensor t1, const int32_t* __restrict__ pos, const __half* __restrict__ cos_tbl,
                const __half* __restrict__ sin_tbl, int half_d) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool second = blockIdx.x >= t0.blocks;
  const RopeTensor& t = second ? t1 : t0;
  const int per_row = t.heads * (half_d / 8);
  const int64_t idx = (int64_t)(blockIdx.x - (second ? t0.blocks : 0)) * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)t.rows * per_row) return;
  const int r = (int)(idx / per_row), i = (int)(idx - (int64_t)r * per_row);
  const int h = i / (half_d / 8), d = (i % (half_d / 8)) * 8;
  const int64_t tb = (int64_t)pos[r] * half_d + d;
  const uint4 c = *reinterpret_cast<const uint4*>(cos_tbl + tb), s = *reinterpret_cast<const uint4*>(sin_tbl + tb);
  __half* px = t.x + (int64_t)r * t.row_stride + (int64_t)h * 2 * half_d + d;
  uint4 lo = *reinterpret_cast<const uint4*>(px), hi = *reinterpret_cast<const uint4*>(px + half_d);
  const __half2 *ch = reinterpret_cast<const __half2*>(&c), *sh = reinterpret_cast<const __half2*>(&s);
  __half2 *l2 = reinterpret_cast<__half2*>(&lo), *h2 = reinterpret_cast<__half2*>(&hi);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2 x1 = l2[j], x2 = h2[j];
    l2[j] = __hadd2_rn(__hmul2_rn(x1, ch[j]), __hmul2_rn(__hneg2(x2), sh[j]));
    h2[j] = __hadd2_rn(__hmul2_rn(x2, ch[j]), __hmul2_rn(x1, sh[j]));
  }
  *reinterpret_cast<uint4*>(px) = lo;
  *reinterpret_cast<uint4*>(px + half_d) = hi;
}

__global__ void __launch_bounds__(256)
silu_mul_kernel(const __half* __restrict__ a, const __half* __restrict__ b, __half* __restrict__ y,
                int64_t n) {
  asm volatile("griddepcontrol.launch_dependents;");   // a dependent may start prefetching its weights
  asm volatile("griddepcontrol.wait;" ::: "memory");               // ... but nothing of the previous launch is read before it is done
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  if (i + 8 <= n) {
    uint4 av = *reinterpret_cast<const uint4*>(a + i);
    const uint4 bv = *reinterpret_cast<const uint4*>(b + i);
    __half2* ah = reinterpret_cast<__half2*>(&av);
    const __half2* bh = reinterpret_cast<const __half2*>(&bv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(ah[j]);
      const __half2 s = __floats2half2_rn(f.x / (1.0f + expf(-f.x)), f.y / (1.0f + expf(-f.y)));
      ah[j] = __hmul2(s, bh[j]);
    }
    *reinterpret_cast<uint4*>(y + i) = av;
  } else {
    for (int64_t j = i; j < n; ++j) {
      const float f = __half2float(a[j]);
      y[j] = __hmul(__float2half_rn(f / (1.0f + expf(-f))), b[j]);
    }
  }
}

// One CTA per row: h[r] = emb[token[r]] and the row's sum of squares in ss[r][0] (ss[r][1..] = 0),
// the form in which the fused decode matmuls expect it.
__global__ void __launch_bounds__(256)
embed_rows_kernel(const __half* __restrict__ emb, const int64_t* __restrict__ tokens, __half* __restrict__ h,
                  float* __restrict__ ss, int ss_count, int dim, int vocab) {
  __shared__ float red[8];
  asm volatile("griddepcontrol.launch_dependents;");
  const int r = blockIdx.x, tid = threadIdx.x;
  int64_t tok = tokens[r];
  tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
  const __half* src = emb + tok * dim;
  float s = 0.f;
  for (int i = tid * 8; i < dim; i += blockDim.x * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(src + i);
    *reinterpret_cast<uint4*>(h + (int64_t)r * dim + i) = v;
    const __half2* vh = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(vh[j]);
      s = fmaf(f.x, f.x, s);
      s = fmaf(f.y, f.y, s);
    }
  }
  s = warp_sum(s);
  if ((tid & 31) == 0) red[tid >> 5] = s;
  __syncthreads();
  for (int i = tid; i < ss_count; i += blockDim.x) {
    float tot = 0.f;
    if (i == 0)
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    ss[(int64_t)r * ss_count + i] = tot;
  }
}

}  // namespace q40

extern "C" int q40_embed_rows(const void* emb, const int64_t* tokens, void* h, float* ss, int ss_count,
                              int rows, int dim, int vocab, void* stream) {
  if (!emb || !tokens || !h || !ss) return Q40_E_NULL;
  if (rows < 0 || dim <= 0 || dim % 8 != 0 || vocab <= 0 || ss_count < 1) return Q40_E_SHAPE;
  if (rows == 0) return Q40_OK;
  if (!q40_aligned(emb, 16) || !q40_aligned(h, 16)) return Q40_E_ALIGN;
  q40::embed_rows_kernel<<<rows, 256, 0, (cudaStream_t)stream>>>((const __half*)emb, tokens, (__half*)h, ss,
                                                              ss_count, dim, vocab);
  Q40_LAUNCH_CHECK();
  return Q40_OK;
}

extern "C" int q40_rmsnorm(const void* x, const void* residual, const void* w, void* y, void* h_out,
                           int rows, int dim, float eps, void* stream) {
  if (!x || !w || !y) return Q40_E_NULL;
  if (rows < 0 || dim <= 0 || dim % 8 != 0 || dim > 65536) return Q40_E_SHAPE;
  if (rows == 0) return Q40_OK;
  if (!q40_aligned(x, 16) || !q40_aligned(w, 16) || !q40_aligned(y, 16) ||
      (residual && !q40_aligned(residual, 16)) || (h_out && !q40_aligned(h_out, 16)))
    return Q40_E_ALIGN;
  // up to four vectors a thread in registers (beyond, what a thread holds no longer leaves room for eight CTAs on an SM)
  auto reg = dim <= 2048 ? q40::rmsnorm_reg_kernel<1> : dim <= 4096 ? q40::rmsnorm_reg_kernel<2> : q40::rmsnorm_reg_kernel<4>;
  if (dim <= 8192)
    return (int)q40_launch_pdl(reg, dim3(rows), dim3(256), 0, (cudaStream_t)stream, (const __half*)x, (const __half*)residual,
                               (const __half*)w, (__half*)y, (__half*)h_out, dim, eps);
  const size_t smem = (size_t)dim * 2;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(q40::rmsnorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  const cudaError_t e2 = q40_launch_pdl(q40::rmsnorm_kernel, dim3(rows), dim3(256), smem, (cudaStream_t)stream,
                                        (const __half*)x, (const __half*)residual, (const __half*)w, (__half*)y,
                                        (__half*)h_out, dim, eps);
  if (e2 != cudaSuccess) return (int)e2;
  return Q40_OK;
}

extern "C" int q40_rope(void* x, const int32_t* pos, const void* cos_tbl, const void* sin_tbl, int rows,
                        int n_heads, int D, int64_t row_stride, void* stream) {
  if (!x || !pos || !cos_tbl || !sin_tbl) return Q40_E_NULL;
  if (rows < 0 || n_heads <= 0 || D <= 0 || D % 2 != 0 || row_stride < (int64_t)n_heads * D)
    return Q40_E_SHAPE;
  if (rows == 0) return Q40_OK;
  if (D % 16 == 0 && row_stride % 8 == 0 && q40_aligned(x, 16) && q40_aligned(cos_tbl, 16) && q40_aligned(sin_tbl, 16)) {
    const int64_t blocks = ((int64_t)rows * n_heads * (D / 16) + 255) / 256;
    if (blocks > 0x7fffffffLL) return Q40_E_SHAPE;
    const q40::RopeTensor t{(__half*)x, row_stride, rows, n_heads, (unsigned)blocks};
    return (int)q40_launch_pdl(q40::rope_vec_kernel, dim3(t.blocks), dim3(256), 0, (cudaStream_t)stream, t, t, pos,
                               (const __half*)cos_tbl, (const __half*)sin_tbl, D / 2);
  }
  const int64_t total = (int64_t)rows * n_heads * (D / 2);
  const int64_t grid = (total + 255) / 256;
  if (grid > 0x7fffffffLL) return Q40_E_SHAPE;
  q40::rope_kernel<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(
      (__half*)x, pos, (const __half*)cos_tbl, (const __half*)sin_tbl, rows, n_heads, D, row_stride);
  Q40_LAUNCH_CHECK();
  return Q40_OK;
}

extern "C" int q40_rope_qk(void* q, int q_heads, int64_t q_stride, void* k, int k_heads, int64_t k_stride, const int32_t* pos,
                           const void* cos_tbl, const void* sin_tbl, int rows, int D, void* stream) {
  if (!q || !k || !pos || !cos_tbl || !sin_tbl) return Q40_E_NULL;
  if (rows < 0 || q_heads <= 0 || k_heads <= 0 || D <= 0 || D % 2 != 0 || q_stride < (int64_t)q_heads * D ||
      k_stride < (int64_t)k_heads * D)
    return Q40_E_SHAPE;
  if (rows == 0) return Q40_OK;
  const int64_t qb = ((int64_t)rows * q_heads * (D / 16) + 255) / 256, kb = ((int64_t)rows * k_heads * (D / 16) + 255) / 256;
  if (D % 16 != 0 || q_stride % 8 != 0 || k_stride % 8 != 0 || !q40_aligned(q, 16) || !q40_aligned(k, 16) ||
      !q40_aligned(cos_tbl, 16) || !q40_aligned(sin_tbl, 16) || qb + kb > 0x7fffffffLL) {
    const int rc = q40_rope(q, pos, cos_tbl, sin_tbl, rows, q_heads, D, q_stride, stream);
    return rc ? rc : q40_rope(k, pos, cos_tbl, sin_tbl, rows, k_heads, D, k_stride, stream);
  }
  const q40::RopeTensor tq{(__half*)q, q_stride, rows, q_heads, (unsigned)qb}, tk{(__half*)k, k_stride, rows, k_heads, (unsigned)kb};
  return (int)q40_launch_pdl(q40::rope_vec_kernel, dim3((unsigned)(qb + kb)), dim3(256), 0, (cudaStream_t)stream, tq, tk, pos,
                             (const __half*)cos_tbl, (const __half*)sin_tbl, D / 2);
}

extern "C" int q40_silu_mul(const void* a, const void* b, void* y, int64_t n, void* stream) {
  if (!a || !b || !y) return Q40_E_NULL;
  if (n < 0) return Q40_E_SHAPE;
  if (n == 0) return Q40_OK;
  if (!q40_aligned(a, 16) || !q40_aligned(b, 16) || !q40_aligned(y, 16)) return Q40_E_ALIGN;
  const int64_t threads = (n + 7) / 8;
  const int64_t grid = (threads + 255) / 256;
  if (grid > 0x7fffffffLL) return Q40_E_SHAPE;
  const cudaError_t e = q40_launch_pdl(q40::silu_mul_kernel, dim3((unsigned)grid), dim3(256), 0, (cudaStream_t)stream,
                                       (const __half*)a, (const __half*)b, (__half*)y, n);
  if (e != cudaSuccess) return (int)e;
  return Q40_OK;
}
