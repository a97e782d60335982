// Status strings and ABI version of the q40b200 library.
#include "q40_common.cuh"

extern "C" int q40_abi_version(void) { return 2; }

extern "C" const char* q40_strerror(int status) {
  switch (status) {
    case Q40_OK: return "ok";
    case Q40_E_NULL: return "q40: a required pointer is NULL";
    case Q40_E_SHAPE: return "q40: a size violates a divisibility or range rule";
    case Q40_E_ALIGN: return "q40: a pointer or stride is misaligned";
    case Q40_E_WORKSPACE: return "q40: workspace missing or too small";
    case Q40_E_UNSUPPORTED: return "q40: unsupported group size, head dim or index width";
    default: break;
  }
  if (status > 0) return cudaGetErrorString((cudaError_t)status);
  return "q40: unknown status";
}

extern "C" int q40_capture_id(void* stream, uint64_t* id) {
  if (!id) return Q40_E_NULL;
  cudaStreamCaptureStatus status;
  unsigned long long of = 0;
  const cudaError_t e = cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, &of);
  if (e != cudaSuccess) return (int)e;
  *id = status == cudaStreamCaptureStatusNone ? 0 : of;
  return Q40_OK;
}

#ifdef Q40_TRACE
void* q40_trace_ptr = nullptr;
extern "C" void q40_debug_trace(void* buf) { q40_trace_ptr = buf; }
#endif

// One call per projection costs the host more than the launch when its arguments are arrays: the plain form.
extern "C" int q40_matmul_tiled(const void* bw_tiled, void* c, int64_t ldc, const void* a, int64_t lda, int M, int N,
                                int K, int max_cluster, int* err, int use_pdl, void* stream) {
  const void* none = nullptr;
  // From 9 rows on the tensor-core kernel is the faster one, or as fast (9 rows x 4096 x 4096 8.4 against 9.4 us, x 11008 x 4096
  // 13.0 against 16.7, x 4096 x 32000 21 against 31, x 1024 x 1024 4.6 against 4.5): the narrow one does two MMAs per weight fragment
  if (M > 16 || (M > 8 && err && K % 64 == 0 && N % 256 == 0 && ldc % 2 == 0 && q40_aligned(c, 4) && (max_cluster == 8 || max_cluster == 16))) {
    const int rc = q40_gemm_tiled_tc_multi(1, a, lda, &bw_tiled, &c, &ldc, &N, M, K, err, use_pdl, stream);
    if (M > 16 || rc != Q40_E_UNSUPPORTED) return rc;
  }
  return q40_gemv_tiled(0, 1, &bw_tiled, &none, &c, &N, ldc, a, lda, M, K, nullptr, nullptr, 0, 0.f, nullptr, 0,
                        nullptr, 0, max_cluster, use_pdl, stream);
}
