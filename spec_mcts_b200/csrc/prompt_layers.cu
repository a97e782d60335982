// All layers of a prompt pass enqueued by one native call.
//
// A prompt of up to 128 tokens takes the GPU 1.9 to 2.6 ms (7B geometry) and its 289 launches, call by call from Python, 2.6 ms of
// the host: 9 us each, of which 3.5 to 4.2 are the library's and the runtime's.  From here a pass takes the host 1.7 to 1.9 ms, with
// what Python looks up per layer (77 tokens: 2612 us a pass and 2375 here, 17 tokens 2640 and 2098).
#include "q40_common.cuh"

extern "C" int q40_prompt_layers(const void* const* layers, int n_layers, int S, int dim, int hidden, int H, int Hkv, float eps, void* h, void* xn,
                                 void* q, void* ao, void* o, void* g, void* f, const int32_t* pos, const void* cos_tbl, const void* sin_tbl,
                                 void* workspace, size_t workspace_bytes, int* err, int use_pdl, void* stream) {
  constexpr int D = 128, PER = Q40_PROMPT_LAYER_POINTERS;
  if (!layers || !h || !xn || !q || !ao || !o || !g || !f || !pos || !cos_tbl || !sin_tbl || !err) return Q40_E_NULL;
  if (n_layers < 0 || S < 1 || H < 1 || Hkv < 1 || H % Hkv != 0) return Q40_E_SHAPE;
  const int wq = H * D, wkv = Hkv * D;
  const int64_t ld_qkv[3] = {wq, wkv, wkv}, ld_dim[1] = {dim}, ld_h[2] = {hidden, hidden};
  const int n_qkv[3] = {wq, wkv, wkv}, n_dim[1] = {dim}, n_h[2] = {hidden, hidden};
  void* const to_o[1] = {o};
  void* const to_f[1] = {f};
  void* const to_g[2] = {g, g};
  const void* pending = nullptr;                // output of the previous sub-block, added to h by the next norm kernel
  for (int i = 0; i < n_layers; ++i) {
    const void* const* l = layers + (int64_t)i * PER;
    void *ck = (void*)l[9], *cv = (void*)l[10]; // keys and values go straight to their place in the prompt cache
    void* const to_qkv[3] = {q, ck, cv};
    int rc = q40_rmsnorm(h, pending, l[7], xn, pending ? h : nullptr, S, dim, eps, stream);
    if (!rc) rc = q40_gemm_tiled_tc_multi(3, xn, dim, l, to_qkv, ld_qkv, n_qkv, S, dim, err, use_pdl, stream);
    if (!rc) rc = q40_rope_qk(q, H, wq, ck, Hkv, wkv, pos, cos_tbl, sin_tbl, S, D, stream);
    if (!rc) rc = q40_attn_causal(q, wq, ck, wkv, cv, wkv, ao, wq, S, H, Hkv, D, stream);
    if (!rc) rc = q40_gemm_tiled_tc_multi(1, ao, wq, l + 3, to_o, ld_dim, n_dim, S, wq, err, use_pdl, stream);
    if (!rc) rc = q40_rmsnorm(h, o, l[8], xn, h, S, dim, eps, stream);
    if (!rc) rc = q40_gemm_tiled_tc_ws(2, xn, dim, l + 4, to_g, ld_h, n_h, S, dim, 1, workspace, workspace_bytes, err, use_pdl, stream);
    if (!rc) rc = q40_gemm_tiled_tc_multi(1, g, hidden, l + 6, to_f, ld_dim, n_dim, S, hidden, err, use_pdl, stream);
    if (rc) return rc;
    pending = f;
  }
  return Q40_OK;
}
