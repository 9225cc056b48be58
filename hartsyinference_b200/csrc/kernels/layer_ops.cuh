// Entry points that the library's own layer loop (dense_layers.cu) calls across files. Each defining file includes this, so the compiler
// holds a declaration and its definition together: with C linkage a changed parameter list would link all the same.
#pragma once
#include "common.cuh"

// attention.cu
B200_API int b200_attn_prefill(const void* q, const void* k, const void* v, void* out, const int* block_table, const int* kv_lens,
                               const int* cu_q, const int* cu_kv, int seqs, int max_q_len, int q_len_single, int kv_len_single, int hq,
                               int hkv, int d, int page, int max_pages, int paged, int causal, int window, float scale, float softcap,
                               cudaStream_t stream);

// attention_pf.cu
B200_API int b200_attn_prefill_tc(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table,
                                  const int* kv_lens, const int* cu_q, int seqs, int total_q, int max_q_len, int hq, int hkv, int page,
                                  int max_pages, long long pages, int max_kv_len, float scale, void* status, cudaStream_t stream);

// fused_ops.cu
B200_API int b200_norm(const void* x, const void* residual, void* residual_out, const void* weight, const void* bias, const void* shift,
                       const void* scale, void* out, void* out_fp8, float* out_scale, int rows, int dim, int rows_per_batch,
                       int mod_stride, float eps, int layernorm, int weight_plus_one, int sf_tile_rows, const float* part_ws,
                       int part_splits, int part_bn, cudaStream_t stream);
B200_API int b200_rope_kv(const void* qkv, void* q_out, void* k_cache, void* v_cache, void* k_out, void* v_out, const int* positions,
                          const long long* slot_mapping, const void* q_norm_w, const void* k_norm_w, const float* inv_freq, int tokens,
                          int hq, int hkv, int d, int rot, int style, int page, float theta, float eps, const float* part_ws,
                          int part_splits, int part_bn, const void* part_bias, cudaStream_t stream);
B200_API int b200_glu(const void* in, void* out, void* out_fp8, float* out_scale, int rows, int f, int act, int sf_tile_rows,
                      const float* part_ws, int part_splits, int part_bn, cudaStream_t stream);

// gemm_tcgen05.cu
B200_API int b200_gemm(const void* x, const void* w, void* out, int m, int n, int k, long long ldx, long long ldw, long long ldc,
                       int dtype, const float* x_scale, const float* w_scale, const void* bias, const void* gate, const void* residual,
                       int act, int splits, void* workspace, long long workspace_bytes, void* status, cudaStream_t stream);
B200_API int b200_gemm_deferred_plan(int m, int n, int k, int dtype, long long workspace_bytes);
B200_API int b200_gemm_deferred(const void* x, const void* w, int m, int n, int k, long long ldx, long long ldw, int dtype,
                                const float* x_scale, const float* w_scale, void* workspace, long long workspace_bytes, float* part_ws,
                                void* status, cudaStream_t stream);
B200_API int b200_glu_form(int m, int f, int k, int dtype);
B200_API int b200_gemm_glu(const void* x, const void* w, void* out, void* out_q, void* out_sf, int m, int f, int k, long long ldx,
                           long long ldw, long long ldc, int dtype, const float* x_scale, const float* w_scale, int act, int sf_rows,
                           void* status, cudaStream_t stream);

// gemv_bf16.cu
B200_API int b200_gemv_glu(const void* x, const void* w, void* out, int m, int f, int k, long long ldx, long long ldw, long long ldc,
                           int act, cudaStream_t stream);
