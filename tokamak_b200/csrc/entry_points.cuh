// The C entry points that other files of the library call.  The files that define them include this too, so that a definition
// and its callers cannot drift apart unnoticed: two argument lists for one C name do not compile.
#pragma once

#include "common.cuh"

TK_API int tk_add_rmsnorm(float* resid, const void* delta, const float* parts, int n_parts, long long part_stride, const float* weight,
                   void* out, const int* rows, int n_rows, int hidden, float eps, int dtype, cudaStream_t stream);
TK_API int tk_swiglu(const void* gate_up, const float* parts, int n_parts, long long part_stride, void* out, int n_tokens, int inter,
              int block, int dtype, int act, cudaStream_t stream);
TK_API int tk_rope_kv(const void* qkv, const float* qkv_parts, int n_parts, void* q_out, void* k_cache, void* v_cache,
               const int* positions, const int* tok_req, const int* req_slot, const int* block_table, const int* req_q_len,
               const int* req_kv_len, const float* q_norm_w, const float* k_norm_w, const float* rope_table, int* err,
               int n_tokens, int n_reqs, int n_q_heads, int n_kv_heads, int head_dim, int rotary_dim, int row_stride,
               int page_size, int max_pages, int num_pages, int write_kv, float eps, int dtype, cudaStream_t stream);
TK_API int tk_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                long long batch_a, long long batch_w, long long batch_c, int tile, cudaStream_t stream);
TK_API int tk_gemm_bf16_pair(const void* x, const void* w, void* out, int* err, int rows, int cols, int k, long long ld_x,
                      long long ld_w, long long ld_out, int mode, cudaStream_t stream);
TK_API int tk_gemm_bf16_tokens(const void* x, const void* w, void* out, int* err, int tokens, int rows, int k, long long ld_x,
                        long long ld_w, long long ld_out, int mode, int groups, int splits, int* launches, cudaStream_t stream);
TK_API int tk_gemm_bf16_tcgen05(const void* r, const void* c, void* out, int* err, int rows, int cols, int k, long long ld_r,
                         long long ld_c, int bn, int n_splits, int max_stages, int cluster_reduce, int epilogue,
                         const float* colscale_parts, int n_colscale_parts, float colscale_inv_dim, float colscale_eps,
                         float* resid, const float* norm_w, void* xb_out, float* sumsq_out, cudaStream_t stream);
TK_API int tk_gemm_qkv_rope(const void* w, const void* x, int* err, int tokens, int k, long long ld_w, long long ld_x, int bn,
                     int n_splits, int max_stages, const float* colscale_parts, int n_colscale_parts,
                     float colscale_inv_dim, float colscale_eps, void* q_out, void* k_cache, void* v_cache,
                     const int* positions, const int* tok_req, const int* req_slot, const int* block_table,
                     const int* req_q_len, const int* req_kv_len, const float* q_norm_w, const float* k_norm_w,
                     const void* rope_table, int n_reqs, int n_q_heads, int n_kv_heads, int page_size, int max_pages,
                     int num_pages, float eps, cudaStream_t stream);
TK_API int tk_attention_decode(const void* q, void* out, const void* k_cache, const void* v_cache, float* scratch, int* counters,
                        const int* items, const int* positions, const int* tok_req, const int* req_slot,
                        const int* block_table, int* err, int n_items, int n_reqs, int n_q_heads, int n_kv_heads,
                        int head_dim, int page_size, int max_pages, int num_pages, int window, int n_splits, float scale,
                        float softcap, const float* sinks, int chunk, const float* slopes, const float* dist_bias,
                        int dist_len, cudaStream_t stream);
TK_API int tk_attention_decode_balanced(const void* q, void* out, const void* k_cache, const void* v_cache, float* scratch,
                                 int* counters, const int* items, const int* positions, const int* tok_req,
                                 const int* req_slot, const int* block_table, int* err, int n_items, int n_reqs,
                                 int n_q_heads, int n_kv_heads, int head_dim, int page_size, int max_pages, int num_pages,
                                 int window, int blocks, float scale, float softcap, const float* sinks, int chunk,
                                 const float* slopes, const float* dist_bias, int dist_len, cudaStream_t stream);
TK_API int tk_attention_prefill_tc(const void* q, void* out, const void* k_cache, const void* v_cache, const int* records,
                            const int* block_table, int* err, int* sched, float* part_o, float* part_ml, int* part_count,
                            int n_tokens, int n_records, int n_q_heads, int n_kv_heads, int head_dim, int page_size,
                            int max_pages, int num_pages, int window, float scale, float softcap, const float* sinks,
                            int chunk, const float* slopes, const float* dist_bias, int dist_len, cudaStream_t stream);
TK_API int tk_attention_plain(const void* q, void* out, const void* k_cache, const void* v_cache, const int* positions,
                       const int* tok_req, const int* req_slot, const int* block_table, const int* items, int* err,
                       int n_tokens, int n_reqs, int n_q_heads, int n_kv_heads, int head_dim, int page_size, int max_pages,
                       int num_pages, int window, float scale, int dtype, int v_dim, float softcap, const float* sinks,
                       int q_dtype, long long q_tok_stride, long long q_head_stride, int k_stride, int v_stride, int chunk,
                       const float* slopes, const float* dist_bias, int dist_len, cudaStream_t stream);
