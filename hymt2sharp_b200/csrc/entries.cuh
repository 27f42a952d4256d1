// Entry points of this library that other sources of it call.
#pragma once

#include "common.cuh"

HYMT2_API int hymt2_gemm_tc_norm(void* C, int c_dtype, const void* X, const void* W, int T, int N, int K, long lda, long ldw, long ldc, int epilogue,
                                 float* workspace, long workspace_floats, int* counters, int num_counters, int* status, cudaStream_t stream,
                                 const float* ss_in, int ss_in_tiles, int ss_width, float ss_eps, void* norm_out, const void* norm_gain,
                                 int norm_gain_dtype, float* ss_out, int glu_kind, float glu_limit, float glu_alpha, const float* glu_bias);
HYMT2_API int hymt2_gemm_tc_rope_kv(const void* X, const void* W, int T, int K, long lda, long ldw, void* q_out, void* k_cache, void* v_cache,
                                    const int* block_table, int table_stride, int block_tokens, const int* token_seq, const int* token_pos,
                                    const int* slot_ids, const float* inv_freq, const float* angles, int rope_dim, const void* q_gain,
                                    const void* k_gain, int gain_dtype, float eps, int nh, int nkv, int write_kv, int* status, cudaStream_t stream,
                                    const float* ss_in, int ss_in_tiles, int ss_width, float ss_eps);
HYMT2_API int hymt2_attention_prefill_tc(void* out, const void* q, const void* k_cache, const void* v_cache, long cache_blocks,
                                         const int* block_table, int table_stride, int block_tokens, const int* cu_seqlens, const int* slot_ids,
                                         const int* kv_lens, int batch, int tokens, int max_new_tokens, int nh, int nkv, int d, float scale,
                                         int window, int* status, cudaStream_t stream);
