// A dense block's step launched by one call (host code only): projection with rotation and cache append, attention of the prompt,
// output projection, gate and up, down, each through its own entry point with the arguments that a caller would give it one by one.
// A short prompt's step is as long as the host takes to launch it: five calls with some thirty arguments each, their checks and the
// tensors in between cost the interpreter 120 us a block, this call and its arguments 25.
#include "entries.cuh"

// One step of one block.  All sizes in elements; null pointers where the text says "or null".
struct Hymt2DenseBlock {
    const void* x;               // [T, hidden] bfloat16: the first norm's output, or bf16(row * gain) with its sums of squares in ss_in
    const float* ss_in;          // or null
    float* residual;             // [T, hidden] float32
    const void *w_qkv, *w_o, *w_gate_up, *w_down;                // contiguous, bfloat16
    const void *q_gain, *k_gain;                                 // or null
    const void *norm2_gain, *next_gain;                          // the second norm's; that of the norm behind the block, or null
    void *q, *att, *act, *normed;                                // [T, nh * 128] twice, [T, inner], [T, hidden], bfloat16
    float* ss;                                                   // [T, norm tiles]
    void *k_plane, *v_plane;                                     // one layer's planes
    const int *block_table, *token_seq, *token_pos, *slot_ids, *cu_seqlens, *kv_lens;
    const float *inv_freq, *angles;                              // or null
    float* workspace;                                            // the gate and up product's, or null
    int *counters, *status;
    long cache_blocks, workspace_floats, ldx;
    int T, hidden, inner, nh, nkv, batch, max_new_tokens, table_stride, block_tokens, rope_dim, write_kv, window;
    int gain_dtype, norm2_dtype, next_dtype, ss_in_tiles, ss_tiles, num_counters;
    float qk_eps, norm1_eps, norm2_eps, scale;
};

HYMT2_API int hymt2_dense_block_bytes() { return (int)sizeof(Hymt2DenseBlock); }

// Five kernels on `stream`.
HYMT2_API int hymt2_dense_block(const Hymt2DenseBlock* b, cudaStream_t stream) {
    HYMT2_REQUIRE(b, "dense_block: no arguments");
    constexpr int HEAD = 128, ADD = 1, SWIGLU = 2;
    const int wide = b->nh * HEAD;
    int rc = hymt2_gemm_tc_rope_kv(b->x, b->w_qkv, b->T, b->hidden, b->ldx, b->hidden, b->q, b->write_kv ? b->k_plane : nullptr,
                                   b->write_kv ? b->v_plane : nullptr, b->block_table, b->table_stride, b->block_tokens, b->token_seq, b->token_pos,
                                   b->slot_ids, b->inv_freq, b->angles, b->rope_dim, b->q_gain, b->k_gain, b->gain_dtype, b->qk_eps, b->nh, b->nkv,
                                   b->write_kv, b->status, stream, b->ss_in, b->ss_in_tiles, b->ss_in ? b->hidden : 0, b->norm1_eps);
    if (rc) return rc;
    rc = hymt2_attention_prefill_tc(b->att, b->q, b->k_plane, b->v_plane, b->cache_blocks, b->block_table, b->table_stride, b->block_tokens,
                                    b->cu_seqlens, b->slot_ids, b->kv_lens, b->batch, b->T, b->max_new_tokens, b->nh, b->nkv, HEAD, b->scale,
                                    b->window, b->status, stream);
    if (rc) return rc;
    rc = hymt2_gemm_tc_norm(b->residual, HYMT2_F32, b->att, b->w_o, b->T, b->hidden, wide, wide, wide, b->hidden, ADD, nullptr, 0, nullptr, 0,
                            b->status, stream, nullptr, 0, 0, 0.f, b->normed, b->norm2_gain, b->norm2_dtype, b->ss, GLU_SILU, 0.f, 1.f, nullptr);
    if (rc) return rc;
    rc = hymt2_gemm_tc_norm(b->act, HYMT2_BF16, b->normed, b->w_gate_up, b->T, b->inner, b->hidden, b->hidden, b->hidden, b->inner, SWIGLU,
                            b->workspace, b->workspace_floats, b->counters, b->num_counters, b->status, stream, b->ss, b->ss_tiles, b->hidden,
                            b->norm2_eps, nullptr, nullptr, HYMT2_F32, nullptr, GLU_SILU, 0.f, 1.f, nullptr);
    if (rc) return rc;
    return hymt2_gemm_tc_norm(b->residual, HYMT2_F32, b->act, b->w_down, b->T, b->hidden, b->inner, b->inner, b->inner, b->hidden, ADD, nullptr, 0,
                              nullptr, 0, b->status, stream, nullptr, 0, 0, 0.f, b->next_gain ? b->normed : nullptr, b->next_gain, b->next_dtype,
                              b->next_gain ? b->ss : nullptr, GLU_SILU, 0.f, 1.f, nullptr);
}
