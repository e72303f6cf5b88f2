// Internal interface of the decode-attention kernels (shared with the model runner).
#pragma once
#include "kv.cuh"
#include "rowops.cuh"

struct AttnPlan {
    int chunk;         // KV positions per CTA (multiple of 64)
    int n_splits;      // grid.x = clusters * cluster_size
    int cluster_size;  // CTAs whose shares are merged through distributed shared memory (1, 2, 4, 8 or 16)
    int mt;            // 16-query tiles per CTA (1 or 2)
    int n_qtiles;      // query tiles per (stream, kv head)
    int groups;        // streams in the batch
};
AttnPlan attn_plan(const tsb_ctx* ctx, const tsb_kv* kv, int rows, int rows_per_seq, int n_q_heads, int max_len);
size_t attn_scratch_bytes(int rows, int n_q_heads, int head_dim);
// out (natural f16 rows, may be null) and/or act (matmul operand) receive the attention output.  scratch was sized
// by attn_scratch_bytes(rows_cap, ...) and its trailing ticket words are zero (they reset themselves).  prompt_chunk > 0: the
// groups are consecutive rows of one stream, and cache rows below a group's `base` may come from the preceding launch.  The context is
// cut every prompt_chunk positions and the kernel is chosen by the model's shape alone, so that a row's sums do not depend on how many
// rows its pass, or its group, has.
cudaError_t launch_attn_decode_rows(tsb_ctx* ctx, cudaStream_t st, tsb_kv* kv, int layer, const __half* q, int64_t q_stride,
                                    __half* out, ActOut act, const tsb_row_desc* rows_dev, int rows, int rows_per_seq,
                                    int n_q_heads, float scale, int max_len, void* scratch, int rows_cap, int prompt_chunk = 0);
// How many shares of a query a prompt's call leaves in `scratch`: rows * n_q_heads * this many of (head_dim + 2) floats.
int attn_prompt_splits(int max_len, int prompt_chunk);
// A model's prompt_chunk: 1024 positions, more only where its whole window would be more than 64 of them.
inline int attn_prompt_chunk(int max_context) { return ((max_context + 63) / 64 + 1023) / 1024 * 1024; }
// Partials only: every (stream, kv head, query tile, KV chunk) CTA leaves its share (O, and (m, l)) in `scratch`,
// laid out [rows * n_q_heads][n_splits]; nobody merges (attn_merge_kernel, launched next, does).  Returns where
// the shares sit and how many splits were cut.  When the plan cuts the context into ONE split there is nothing to
// merge: the launch then writes out_single / act_single itself and the caller skips the merge.
cudaError_t launch_attn_partials(tsb_ctx* ctx, cudaStream_t st, tsb_kv* kv, int layer, const __half* q, int64_t q_stride,
                                 const tsb_row_desc* rows_dev, int rows, int rows_per_seq, int n_q_heads, float scale, int max_len,
                                 void* scratch, const float** part_o_out, const float2** part_ml_out, int* n_splits_out,
                                 __half* out_single = nullptr, ActOut act_single = ActOut{nullptr, nullptr}, int prompt_chunk = 0);
// The tensor-memory (tcgen05) kernel at head_dim 128: for passes with more than 64 queries per (stream, kv head), and for
// passes whose streams x kv heads alone give every SM a CTA; for prompts of any length.  The same partials in the same layout; the merge
// launch always follows (also after a single split).
bool attn_tc_applicable(const tsb_ctx* ctx, const tsb_kv* kv, int rows, int rows_per_seq, int n_q_heads, bool prompt);
cudaError_t launch_attn_tc_partials(tsb_ctx* ctx, cudaStream_t st, tsb_kv* kv, int layer, const __half* q, int64_t q_stride,
                                    const tsb_row_desc* rows_dev, int rows, int rows_per_seq, int n_q_heads, float scale, int max_len,
                                    void* scratch, const float** part_o_out, const float2** part_ml_out, int* n_splits_out, int prompt_chunk = 0);
cudaError_t launch_rope_store_kv(tsb_ctx* ctx, cudaStream_t st, tsb_kv* kv, int layer, __half* qkv,
                                 const tsb_row_desc* rows_dev, int rows, int n_q_heads, float theta,
                                 const float* table = nullptr);
// table [rows, head_dim]: the cosines, then the sines, of every row's position
cudaError_t launch_rope_table(tsb_ctx* ctx, cudaStream_t st, const tsb_row_desc* rows_dev, int rows, int head_dim, float theta, float* table);
