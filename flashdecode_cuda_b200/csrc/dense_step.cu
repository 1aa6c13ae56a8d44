// The launches of a prompt step through pre-norm layers of grouped-query attention and a gated feed-forward (bfloat16), in native
// code: one call per step, or two per layer where library products stand between, instead of one per kernel.
//
// A prompt step of the smallest preset is 200 launches; driven one by one from Python they took the host 2.4 ms, more than
// the GPU needs for prompts of up to some hundred tokens (19 tokens: 1.7 ms).  The kernels and their order are those of the
// parts (parts/attention.py, mlp.py, norm.py); which step may come this way is decided in engine/native.py.
#include "common.cuh"
#include "dense_step.cuh"

extern "C" {
int fd_gemm_stream(const void* x, const void* w, const void* bias, int bias_f32, void* out, int mode, int M, int N, int K,
                   int splits, int* status, void* tail_out, int tail_from, int tail_ld, cudaStream_t stream);
int fd_gemm_stream_qkv_rope(const void* x, const void* w, const void* bias, int bias_f32, void* q_out, int M, int K, int splits,
                            const float* cos_t, const float* sin_t, int table_len, const int* tok_row, const int* tok_pos,
                            const int* row_slot, void* k_pool, void* v_pool, const int* block_table, int max_blocks,
                            int num_blocks, int block_size, int n_q, int n_kv, int d, int write_kv, int* status,
                            cudaStream_t stream);
int fd_gemm_tc(const void* x, const void* w, const void* bias, int bias_f32, void* out, int mode, int M, int N, int K,
               int* status, cudaStream_t stream);
int fd_gemm_tc_qkv_rope(const void* x, const void* w, const void* bias, int bias_f32, void* q_out, int M, int K,
                        const float* cos_t, const float* sin_t, int table_len, const int* tok_row, const int* tok_pos,
                        const int* row_slot, void* k_pool, void* v_pool, const int* block_table, int max_blocks, int num_blocks,
                        int block_size, int n_q, int n_kv, int d, int write_kv, int* status, cudaStream_t stream);
int fd_attention(const void* q, const void* k_pool, const void* v_pool, void* out, int dtype, const int* block_table,
                 int max_blocks, int num_blocks, int block_size, const int* tok_row, const int* row_slot,
                 const int* row_q_start, const int* row_q_len, const int* row_ctx_len, int n_rows, int T, int max_q_len,
                 int n_q, int n_kv, int d, float scale, int window, int dv, int chunk, int n_splits, int split_len,
                 float* scratch, int* counters, int* status, const void* prefetch, unsigned long long prefetch_bytes,
                 int out_ld, float out_scale, float* prompt_scratch, int kv_len, cudaStream_t stream);
}

// A step: its buffers and index arrays; the cache's pools by group (a layer's pool is `stride` bytes after the one before) and
// the rotation tables by position.
struct FdDenseStep {
    float* resid;
    void *normed, *q, *attn, *mixer_out, *act, *ffn_out;
    const int *tok_row, *tok_pos, *row_slot, *row_q_start, *row_q_len, *row_ctx_len;
    int* status;
    cudaStream_t stream;
    float* attn_scratch;                           // null: the attention's keys are not cut into parts
    long long T, n_rows, max_q_len, kv_len, num_blocks, block_size;
    long long streams;                             // the products are the weight-streaming kernel's (up to 128 tokens)
    char *k_base[8], *v_base[8];
    const int* table[8];
    long long k_stride[8], v_stride[8], max_blocks[8];
    const float *cos_t[4], *sin_t[4];
    long long table_len[4];
};

// norm, q/k/v with rotation and append, attention.  delta: the output still to be added to the stream, or null.
extern "C" int fd_dense_mixer(const FdDenseStep* s, const FdDenseLayer* L, const void* delta) {
    const int T = (int)s->T, H = (int)L->hidden, g = (int)L->group, r = (int)L->position;
    char* kp = s->k_base[g] + L->index * s->k_stride[g];
    char* vp = s->v_base[g] + L->index * s->v_stride[g];
    int rc = fd::add_rmsnorm(delta, 1, 1, 0, s->resid, 1, L->norm1, L->norm1_f32 ? 0 : 1, (float)L->eps1, s->normed, 1, nullptr, T, H,
                             1.f, true, s->stream);
    if (rc != 0) return rc;
    if (s->streams)
        rc = fd_gemm_stream_qkv_rope(s->normed, L->w_qkv, L->b_qkv, (int)L->bias_f32, s->q, T, H, 0, s->cos_t[r], s->sin_t[r],
                                     (int)s->table_len[r], s->tok_row, s->tok_pos, s->row_slot, kp, vp, s->table[g],
                                     (int)s->max_blocks[g], (int)s->num_blocks, (int)s->block_size, (int)L->n_q, (int)L->n_kv,
                                     (int)L->d, (int)L->write_kv, s->status, s->stream);
    else
        rc = fd_gemm_tc_qkv_rope(s->normed, L->w_qkv, L->b_qkv, (int)L->bias_f32, s->q, T, H, s->cos_t[r], s->sin_t[r],
                                 (int)s->table_len[r], s->tok_row, s->tok_pos, s->row_slot, kp, vp, s->table[g],
                                 (int)s->max_blocks[g], (int)s->num_blocks, (int)s->block_size, (int)L->n_q, (int)L->n_kv,
                                 (int)L->d, (int)L->write_kv, s->status, s->stream);
    if (rc != 0) return rc;
    return fd_attention(s->q, kp, vp, s->attn, 1, s->table[g], (int)s->max_blocks[g], (int)s->num_blocks, (int)s->block_size,
                        s->tok_row, s->row_slot, s->row_q_start, s->row_q_len, s->row_ctx_len, (int)s->n_rows, T,
                        (int)s->max_q_len, (int)L->n_q, (int)L->n_kv, (int)L->d, (float)L->scale, (int)L->window, (int)L->d,
                        (int)L->chunk, 1, 0, nullptr, nullptr, s->status, nullptr, 0, 0, 1.f, s->attn_scratch,
                        (int)s->kv_len, s->stream);
}

// norm of the stream with the mixer's output added, gate/up with the activation.
extern "C" int fd_dense_gate_up(const FdDenseStep* s, const FdDenseLayer* L) {
    const int T = (int)s->T, H = (int)L->hidden, I = (int)L->inter;
    const int rc = fd::add_rmsnorm(s->mixer_out, 1, 1, 0, s->resid, 1, L->norm2, L->norm2_f32 ? 0 : 1, (float)L->eps2, s->normed, 1,
                                  nullptr, T, H, 1.f, true, s->stream);
    if (rc != 0) return rc;
    if (s->streams) return fd_gemm_stream(s->normed, L->w_gate_up, nullptr, 0, s->act, 3, T, 2 * I, H, 0, s->status, nullptr, 0, 0, s->stream);
    return fd_gemm_tc(s->normed, L->w_gate_up, nullptr, 0, s->act, 3, T, 2 * I, H, s->status, s->stream);
}

// All entries of a step whose products are all the weight-streaming kernel's; the last one's output stays in ffn_out.
extern "C" int fd_dense_layers(const FdDenseStep* s, const FdDenseLayer* layers, int n) {
    const int T = (int)s->T;
    for (int i = 0; i < n; ++i) {
        const FdDenseLayer* L = layers + i;
        const int H = (int)L->hidden;
        int rc = fd_dense_mixer(s, L, i > 0 ? s->ffn_out : nullptr);
        if (rc == 0) rc = fd_gemm_stream(s->attn, L->w_o, nullptr, 0, s->mixer_out, 1, T, H, (int)(L->n_q * L->d), 0, s->status, nullptr, 0, 0, s->stream);
        if (rc == 0) rc = fd_dense_gate_up(s, L);
        if (rc == 0) rc = fd_gemm_stream(s->act, L->w_down, nullptr, 0, s->ffn_out, 1, T, H, (int)L->inter, 0, s->status, nullptr, 0, 0, s->stream);
        if (rc != 0) return rc;
    }
    return 0;
}
