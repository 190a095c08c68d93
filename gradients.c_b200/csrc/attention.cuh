// Internal interface between the attention entry points (attention.cu) and the tensor-core
// flash kernels (attention_flash.cu).
#pragma once
#include "common.cuh"

struct gdb_flash_args {
    const void *q, *k, *v, *grad_out;
    const int *cu;
    void *out_or_dq;   // forward: out; backward: dQ
    void *dk, *dv;     // backward only
    float *stats;      // [N, Hq, 3] (row max, exp-sum, D); may be NULL in forward
    int n_tokens, batch, hq, hkv, dh;
    int causal, window, prefix, max_seqlen;
    float scale;
    uint32_t dtype;
    int keep_dq32;     // single-pass backward: leave the query gradient unrounded in the FP32 accumulator, do not write dQ
};

// Both return GD_ERR_UNSUPPORTED when the configuration is outside the fast path; the caller
// then runs the general kernels.
gd_status gdb_flash_varlen_forward(gd_backend *be, const gdb_flash_args *a);
gd_status gdb_flash_varlen_backward(gd_backend *be, const gdb_flash_args *a, bool have_forward_stats);
// Backward when the forward output is available (attention_flash.cu); dq32: FP32 scratch [N, Hq, Dh] (used at head_dim 64).
gd_status gdb_flash_varlen_backward_with_out(gd_backend *be, const gdb_flash_args *a, const void *out, float *dq32);
// tcgen05 / tensor-memory forward (attention_tcgen05.cu); GD_ERR_UNSUPPORTED outside its fast path.
gd_status gdb_attn5_forward(gd_backend *be, const gdb_flash_args *a);
// What the preparation kernel (attention_flash.cu) leaves for the tensor-memory backward, all in device memory:
struct gdb_attn_bwd_meta {
    int n_pad;         // tokens rounded up to the query tile of 64: row pitch of the two arrays of statistics
    float *neg_m2;     // [Hq, n_pad]  -(m log2e + log2 l)
    float *neg_d;      // [Hq, n_pad]  -D scale (head_dim 128: zero here, written with dQ)
    int *row_hi;       // [N]  last query that may see this key (-1: none)
    int *row_lo;       // [N]  first key that this query may see (behind the last sequence: not written)
    int *tile_nqt;     // [ceil(N / 128)]  64-row query tiles, from the key tile's own first row on, that may see one of its keys
};
// head_dim 128: dQ and D, query-stationary (attention_tcgen05_dq.cu); gdb_attn5_backward launches it in front of its own kernel.
gd_status gdb_attn5_query_gradient(gd_backend *be, const gdb_flash_args *a, const gdb_attn_bwd_meta *m);
// Workspace that the tensor-memory backward's preparation needs (it runs the general kernels with less).
size_t gdb_attn_bwd_ws_bytes(int n_tokens, int hq);
// tcgen05 / tensor-memory backward (attention_tcgen05_bwd.cu): dK, dV and, head_dim 64, the FP32 dQ accumulator dq32 [N, Hq, 64] (zero
// on entry), head_dim 128, dQ itself. GD_ERR_UNSUPPORTED outside its fast path.
gd_status gdb_attn5_backward(gd_backend *be, const gdb_flash_args *a, float *dq32, const gdb_attn_bwd_meta *m);
