/* Public C interface of libnsa_b200.so (sm_100a).  Every function takes device pointers,
 * sizes and a CUDA stream, launches asynchronously on that stream and returns 0 on success
 * or an NSA_ERR_* code (text from nsa_last_error()).  Unless a function says otherwise, it
 * allocates nothing: outputs and scratch buffers are provided by the caller.
 * bf16 tensors are row-major; "ld" arguments are row pitches in elements. */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

const char* nsa_last_error(void);
long long nsa_launch_count(void);
void nsa_launch_count_reset(void);
int nsa_status_read(int* out4, int reset);   /* {code, block, info, count}; see status.cuh */
int nsa_sm_count(void);

/* C[M,N] = op(A) op(B), fp32 accumulate on tcgen05 tensor cores.  a_mn/b_mn select the
 * storage of each operand (0: reduction dimension contiguous, 1: M resp. N contiguous). */
int nsa_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                  int a_mn, int b_mn, int out_fp32, int accumulate, int max_ctas, cudaStream_t stream);

/* Kernel of plain GEMMs from now on: 0 default, 1 one CTA per tile, 2 CTA pairs. */
void nsa_gemm_select(int which);
/* CTA pairs that run at once. */
int nsa_gemm_pair_clusters(void);

/* mode 0: y = rmsnorm(x) w; 1: rmsnorm(x) w silu(gate); 2: rmsnorm(x silu(gate)) w. */
int nsa_rmsnorm_fwd(const void* x, const void* gate, const void* w, void* y, float* rstd, long rows, int d,
                    float eps, int mode, cudaStream_t st);
int nsa_rmsnorm_bwd_parts(long rows, int d);
/* partial: scratch of nsa_rmsnorm_bwd_parts(rows, d) * d floats. */
int nsa_rmsnorm_bwd(const void* x, const void* gate, const void* w, const void* dy, const float* rstd, void* dx,
                    void* dgate, void* dw_bf16, float* dw_f32, float* partial, long rows, int d, int mode,
                    cudaStream_t st);
/* RMSNorm backward that allocates nothing and takes no scratch argument: the partial-sum
 * scratch is a 9.25 MiB array built into the library (held by every GPU that loads it).
 * For hosts that may not call cudaMalloc where they run the backward pass.  Rejects
 * problems with nsa_rmsnorm_bwd_parts(rows, d) * d > 592 * 4096 (NSA_ERR_LIMIT).  First call
 * per device does a one-time address lookup: make it before any stream capture.  Calls
 * share the scratch: do not let two of them overlap on the GPU.
 * This entry point has no counterpart in the reference project. */
int nsa_rmsnorm_bwd_noalloc(const void* x, const void* gate, const void* w, const void* dy, const float* rstd,
                            void* dx, void* dgate, void* dw_bf16, float* dw_f32, long rows, int d, int mode,
                            cudaStream_t st);
/* A gate of row pitch ldg (gated modes), a gradient dres added to dx, and h = x + r with y = rmsnorm(h) w. */
int nsa_rmsnorm_fwd_ldg(const void* x, const void* gate, long ldg, const void* w, void* y, float* rstd, long rows, int d,
                        float eps, int mode, cudaStream_t st);
int nsa_rmsnorm_bwd_ldg(const void* x, const void* gate, long ldg, const void* w, const void* dy, const float* rstd,
                        void* dx, void* dgate, void* dw_bf16, float* dw_f32, float* partial, long rows, int d, int mode,
                        cudaStream_t st);
int nsa_rmsnorm_bwd_res(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx,
                        void* dw_bf16, float* dw_f32, float* partial, long rows, int d, cudaStream_t st);
int nsa_rmsnorm_add_fwd(const void* x, const void* r, const void* w, void* h, void* y, float* rstd, long rows, int d,
                        float eps, cudaStream_t st);
int nsa_l2norm_fwd(const void* x, void* y, float* rinv, long rows, int d, float eps, cudaStream_t st);
int nsa_l2norm_bwd(const void* y, const void* dy, const float* rinv, void* dx, long rows, int d, cudaStream_t st);
int nsa_swiglu_fwd(const void* g, const void* u, void* y, long rows, int cols, long ldg, long ldu, cudaStream_t st);
int nsa_swiglu_bwd(const void* g, const void* u, const void* dy, void* dg, void* du, long rows, int cols, long ldg,
                   long ldu, long ldo, cudaStream_t st);
int nsa_rope(const void* x, const float* cos_t, const float* sin_t, void* y, long batch, int T, int H, int D,
             int backward, cudaStream_t st);
int nsa_conv1d_fwd(const void* x, const void* w, const void* bias, void* y, int B, int T, int C, long ldx, int width,
                   int act, cudaStream_t st);
long nsa_conv1d_bwd_parts(int B, int T, int C);
/* partial: scratch of nsa_conv1d_bwd_parts(B, T, C) * 5 * C floats; dw [C][4], db [C] or null, fp32 or bf16. */
int nsa_conv1d_bwd(const void* x, const void* w, const void* bias, const void* dy, void* dx, float* partial, void* dw,
                   void* db, int dw_fp32, int B, int T, int C, long ldx, int width, int act, cudaStream_t st);
int nsa_embedding_fwd(const long* ids, const void* w, void* y, long n, int d, long vocab, cudaStream_t st);
int nsa_embedding_bwd(const long* sorted_ids, const long* perm, const void* dy, float* dw, long n, int d, cudaStream_t st);

int nsa_adamw_step(void* p, const void* g, float* m, float* v, float* master, const float* grad_scale, long n,
                   int p_fp32, int g_fp32, int step, float lr, float b1, float b2, float eps, float wd, cudaStream_t st);
int nsa_adamw8bit_step(void* p, const void* g, uint8_t* mq, float* mabs, uint8_t* vq, float* vabs,
                       const float* cb_signed, const float* cb_unsigned, const float* grad_scale, long n, int p_fp32,
                       int g_fp32, int step, float lr, float b1, float b2, float eps, float wd, cudaStream_t st);
/* The same updates over a list of tensors, one launch per 48.  words: 7 per tensor, {p, g, m, v, a, b, n} with a =
 * fp32 master copy or 0 and b unused for fp32 state, a / b = scales of the moments for 8-bit state. */
int nsa_adamw_multi(const long long* words, int tensors, const float* grad_scale, int p_fp32, int g_fp32, int step,
                    float lr, float b1, float b2, float eps, float wd, cudaStream_t st);
int nsa_adamw8bit_multi(const long long* words, int tensors, const float* cb_signed, const float* cb_unsigned,
                        const float* grad_scale, int p_fp32, int g_fp32, int step, float lr, float b1, float b2, float eps,
                        float wd, cudaStream_t st);
int nsa_sumsq_parts(void);
int nsa_sumsq(const void* g, long n, int g_fp32, float* partial, float* out, int accumulate, cudaStream_t st);
int nsa_cross_entropy(void* logits, const long* labels, float* loss_rows, const float* inv_count, long rows, int V,
                      long ld, long ignore_index, int write_grad, cudaStream_t st);
/* dst (bf16) = src (fp32 or bf16) * (*scale); 16-byte aligned bases. */
int nsa_scale_bf16(const void* src, void* dst, const float* scale, long n, int src_fp32, cudaStream_t st);

/* ---- attention family: (B, T, H, D) bf16 tensors, L = log2-sum-exp per row (csrc/attention.cu) ---- */
int nsa_attn_fwd(const void* q, const void* k, const void* v, void* o, float* L, int B, int T, int S, int Hq, int
    Hkv, int D, float scale, int causal, int window, int kp_stride, int kp_off, const int* tile_blocks, const unsigned
    long long* tile_masks, const int* tile_counts, int max_u, cudaStream_t st);
int nsa_attn_importance(const void* q, const void* k_cmp, const float* L_in, float* imp, int B, int T, int S, int Hq,
    int Hkv, int D, float scale, int kp_stride, int kp_off, int nS, cudaStream_t st);
int nsa_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* L, float*
    delta, void* dq, float* dk, float* dv, int B, int T, int S, int Hq, int Hkv, int D, float scale, int causal, int
    window, int kp_stride, int kp_off, const int* tile_blocks, const unsigned long long* tile_masks, const int*
    tile_counts, int max_u, cudaStream_t st);
int nsa_attn_bwd_walks(int B, int T, int S, int Hq, int Hkv, int causal, int window, int kp_stride);      // head_dim 128
int nsa_attn_bwd_walks_d64(int B, int T, int S, int Hq, int Hkv, int causal, int window, int kp_stride);  // head_dim 64
int nsa_attn_bwd_split(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* L,
    float* delta, void* dq, void* dk, void* dv, int B, int T, int S, int Hq, int Hkv, int D, float scale, int causal,
    int window, int kp_stride, int kp_off, const int* tile_blocks, const unsigned long long* tile_masks, const int*
    tile_counts, int max_u, const int* tok_list, const int* list_start, const int* item_start, int nS, int item_bound,
    int visits_per_cta, float* part, int walks, int delta_given, int add_dq, int write_kv, cudaStream_t st);
int nsa_union_blocks(const int* idx, int* tile_blocks, unsigned long long* tile_masks, int* tile_counts, int B, int
    T, int Hkv, int G, int top_n, int nS, int max_u, cudaStream_t st);

/* ---- peer-memory collectives and the IPC arena (csrc/comm.cu) ---- */
int nsa_enable_peer_access(int peer_device);
int nsa_comm_signal(unsigned* const* flag_rows, int W, int slot, unsigned epoch, cudaStream_t st);
int nsa_comm_wait(const unsigned* flags, int n, unsigned epoch, long long max_cycles, cudaStream_t st);
int nsa_comm_allgather(const void* const* shards, void* out, long shard_bytes, int W, int rank, const unsigned*
    flags, unsigned epoch, long long max_cycles, int ctas_per_peer, cudaStream_t st);
int nsa_comm_reduce_scatter_parts(void);
int nsa_comm_reduce_scatter(const float* const* grads, float* grad_shard, long S, int W, int rank, float scale, int
    accumulate, float* sumsq_partial, const unsigned* flags, unsigned epoch, long long max_cycles, cudaStream_t st);
int nsa_comm_rs_adamw8bit(const float* const* grads, void* p_shard, int p_fp32, uint8_t* mq, float* mabs, uint8_t*
    vq, float* vabs, const float* cb_signed, const float* cb_unsigned, const uint8_t* wd_mask, long S, int W, int rank,
    float scale, int step, float lr, float b1, float b2, float eps, float wd, const unsigned* flags, unsigned epoch, long
    long max_cycles, cudaStream_t st);
int nsa_ipc_alloc(long nbytes, void** out_ptr, unsigned char* handle64);
int nsa_ipc_open(const unsigned char* handle64, void** out_ptr);
int nsa_ipc_close(void* p);
int nsa_ipc_free(void* p);

/* ---- more element-wise kernels (csrc/elementwise.cu) ---- */
int nsa_gate_combine_fwd(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2, const void*
    g3, void* o, long rows, int D, cudaStream_t st);
int nsa_gate_combine_bwd(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2, const void*
    g3, const void* d_o, void* do1, void* do2, void* do3, void* dg1, void* dg2, void* dg3, long rows, int D, cudaStream_t
    st);

/* Gates (or, with sig, their logits) of row pitch ldg; e1..e3 null or rowsum(do_i * o_i).  Mean pooling of windows. */
int nsa_gate_combine_fwd_ex(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2, const void*
    g3, long ldg, int Hq, int sig, void* o, long rows, int D, cudaStream_t st);
int nsa_gate_combine_bwd_ex(const void* o1, const void* o2, const void* o3, const void* g1, const void* g2, const void*
    g3, long ldg, int Hq, int sig, const void* d_o, void* do1, void* do2, void* do3, void* dg1, void* dg2, void* dg3,
    float* e1, float* e2, float* e3, long rows, int D, cudaStream_t st);
int nsa_pool_fwd(const void* x, void* y, int B, int T, int width, long ldx, int block, int stride, cudaStream_t st);
int nsa_pool_bwd(const void* dy, void* dx, int B, int T, int width, int block, int stride, cudaStream_t st);

/* ---- Gated DeltaNet: per-chunk kernels (csrc/gdn_chunk.cu), state recurrence (csrc/gdn.cu) ---- */
int nsa_gdn_prep(const void* q, const void* k, const void* v, const float* g, const float* beta, void* w, void* u,
    void* qk, float* X, float* gc, int B, int T, int H, int K, int V, float scale, cudaStream_t st);
int nsa_gdn_seq_fwd(const void* q, const void* k, const void* w, const void* u, const void* qk, const float* gc, void*
    o, void* v_new, void* S_all, int B, int T, int H, int K, int V, float scale, cudaStream_t st);
int nsa_gdn_seq_bwd(const void* q, const void* k, const void* w, const void* qk, const void* S_all, const void* d_o,
    const float* gc, void* du, void* dS_all, float* dgamma_part, int B, int T, int H, int K, int V, float scale,
    cudaStream_t st);
int nsa_gdn_post(const void* q, const void* k, const void* v, const void* d_o, const float* beta, const float* gc,
    const float* X, const void* v_new, const void* du, const void* S, const void* dS, const float* dgamma, void* dq,
    void* dk, void* dv, float* dg, float* dbeta, int B, int T, int H, int K, int V, float scale, cudaStream_t st);

/* ---- step sizes and gates of the recurrent mixers (csrc/gates.cu), rows of pitch lda / ldb; b null: dt and A ---- */
int nsa_gates(const void* a, long lda, const void* b, long ldb, const void* bias, int bias_fp32, const void* A_log, int A_fp32,
    float* out0, float* out1, long rows, int H, cudaStream_t st);

/* ---- GEMM (csrc/gemm.cu) ---- */
/* C32 (zeroed or to be added to) += op(A) op(B), the reduction cut into split_k parts. */
int nsa_gemm_bf16_splitk(const void* A, const void* B, float* C32, int M, int N, int K, int lda, int ldb, int ldc,
    int a_mn, int b_mn, int split_k, cudaStream_t stream);
int nsa_gemm_bf16_ag(const void* A, void* C, int M, int N, int K, int lda, int ldc, const void* const* shards, void*
    full, long shard_elems, long b_elem_offset, int W, int rank, unsigned* chunk_flags, int chunks_per_shard, const
    unsigned* peer_flags, unsigned epoch, long long max_cycles, int copy_ctas, cudaStream_t stream);

/* ---- forward-only scan of the complex-state block (csrc/mamba3.cu) ---- */
int nsa_mamba3_scan(const float* u, const float* dt, const float* A, const float* Bc, const float* Cc, const float*
    D, float* gate, int B, int L, int H, int N, cudaStream_t st);

/* ---- Mamba-2 SSD chunk kernels (csrc/ssd.cu) ---- */
int nsa_ssd_state_fwd(const float* S, const float* gamma, float* Hprev, void* Hprev_bf16, float* Hlast, int B, int
    nc, int H, long E, cudaStream_t st);
int nsa_ssd_state_bwd(const float* dHprev, const float* gamma, float* dS, void* dS_bf16, int B, int nc, int H, long
    E, cudaStream_t st);
int nsa_ssd_grad_slots(int B, int T, int H);
int nsa_ssd_finish(const float* dB_part, const float* dC_part, const float* q, const float* k, const float* r, const
    float* dt, const float* A, float* scratch, void* dB, void* dC, float* ddt, float* dA, float* dD, int B, int T, int H,
    cudaStream_t st);
int nsa_ssd_states_in_one(int B, int T, int H);
int nsa_ssd_states_form(int B, int T, int H);
int nsa_ssd_states(int back, const void* bc, long ld_bc, const void* v, long ld_v, const float* dt, const float* A, void*
    out, int B, int T, int H, int N, int P, cudaStream_t st);
int nsa_ssd_chunk_state(int mode, const void* bc, long ld_bc, const void* v, long ld_v, const float* dt, const float*
    A, float* S_out, float* gamma_out, int B, int T, int H, int N, int P, cudaStream_t st);
int nsa_ssd_chunk_out(const void* Cm, long ld_c, const void* Bm, long ld_b, const void* x, long ld_x, const void*
    Hprev_bf16, const float* dt, const float* A, const float* Dskip, void* y, int B, int T, int H, int N, int P,
    cudaStream_t st);
int nsa_ssd_chunk_grad(const void* Cm, long ld_c, const void* Bm, long ld_b, const void* x, long ld_x, const void*
    dy, const void* Hprev_bf16, const void* dHn_bf16, const float* dt, const float* A, const float* Dskip, void* dx, float*
    dB_part, float* dC_part, float* q_out, float* k_out, float* r_out, int B, int T, int H, int N, int P, cudaStream_t st);

/* ---- further entry points of attention.cu ---- */
int nsa_inverse_chunks(int BH, int T, int nS);
int nsa_inverse_blocks(const int* idx, int* tok_list, int* list_start, int* item_start, int* hist, int* count, int BH,
    int T, int n, int nS, int R, int visits_per_cta, cudaStream_t st);
int nsa_select_blocks(const float* imp, int* idx, long rows, int T, int nS, int sel_block, int top_n, cudaStream_t
    st);

/* ---- further entry points of optim.cu ---- */
int nsa_affine_quant(const float* t, uint8_t* q, float* scale, float* zero, long rows, int cols, int q_block, int
    bits, cudaStream_t st);
int nsa_affine_dequant(const uint8_t* q, const float* scale, const float* zero, float* out, long rows, int cols, int
    q_block, cudaStream_t st);

/* ---- further entry points of runtime.cu ---- */
int nsa_copy2d(void* dst, long dst_pitch_bytes, const void* src, long src_pitch_bytes, long width_bytes, long rows,
    cudaStream_t st);

#ifdef __cplusplus
}
#endif
