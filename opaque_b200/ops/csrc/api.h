// C entry points of libopaque_b200.so (every function returns 0 on success, a negative
// code on a host-side failure; device-side wait timeouts are reported through `status`).
#pragma once
#ifdef __cplusplus
extern "C" {
#endif

int ob_wgrad_clip(const void* a, const void* b, int T, int M, int N, long long lda, long long ldb,
                  const float* row_scale, const int* seg_offsets, int num_groups, int splits, float* out,
                  float* const* peer_out, long long shard_elems, const long long* group_out_offset,
                  long long group_stride, long long out_offset, long long ldm, long long ldn, int n_valid,
                  int accumulate, int block_n, int* status, double wait_budget_s, int num_sms, void* stream);

// Several problems in one launch (host arrays of descriptions; launches hold up to 56): the layers of a backward pass
// share one work list; put problems with more work per item first.
//   ghost        norm2[i] += || A_i^T G_i ||_F^2 for every segment i of rows, from Gram matrices (ids: one-hot inputs)
//   wgrad        ob_wgrad_clip
//   wgrad_pe     out[m, n] (+)= sum over examples e of ex_scale[e] * A_e^T B_e, where example e owns rows
//                [e * ex_rows, (e + 1) * ex_rows) of a [T, M] and b [T, N] (any ex_rows); the factor is applied to each example's
//                fp32 partial product in the epilogue, operands are not modified; splits > 1 needs accumulate = 1.
//                norm2 != NULL in every description: norm2[e] += || A_e^T B_e ||_F^2 instead, nothing else is written
typedef struct {
  const void *a, *g;
  const int* ids;
  float* norm2;
  const int *seg, *seg_out;
  long long lda, ldg, total_rows;
  int B, T, Da, Dg;
} ob_ghost_desc;
typedef struct {
  const void *a, *b;
  const float* row_scale;
  const int* seg_offsets;
  const long long* group_out_offset;
  long long lda, ldb, group_stride, out_offset, ldm, ldn;
  int T, M, N, num_groups, splits, n_valid, accumulate;
} ob_wgrad_desc;
typedef struct {
  const void *a, *b;
  const float* ex_scale;
  float* norm2;
  long long lda, ldb, out_offset, ldm;
  int num_examples, ex_rows, M, N, splits, accumulate;
} ob_wgrad_pe_desc;
int ob_ghost_norm_batch(const ob_ghost_desc* descs, int count, int* status, double wait_budget_s, int num_sms, void* stream);
int ob_wgrad_clip_batch(const ob_wgrad_desc* descs, int count, float* out, float* const* peer_out, long long shard_elems,
                        int block_n, int* status, double wait_budget_s, int num_sms, void* stream);
int ob_wgrad_clip_pe_batch(const ob_wgrad_pe_desc* descs, int count, float* out, float* const* peer_out,
                           long long shard_elems, int* status, double wait_budget_s, int num_sms, void* stream);

// D[M, N] = A[M, K1] op(B) + A2[M, K2] B2[N, K2]^T + bias, bf16 in / bf16 out, fp32 accumulation.  b_kn = 0: B is
// [N, K1] row-major (per group: [groups * N, K1]); b_kn = 1: B is [K1, N] row-major (per group: [groups * K1, N]).
// group_offs (int32 device array [num_groups + 1]) switches on the grouped mode: rows [offs[e], offs[e+1]) use slab e.
// b2_kn = 1: B2 is [K2, N] row-major.  alpha scales the products, not the bias.  block_n: columns per tile, 256 or (ungrouped) 64.
int ob_gemm_tn(const void* a, const void* b, const void* a2, const void* b2, const void* bias, void* out,
               long long rows_a, int N, int K1, int K2, long long lda, long long ldb, long long lda2, long long ldb2,
               long long ldo, int b_kn, int b2_kn, float alpha, const int* group_offs, int num_groups, int block_n,
               int* status, double wait_budget_s, int num_sms, void* stream);

// The same kernel (64-column tiles, N % 64 == 0, contiguous out and pre) with a plain activation in its epilogue (0 silu, 1 gelu erf,
// 2 gelu tanh): out = act(D) and, where given, pre = D; backward: out = D * act'(pre).
int ob_gemm_tn_act(const void* a, const void* b, const void* bias, void* out, void* pre, long long rows_a, int N, int K, long long lda,
                   long long ldb, int b_kn, int act, int backward, int* status, double wait_budget_s, int num_sms, void* stream);

// Dense GEMM on CTA pairs (tcgen05 cta_group::2):  D = A op1(B) + A2 op2(B2) + bias.
// tile (without glu): 1 = 256 x 256 tiles with two alternating accumulators, 0 = 512 x 256 tiles, -1 = by size; the same bits.
// b_kn / b2_kn = 1: that B operand is stored [K, N] row-major, 0: [N, K].  glu != 0: `b` holds the gate rows and `b_up`
// the up rows of a gated MLP ([N/2, K] each; N counts both), out [M, N/2] = act(gate) * up (glu_act: 0 silu, 1 gelu erf,
// 2 gelu tanh) and the optional out_gate / out_up receive the pre-activations; glu = 2: out = act(D), out_gate (optional) = D.
int ob_gemm_pair(const void* a, const void* b, const void* b_up, const void* a2, const void* b2, const void* b2_up,
                 const void* bias, void* out, void* out_gate, void* out_up, long long rows_a, int N, int K1, int K2,
                 long long lda, long long ldb, long long lda2, long long ldb2, long long ldo, int b_kn, int b2_kn, int glu,
                 int glu_act, int tile, int* status, double wait_budget_s, int num_sms, void* stream);
// Data gradient of a gated MLP's down projection with the activation's backward in the epilogue: dH = dY op(W) stays in
// tensor memory; dGate = dH * up * act'(gate) and dUp = dH * act(gate) are stored (bf16 [M, N], pitch ld_out).  N % 64 == 0.
// up = dup = NULL: a plain activation, dGate = dH * act'(gate).
int ob_gemm_pair_glu_bwd(const void* dy, const void* w, const void* gate, const void* up, void* dgate, void* dup,
                         long long rows_a, int N, int K, long long lddy, long long ldw, long long ld_gu, long long ld_out,
                         int b_kn, int glu_act, int* status, double wait_budget_s, int num_sms, void* stream);
// Die map of the current device (which SMs share a die, probed by atomic latency; once per device and process).
// ob_pair_init: probes if needed, returns 1000 * (SM pairs on die 0) + (SM pairs on die 1), 0 if no two-die split was
// found; call it outside stream captures.  ob_die_map: smid -> 0 / 1 into out[0 .. n), returns the SM count or 0.
int ob_pair_init(void);
int ob_pair_set_die_aware(int on);   // die-aware tile assignment of the pair GEMMs (default off); returns the old value
int ob_die_map(unsigned char* out, int n);
// Output head fused with cross-entropy statistics on CTA pairs: logits tiles stay in tensor memory, per-tile partials
// (scratch: rows * 2 * ceil(N / 256) float4) are combined in a fixed order into nll[rows], lse[rows]; `logits_out` (optional)
// receives the bf16 soft-capped logits for the backward pass.
int ob_linear_ce_fwd(const void* hidden, const void* weight, const long long* labels, void* logits_out, float* partials,
                     float* nll, float* lse, long long rows, int N, int K, long long ldh, long long ldw, long long ldo,
                     float softcap, float smoothing, long long ignore_index, int* status, double wait_budget_s,
                     int num_sms, void* stream);
// In place on those stored logits: z <- row_weight * d nll / d (raw logits), one read and one write per element.
int ob_linear_ce_dlogits(void* logits, const long long* labels, const float* lse, const float* row_weight, long long rows,
                         int N, long long ld, float softcap, float smoothing, long long ignore_index, void* stream);
unsigned int ob_debug_idesc_bf16(int m, int n, int a_mn_major, int b_mn_major);

// Mixture of experts: out[t] = sum_j w[t * k + j] * y[pos[t * k + j]] (w NULL: plain sum), rows of H bf16 values, H % 8 == 0.
int ob_moe_combine(const void* y, const void* w, const long long* pos, void* out, long long tokens, int k, int H, int sms,
                   void* stream);
// Its backward by sorted row i: dy[i] = w[slot[i]] * dout[token[i]], dw[slot[i]] = <dout[token[i]], y[i]> (fp32).
int ob_moe_row_grad(const void* dout, const void* y, const void* w, const long long* token, const long long* slot, void* dy,
                    float* dw, long long rows, int H, int sms, void* stream);
// [dGate | dUp] (rows of 2I) of silu(gate) * up for gate_up = [gate | up], dh rows of I bf16 values, I % 8 == 0; exact fp32 steps.
int ob_moe_glu_bwd(const void* dh, const void* gate_up, void* dgate_up, long long rows, int I, int sms, void* stream);

// ob_rows_group_sum for several matrices with the same rows in one launch per 128 (host array of descriptions): g and x
// [num_examples * rows_per_example, N] with pitch ldg, out / out2 rows with pitch ld_out / ld_out2, modes as there.
typedef struct {
  const void *g, *x;
  const float *mean, *rstd;
  float *out, *out2;
  long long ldg, ld_out, ld_out2;
  int N, mode;
} ob_rowsum_desc;
int ob_rows_sum_batch(const ob_rowsum_desc* descs, int count, int num_examples, int rows_per_example, void* stream);
// a_cat [3r, in] = (aq; ak; av), b_block [oq + ok + ov, 3r] = blockdiag(bq, bk, bv); contiguous bf16, r % 8 == 0.
int ob_lora_pack(const void* aq, const void* ak, const void* av, const void* bq, const void* bk, const void* bv, void* a_cat,
                 void* b_block, int r, int in, int oq, int ok, int ov, int sms, void* stream);
// Per-example clipping of a materialised fp32 gradient tree: leaf[i] is [E, numel[i]] contiguous, out[i] [numel[i]] receives
// factor * sum_e scale[e] * leaf[i][e]; scale = bound / (norm + gamma) (automatic) or min(1, bound / norm), times `shrink`
// minus `ulp`, 0 where not finite.  `partial` is scratch of E * ob_clip_tree_chunks(...) doubles.  At most 64 leaves.
long long ob_clip_tree_chunks(const long long* numel, int leaves);
int ob_clip_tree(const void* const* leaf, void* const* out, const long long* numel, int leaves, int E, double bound,
                 double gamma, double shrink, double ulp, int automatic, float factor, double* partial, float* norms,
                 float* scale, float* clipped, void* stream);

// RMSNorm: y = x * rsqrt(mean(x^2) + eps) * (offset + w); with `residual` x + residual first, stored to sum_out.  mode: casting.
int ob_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* sum_out, float* rstd, long long rows, int H,
                   float eps, float offset, int mode, void* stream);
int ob_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dsum_in, void* dx,
                   float* dw_per_example, const int* seg_offsets, int num_examples, int rows_per_example, long long rows, int H,
                   float offset, void* stream);
// dgate, dup (pitch ld_out) of act(gate) * up (pitch ld_in) for dh [rows, I]; act: 0 silu, 1 gelu erf, 2 gelu tanh.
int ob_glu_bwd(const void* dh, const void* gate, const void* up, void* dgate, void* dup, long long rows, int I, long long ld_in,
               long long ld_out, int act, int sms, void* stream);
// Rotary embedding of q and k read through element strides (batch, token, head); contiguous outputs [rows, heads, D].
int ob_rope_qk_oop(const void* q_in, const void* k_in, void* q_out, void* k_out, const float* cos_t, const float* sin_t,
                   const int* pos, long long rows, int seq_len, int Hq, int Hk, int D, long long q_sb, long long q_st,
                   long long q_sh, long long k_sb, long long k_st, long long k_sh, int backward, int sms, void* stream);

// The same with v, copied, and one output [rows, (Hq + 2 Hk) D]; strides[9] (host): batch, token, head stride of q, k, v.
int ob_rope_qkv_gather(const void* q_in, const void* k_in, const void* v_in, void* out, const float* cos_t, const float* sin_t,
                       const long long* strides, long long rows, int seq_len, int Hq, int Hk, int D, int backward, int sms, void* stream);

// LayerNorm over the last dimension (bf16 in/out, fp32 statistics saved per row).
int ob_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, long long rows,
                     int H, float eps, void* stream);
int ob_layernorm_bwd_dx(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx,
                        long long rows, int H, void* stream);
// The same with a residual addition in front (H <= 1024): sum = x + res (bf16), y = layernorm(sum); backward: dx = ... + ds.
int ob_add_layernorm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* sum, float* mean,
                         float* rstd, long long rows, int H, float eps, void* stream);
int ob_add_layernorm_bwd_dx(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* ds,
                            void* dx, long long rows, int H, void* stream);
// Either backward (ds NULL or not, H <= 1024) with the per-example sums of ob_rows_group_sum mode 1 into out_w, out_b (may be NULL).
int ob_layernorm_bwd_sums(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* ds,
                          void* dx, int num_examples, int rows_per_example, int H, float* out_w, float* out_b, long long ld_out,
                          void* stream);
// out[e, :N] += sum over the rows of example e of g (mode 0), g * (x - mean) * rstd (mode 1) or g * x * rstd (mode 2);
// out row pitch ld_out.  In modes 1 and 2 a non-NULL out2 (row pitch ld_out2) also receives the plain sums of g.
int ob_rows_group_sum(const void* g, const void* x, const float* mean, const float* rstd, int num_examples,
                      int rows_per_example, int N, long long ldg, float* out, long long ld_out, int mode, float* out2,
                      long long ld_out2, void* stream);
// q, k, v gradients [B, heads, T, hd] (strides[9] = batch, head, token stride of each, in elements; head vectors
// contiguous) -> out [B*T, 3*heads*hd] bf16.
int ob_merge_heads3(const void* q, const void* k, const void* v, const long long* strides, void* out, long long B, int T,
                    int heads, int hd, int sms, void* stream);
// out = act(x) (dy == NULL) or dy * act'(x); act: 0 silu, 1 gelu erf, 2 gelu tanh, 3 relu.
int ob_activation(const void* x, const void* dy, void* out, long long numel, int act, int sms, void* stream);

#ifdef __cplusplus
}
#endif
