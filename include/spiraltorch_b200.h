/* C ABI of libst_b200.so (sm_100a kernels) and libst_host.so (host runtime).
 * Generated by csrc/gen_header.py from the sources; do not edit.
 *
 * Conventions: launchers return an StStatus code (0 = ok) and take the CUDA stream as a void*
 * (cudaStream_t); device pointers are raw; bf16 tensors are passed as void*.  Argument blocks are plain
 * structs whose layout is shown here.  st_last_error() returns the message of the last failure. */
#ifndef SPIRALTORCH_B200_H
#define SPIRALTORCH_B200_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

typedef struct __nv_bfloat16_opaque __nv_bfloat16;   /* bf16 element; only pointers cross the ABI */
#ifndef __cplusplus
typedef _Bool bool;
#endif
typedef void (*st_host_task_fn)(void*);
typedef struct SpiralTensor SpiralTensor;     /* opaque host tensor of the tensor-level ABI */
typedef struct RuntimeHandle RuntimeHandle;   /* opaque runtime (worker count) of the tensor-level ABI */

/* csrc/common/host.h */
enum StStatus {
  ST_OK = 0,
  ST_ERR_INVALID = 1,    // bad argument (shape / alignment / unsupported combination)
  ST_ERR_CUDA = 2,       // CUDA runtime or driver error; see st_last_error()
  ST_ERR_TOO_LARGE = 3,  // exceeds a fixed capacity
  ST_ERR_DEVICE = 4,     // a device-side bounded wait or bounds check reported failure
};

#define ST_MAX_RANKS 8
/* csrc/comm/contrastive.cu */
typedef struct StPeerGroup {
  int world, rank;
  unsigned epoch;
  unsigned long long signals[ST_MAX_RANKS];
  unsigned long long signals_mc;
} StPeerGroup;

/* csrc/comm/tp_gemm.cu */
typedef struct StAgGemmArgs {
  StPeerGroup g;
  unsigned long long x_shard;                  // bf16 [T/W, K] contiguous (this rank's rows)
  unsigned long long gather_peers[ST_MAX_RANKS];  // bf16 [T, K] on every rank (symmetric)
  unsigned long long gather_mc;                // multicast alias of the gather buffer or 0
  unsigned long long B;                        // bf16 weights: [N, K] or, b_mn, [K, N]
  unsigned long long C;                        // bf16 [T, N]
  unsigned long long bias, aux_out, aux_in;    // optional epilogue operands (bf16)
  long long ldb, ldc, ld_aux_out, ld_aux_in;
  int T, N, K;
  int b_mn, act;
  float alpha;
  int sub_per_chunk;   // arrival granularity per rank shard (1, 2, 4, 8 or 16)
  int comm_ctas;       // unused (every CTA pushes a slice of the shard)
  int slot_enter, slot_arrive;   // slot_arrive: counter area of THIS sub_per_chunk value (world * 16 words)
  unsigned arrive_target;  // cumulative arrivals per counter: launches with this sub_per_chunk so far
                           // times st_ag_arrivals_per_launch()
  unsigned long long trace;  // optional device buffer of [3 * grid][4] 64-bit time stamps, or 0
  int stages;                // 0: choose by world size; 3 or 4: force that operand-pipeline depth
  int local_in_place;        // x_shard IS this rank's slot of its own gather buffer: nothing is copied locally
  int max_ctas;              // 0: one CTA per SM; > 0: a smaller grid, which leaves SMs to a concurrent kernel.  Every
                             // rank must pass the same value: the grid is also the arrival count per counter.
} StAgGemmArgs;

/* csrc/attention/attn_bwd.cu */
typedef struct StAttnBwdArgs {
  const void* Q; const void* K; const void* V; const void* O; const void* dO;
  const float* lse; float* delta; float* dQ_acc;
  void* dQ; void* dK; void* dV;
  long long q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, o_sb, o_ss, o_sh;
  long long do_sb, do_ss, do_sh, dq_sb, dq_ss, dq_sh, dk_sb, dk_ss, dk_sh, dv_sb, dv_ss, dv_sh;
  int B, H, Sq, Sk, D;
  float scale;
  int causal;
  // optional additive biases (fp32) and valid lengths (int32 [B]) of the forward pass; null = absent
  const float* key_bias;  long long kb_sb, kb_sh;
  const float* attn_bias; long long ab_sb, ab_sh, ab_sq;
  const int* lengths;
} StAttnBwdArgs;

/* csrc/attention/attn_fwd.cu */
typedef struct StAttnFwdArgs {
  const void* Q; const void* K; const void* V; void* O; float* lse;
  long long q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, o_sb, o_ss, o_sh;
  int B, H, Sq, Sk, D;
  float scale;
  int causal;
  // optional additive biases (fp32) and valid lengths (int32 [B]); all null = the plain kernel
  const float* key_bias;  long long kb_sb, kb_sh;            // [B, (H,) Sk]
  const float* attn_bias; long long ab_sb, ab_sh, ab_sq;     // [B, (H,) Sq, Sk], keys contiguous
  const int* lengths;
} StAttnFwdArgs;

/* csrc/conv/conv.cu */
typedef struct StConvArgs {
  const void* x;       // bf16 NHWC [N, H, W, C]
  const void* w;       // bf16 [OC, 9*C] (tap-major)
  const void* bias;    // bf16 [OC] or null
  void* y;             // bf16 NHWC [N, H, W, OC]
  const void* aux_in;  // bf16 [N*H*W, OC]: ReLU mask source for act == 4, or null
  int N, H, W, C, OC;
  int act;             // 0 none, 1 relu, 4 relu_bwd(aux_in)
} StConvArgs;

/* csrc/conv/conv.cu */
typedef struct StConvWgradArgs {
  const void* dy;   // bf16 [N*H*W, OC]
  const void* x;    // bf16 NHWC [N, H, W, C]
  float* dw;        // fp32 [OC, 9*C]; the kernel ADDS into it
  int N, H, W, C, OC;
  int splits;       // K splits over pixels (0 = choose)
} StConvWgradArgs;

/* csrc/comm/dp_step.cu */
typedef struct StDpStepArgs {
  StPeerGroup g;
  unsigned long long grad_local, grad_mc, grad_peers[ST_MAX_RANKS];
  unsigned long long w_local, w_mc, w_peers[ST_MAX_RANKS];
  unsigned long long master, m, v;
  long long n;
  float lr, beta1, beta2, eps, weight_decay, momentum;
  int step;
  float grad_scale;
  unsigned long long scale_ptr;
  int kind;
  int slot_enter, slot_exit;
  unsigned long long cta_counter;
  int max_ctas;
  // two-phase mode for global-norm clipping (phase 0 = the single fused pass, all fields below unused)
  int phase;                              // 1: reduce + squared norm into gred / sumsq_local; 2: clip + update + broadcast
  unsigned long long gred;                // fp32 [n / world] reduced gradient of this bucket's owned shard
  unsigned long long sumsq_local;         // fp32 word, zeroed by the caller at the start of the step
  unsigned long long norm_peers[ST_MAX_RANKS];   // symmetric fp32 [world] on every rank
  float max_norm;
} StDpStepArgs;

/* csrc/spectral/spectral.cu */
typedef struct StFftArgs {
  const float* in;
  float* out;
  const float* window;     // n coefficients or null
  long long in_b0, in_b1, in_i, out_b0, out_b1, out_i;
  int n, batch0, batch1, complex_in, inverse;
} StFftArgs;

/* csrc/gemm/gemm_sm100.cu */
typedef struct StGemmArgs {
  const void* A;      // bf16
  const void* B;      // bf16
  void* C;            // bf16 or fp32
  const void* bias;   // bf16 [N] or null
  const void* residual;  // bf16 [M,N] or null
  void* aux_out;      // bf16 [M,N] or null: receives alpha*acc+bias before the activation
  const void* aux_in; // bf16 [M,N]: pre-activation for ACT_*_BWD
  long long lda, ldb, ldc, ldr, ld_aux_out, ld_aux_in;  // leading dimensions in elements
  long long batch_stride_a, batch_stride_b, batch_stride_c;  // elements (batch > 1)
  int M, N, K, batch;
  int a_mn_major, b_mn_major;
  int out_fp32, accumulate, act;
  float alpha;
  int max_ctas;  // 0 = one CTA per SM; >0 limits the grid (leaves SMs to concurrent kernels)
} StGemmArgs;

/* csrc/comm/tp_gemm.cu */
typedef struct StGemmRsArgs {
  StPeerGroup g;
  unsigned long long A;                          // bf16 [T, K_local]
  unsigned long long B;                          // bf16 [N, K_local] or, b_mn, [K_local, N]
  unsigned long long stage_peers[ST_MAX_RANKS]; // bf16 [W][T/W, N] staging on every rank (symmetric)
  unsigned long long out;                        // bf16 [T/W, N] reduced shard (local)
  unsigned long long residual;                   // optional bf16 [T/W, N] added in the reduction
  long long lda, ldb;
  int T, N, K;
  int b_mn;
  float alpha;
  int slot_enter, slot_done;
  unsigned done_target;                          // cumulative warp arrivals expected per row block
  unsigned long long stage_mc;                   // unused
  unsigned long long trace;                      // optional [grid][4] 64-bit time stamps, or 0
  int groups;                                    // row-block groups per chunk for the remote / local interleave;
                                                 // 0 = choose (up to 8), 1 = all remote tiles first, local last
  int lag;                                       // groups by which a local group trails its remote group (0 = 1)
  int max_ctas;                                  // 0: one CTA per SM; > 0: a smaller grid (SMs left to a concurrent kernel)
} StGemmRsArgs;

/* csrc/comm/contrastive.cu */
typedef struct StInfoNceArgs {
  StPeerGroup g;
  unsigned long long anchors;                       // bf16 [R, D]
  unsigned long long positives;                     // bf16 [R, D] (this rank's shard)
  unsigned long long gather_peers[ST_MAX_RANKS];   // bf16 [W*R, D] on every rank
  unsigned long long gather_mc;
  unsigned long long partial;                       // fp32 [W*R/512][R][3] scratch
  unsigned long long counters;                      // u32 [R/128], zero before the first launch
  unsigned long long row_loss, row_lse;             // fp32 [R]
  int R, D;
  float inv_temperature;
  int slot_enter, slot_arrive;
  int comm_ctas;
  unsigned arrive_target;                           // cumulative arrivals expected per source rank
} StInfoNceArgs;

/* csrc/vision/vision.cu */
typedef struct StPreprocessArgs {
  int B, C, src_h, src_w, resize_h, resize_w, out_h, out_w, crop_y, crop_x, flip, do_jitter;
  float brightness, contrast, saturation, hue;
  float mean[4];
} StPreprocessArgs;

/* csrc/recurrent/scan.cu */
typedef struct StRnnScanArgs {
  const float* zx; const float* w_hh;
  float* h_all; float* hin_all; float* z_all; float* c_all;
  const float* dh_last; float* dz_all; float* dhin_all;
  int B, T, H, cell, dilation, backward;
} StRnnScanArgs;

/* csrc/host/tensor_abi.cpp */
typedef struct StRoundtableSummary {
  size_t above, here, beneath;
  float energy_above, energy_here, energy_beneath;
} StRoundtableSummary;

/* ---- libst_b200.so ---------------------------------------------------------------- */
int st_abi_version();   /* csrc/runtime/runtime.cu */
int st_act_bwd(const void* x, const void* dy, void* dx, long long n, int relu, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_act_fwd(const void* x, void* y, long long n, int relu, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_adamw(void* grad, int grad_is_bf16, float* master, float* m, float* v, void* weight, long long n, float lr, float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale, const float* scale_ptr, int zero_grad, void* stream_v);   /* csrc/optim/optim.cu */
int st_ag_arrivals_for(int max_ctas);   /* csrc/comm/tp_gemm.cu */
int st_ag_arrivals_per_launch();   /* csrc/comm/tp_gemm.cu */
int st_ag_gemm(const StAgGemmArgs* a, void* stream_v);   /* csrc/comm/tp_gemm.cu */
long long st_attn_bias_workspace(int B, int H, int Sk);   /* csrc/attention/attn_fwd.cu */
int st_attn_bwd(const StAttnBwdArgs* a, void* stream_v);   /* csrc/attention/attn_bwd.cu */
int st_attn_bwd_f32(const StAttnBwdArgs* a, const float* dO32, int grad_f32, float* bias_workspace, void* stream_v);   /* csrc/attention/attn_bwd.cu */
int st_attn_bwd_one_pass(const StAttnBwdArgs* a, const float* dO32, int grad_f32, float* bias_workspace, float* dq_workspace, void* stream_v);   /* csrc/attention/attn_bwd.cu */
long long st_attn_bwd_workspace(int B, int H, int Sq, int Sk, int D);   /* csrc/attention/attn_bwd.cu */
long long st_attn_bwd_workspace_f32(int B, int H, int Sq, int Sk, int D);   /* csrc/attention/attn_bwd.cu */
int st_attn_fwd(const StAttnFwdArgs* a, void* stream_v);   /* csrc/attention/attn_fwd.cu */
int st_attn_fwd_f32(const StAttnFwdArgs* a, float* out32, float* bias_workspace, void* stream_v);   /* csrc/attention/attn_fwd.cu */
int st_attn_fwd_get_pair_kernel();   /* csrc/attention/attn_fwd.cu */
int st_attn_fwd_read_trace(unsigned long long* out, int n);   /* csrc/attention/attn_fwd.cu */
void st_attn_fwd_set_pair_kernel(int on);   /* csrc/attention/attn_fwd.cu */
int st_attn_fwd_set_trace(int on);   /* csrc/attention/attn_fwd.cu */
int st_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream_v);   /* csrc/conv/conv.cu */
int st_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream_v);   /* csrc/conv/conv.cu */
int st_canvas_paint(const float* x, unsigned char* rgba, long long n, float lo, float hi, int palette, void* stream_v);   /* csrc/vision/vision.cu */
int st_ce_grad(const void* logits, const long long* target, const float* lse, const float* coef_ptr, float coef, void* dlogits, long long rows, long long ld, int V, int vocab_start, long long ignore_index, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_ce_stats(const void* logits, const long long* target, float* row_max, float* row_sum, float* tgt_logit, long long rows, long long ld, int V, int vocab_start, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_clip_coef(const float* sumsq, float norm_scale, float max_norm, float* coef, float* norm_out, void* stream_v);   /* csrc/optim/optim.cu */
int st_colsum(const void* x, float* out, long long rows, int cols, long long ld, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_colsum_short(const void* x, float* out, long long rows, int cols, long long ld, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_compact_rows(const float* in, float* out_v, int* out_i, int* counts, int rows, int cols, float low, float high, void* stream_v);   /* csrc/rank/rank.cu */
int st_contrastive_views(const float* base, const float* n1, const float* n2, float noise, void* out, long long n, void* stream_v);   /* csrc/elementwise/embed.cu */
int st_conv3x3_dgrad_weights(const void* w, void* wt, int OC, int IC, void* stream_v);   /* csrc/conv/conv.cu */
int st_conv3x3_fwd(const StConvArgs* a, void* stream_v);   /* csrc/conv/conv.cu */
int st_conv3x3_wgrad(const StConvWgradArgs* a, void* stream_v);   /* csrc/conv/conv.cu */
int st_dft_max_len();   /* csrc/spectral/spectral.cu */
int st_dp_step(const StDpStepArgs* s, void* stream_v);   /* csrc/comm/dp_step.cu */
int st_embedding_bwd(const long long* idx, const void* dy, float* dW, float* dpos, long long T, int d, int vocab_start, int vocab_local, int seq_len, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_embedding_bwd_sorted(const long long* uniq_ids, const long long* seg_start, const long long* seg_count, const long long* perm, const void* dy, float* dW, long long n_unique, int d, int vocab_start, int vocab_local, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_embedding_fwd(const long long* idx, const void* W, const void* pos, void* out, long long T, int d, int vocab_start, int vocab_local, int seq_len, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_fft_1d(const StFftArgs* a, void* stream_v);   /* csrc/spectral/spectral.cu */
int st_fft_max_len();   /* csrc/spectral/spectral.cu */
int st_frac_gl(const float* x, const float* w, float* y, int rows, int n, int m, float h_alpha, void* stream_v);   /* csrc/vision/vision.cu */
int st_gather_candidates(const void* vals, const void* idxs, float* dst_v, int* dst_i, int world, int rows, int k, void* stream_v);   /* csrc/rank/rank.cu */
int st_gemm_bf16(const StGemmArgs* a, void* stream_v);   /* csrc/gemm/gemm_sm100.cu */
int st_gemm_rs(const StGemmRsArgs* a, void* stream_v);   /* csrc/comm/tp_gemm.cu */
int st_gemm_rs_arrivals_per_launch(int world, int N);   /* csrc/comm/tp_gemm.cu */
int st_hyper_accumulate(float* g, const float* v, long long n, float curvature, float tol, float saturation, float porosity, int conformal, float scale, void* stream_v);   /* csrc/optim/optim.cu */
int st_hyper_apply(float* w, float* g, float* g_real, int rows, int cols, float curvature, float lr, float lr_real, float tol, float saturation, float porosity, void* stream_v);   /* csrc/optim/optim.cu */
int st_im2col3x3_planes(const void* x, void* col, const void* weights, void* padded, int N, int H, int W, int C, int OC, void* stream_v);   /* csrc/conv/conv.cu */
int st_im2col3x3_small(const void* x, void* col, int N, int H, int W, int C, int Kpad, void* stream_v);   /* csrc/conv/conv.cu */
int st_info_nce_fwd(const StInfoNceArgs* a, void* stream_v);   /* csrc/comm/contrastive.cu */
int st_info_nce_grad(const float* logits, const float* row_lse, const float* coef, void* dl, void* dl_t, int R, int C, int target_offset, void* stream_v);   /* csrc/comm/contrastive.cu */
const char* st_last_error();   /* csrc/runtime/runtime.cu */
int st_lstm_gate_bwd(const float* act, const float* c_prev, const float* c, const float* dh, const float* dc_next, float* dz, float* dc_prev, int B, int H, void* stream);   /* csrc/recurrent/recurrent.cu */
int st_lstm_gate_fwd(const float* z, const float* c_prev, float* c_out, float* h_out, float* act, int B, int H, void* stream);   /* csrc/recurrent/recurrent.cu */
int st_maxpool2_bwd(const void* dy, const void* idx, void* dx, int N, int H, int W, int C, void* stream_v);   /* csrc/conv/conv.cu */
int st_maxpool2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, void* stream_v);   /* csrc/conv/conv.cu */
int st_maxpool2_relu_bwd(const void* dy, const void* idx, const void* pooled, void* dx, float* dbias, int N, int H, int W, int C, void* stream_v);   /* csrc/conv/conv.cu */
int st_mse_backward(const float* p, const float* t, long long n, float* g, int* bad, void* stream_v);   /* csrc/elementwise/multi.cu */
int st_mse_blocks(long long n);   /* csrc/elementwise/multi.cu */
int st_mse_forward(const float* p, const float* t, long long n, float* value, void* workspace, int* bad, void* stream_v);   /* csrc/elementwise/multi.cu */
int st_mse_workspace();   /* csrc/elementwise/multi.cu */
int st_multi(int op, int count, const void* const* src, void* const* dst, const long long* n, float value, int* bad, void* stream_v);   /* csrc/elementwise/multi.cu */
int st_multi_blocks(long long most);   /* csrc/elementwise/multi.cu */
int st_multi_cast_bf16(int count, const void* const* src, void* const* dst, const long long* n, void* stream_v);   /* csrc/elementwise/multi.cu */
int st_multi_max();   /* csrc/elementwise/multi.cu */
int st_multi_step_bf16(int count, const void* const* src, void* const* dst, void* const* half, const long long* n, float value, void* stream_v);   /* csrc/elementwise/multi.cu */
int st_nce_rows(float* s, float* loss, int rows, float temperature, void* stream_v);   /* csrc/elementwise/embed.cu */
int st_nd_indexer(const unsigned* positions, unsigned* out_index, unsigned* out_segment, long long n, const unsigned* dims4, const unsigned* strides4, unsigned segments, unsigned segment_stride, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_nerf_composite_bwd(const float* sigma, const float* rad, const float* deltas, const float* accum, const float* d_accum, float* d_sigma, float* d_rad, int R, int S, float delta_scale, void* stream_v);   /* csrc/vision/vision.cu */
int st_nerf_composite_fwd(const float* sigma, const float* rad, const float* deltas, float* accum, int R, int S, float delta_scale, void* stream_v);   /* csrc/vision/vision.cu */
int st_nerf_sample(const float* rays, float* points, float* ts, float* deltas, int R, int S, int stratified, unsigned seed, void* stream_v);   /* csrc/vision/vision.cu */
int st_norm_bwd(int rms, const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_bwd_f32(int rms, const float* dy, const float* x, const float* gamma, const float* mean, const float* rstd, const float* dres, float* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_bwd_f32_rounded(int rms, const float* dy, const float* x, const float* gamma, const float* mean, const float* rstd, const float* dres, float* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_bwd_noalloc(int rms, const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx, float* dgamma, float* dbeta, int accumulate, int rows, int d, void* stream_v);   /* csrc/norm/norm.cu */
long long st_norm_bwd_scratch_elems(int rows, int d);   /* csrc/norm/norm.cu */
int st_norm_f32_max_features();   /* csrc/norm/norm.cu */
int st_norm_fwd(int rms, const void* x, const void* residual, const void* gamma, const void* beta, void* y, void* sum_out, float* mean, float* rstd, int rows, int d, float eps, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_fwd_f32(int rms, const float* x, const float* residual, const float* gamma, const float* beta, float* y, float* sum_out, float* mean, float* rstd, int rows, int d, float eps, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_fwd_f32_rounded(int rms, const float* x, const float* residual, const float* gamma, const float* beta, float* y, float* sum_out, float* mean, float* rstd, int rows, int d, float eps, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_gelu_bwd(const void* dy, const void* x, const void* gamma, const void* beta, const float* mean, const float* rstd, void* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_gelu_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows, int d, float eps, void* stream_v);   /* csrc/norm/norm.cu */
int st_norm_gelu_max_features();   /* csrc/norm/norm.cu */
int st_poincare_project(const float* x, float* y, int rows, int cols, float curvature, void* stream_v);   /* csrc/optim/optim.cu */
int st_preprocess(const float* in, float* out, const StPreprocessArgs* a, void* stream_v);   /* csrc/vision/vision.cu */
int st_preprocess_own_means(const float* in, float* out, const StPreprocessArgs* a, float* workspace, void* stream_v);   /* csrc/vision/vision.cu */
long long st_preprocess_workspace(int B, int src_h, int src_w);   /* csrc/vision/vision.cu */
int st_rank_select(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, void* stream_v);   /* csrc/rank/rank.cu */
int st_rank_topk(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, void* workspace, void* stream_v);   /* csrc/rank/rank.cu */
long long st_rank_topk_workspace(int rows, int cols, int k);   /* csrc/rank/rank.cu */
int st_read_error_word(unsigned* out, int clear);   /* csrc/runtime/runtime.cu */
int st_reduce_partials(const float* partial, float* out, int parts, int n, int accumulate, void* stream_v);   /* csrc/norm/norm.cu */
int st_rnn_scan(const StRnnScanArgs* a, void* stream_v);   /* csrc/recurrent/scan.cu */
int st_rnn_scan_supported(int H, int cell);   /* csrc/recurrent/scan.cu */
int st_rope(void* x, const float* cos_t, const float* sin_t, long long T, int heads, int D, long long ld, int seq_len, int pos_offset, int backward, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_row_normalize(const void* z, float* y, float* norm, int rows, int d, void* stream_v);   /* csrc/elementwise/embed.cu */
int st_row_normalize_bwd(const float* g, const float* y, const float* norm, void* dz, int rows, int d, void* stream_v);   /* csrc/elementwise/embed.cu */
int st_row_softmax_f32(const float* x, float* y, float* hard, int rows, int cols, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_row_softmax_spiral_f32(const float* x, float* y, float* hard, float* spiral, float* metrics, float* zmetrics, int rows, int cols, float phi, float phi_conj, float phi_bias, float leech_scale, float ramanujan_ratio, float golden_angle, void* stream_v);   /* csrc/elementwise/elementwise.cu */
int st_sequence_last_step(const float* src, float* dst, int B, int steps, int dim, int scatter, void* stream);   /* csrc/recurrent/recurrent.cu */
int st_set_wait_timeout_ns(unsigned long long ns);   /* csrc/runtime/runtime.cu */
int st_sgd(void* grad, int grad_is_bf16, float* master, float* mom, void* weight, long long n, float lr, float momentum, float weight_decay, float grad_scale, const float* scale_ptr, int nesterov, int zero_grad, void* stream_v);   /* csrc/optim/optim.cu */
int st_sm_count();   /* csrc/runtime/runtime.cu */
int st_specmul(const float* x_reim, float* y_reim, long long rows, int cols, float power, float h, int mode, void* stream_v);   /* csrc/spectral/spectral.cu */
int st_sumsq(const void* x, int is_bf16, long long n, float* out, void* stream_v);   /* csrc/optim/optim.cu */
int st_temporal_render(const float* voxels, const float* harmonics, const float* decay, float* out, long long n_voxels, int channels, int frames, float sample_rate_hz, void* stream_v);   /* csrc/spectral/spectral.cu */
int st_wave_gate_bwd(const float* z, const float* dy, float* dz, int B, int H, void* stream);   /* csrc/recurrent/recurrent.cu */
int st_wave_gate_fwd(const float* z, float* y, int B, int H, void* stream);   /* csrc/recurrent/recurrent.cu */

/* ---- libst_host.so ---------------------------------------------------------------- */
void spiraltorch_clear_last_error();   /* csrc/host/tensor_abi.cpp */
void spiraltorch_dlpack_drop_exported_state(void* managed);   /* csrc/host/tensor_abi.cpp */
size_t spiraltorch_last_error_length();   /* csrc/host/tensor_abi.cpp */
size_t spiraltorch_last_error_message(char* buffer, size_t capacity);   /* csrc/host/tensor_abi.cpp */
bool spiraltorch_roundtable_classify(const float* gradient, size_t len, size_t above_k, size_t here_k, size_t beneath_k, float tolerance, uint8_t* assignments, StRoundtableSummary* summary);   /* csrc/host/tensor_abi.cpp */
void spiraltorch_runtime_free(RuntimeHandle* rt);   /* csrc/host/tensor_abi.cpp */
RuntimeHandle* spiraltorch_runtime_new(size_t worker_threads, const char* thread_name);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_add(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_hadamard(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_add_relu(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, const SpiralTensor* residual);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_add_relu_with_backend(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, const SpiralTensor* residual, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_gelu(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_gelu_with_backend(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_relu(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_bias_relu_with_backend(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_matmul_with_backend(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_random_normal(const RuntimeHandle* rt, size_t rows, size_t cols, float mean, float std, uint64_t seed, bool has_seed);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_random_uniform(const RuntimeHandle* rt, size_t rows, size_t cols, float min, float max, uint64_t seed, bool has_seed);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_reshape(const RuntimeHandle* rt, const SpiralTensor* a, size_t rows, size_t cols);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_row_softmax(const RuntimeHandle* rt, const SpiralTensor* a, int /*backend*/);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_scale(const RuntimeHandle* rt, const SpiralTensor* a, float s);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_sub(const RuntimeHandle* rt, const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_runtime_tensor_transpose(const RuntimeHandle* rt, const SpiralTensor* a);   /* csrc/host/tensor_abi.cpp */
size_t spiraltorch_runtime_worker_count(const RuntimeHandle* rt);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_add(const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
bool spiraltorch_tensor_copy_column(const SpiralTensor* t, size_t index, float* out, size_t len);   /* csrc/host/tensor_abi.cpp */
bool spiraltorch_tensor_copy_data(const SpiralTensor* t, float* out, size_t len);   /* csrc/host/tensor_abi.cpp */
bool spiraltorch_tensor_copy_row(const SpiralTensor* t, size_t index, float* out, size_t len);   /* csrc/host/tensor_abi.cpp */
size_t spiraltorch_tensor_elements(const SpiralTensor* t);   /* csrc/host/tensor_abi.cpp */
void spiraltorch_tensor_free(SpiralTensor* t);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_from_dense(size_t rows, size_t cols, const float* data, size_t len);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_from_dlpack(void* managed);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_hadamard(const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul(const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_add_relu(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, const SpiralTensor* residual);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_add_relu_with_backend(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, const SpiralTensor* residual, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_gelu(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_gelu_with_backend(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_relu(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_bias_relu_with_backend(const SpiralTensor* a, const SpiralTensor* b, const float* bias, size_t n, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_matmul_with_backend(const SpiralTensor* a, const SpiralTensor* b, int backend);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_random_normal(size_t rows, size_t cols, float mean, float std, uint64_t seed, bool has_seed);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_random_uniform(size_t rows, size_t cols, float min, float max, uint64_t seed, bool has_seed);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_reshape(const SpiralTensor* a, size_t rows, size_t cols);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_row_softmax(const SpiralTensor* a, int /*backend*/);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_scale(const SpiralTensor* a, float s);   /* csrc/host/tensor_abi.cpp */
bool spiraltorch_tensor_shape(const SpiralTensor* t, size_t* rows_out, size_t* cols_out);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_sub(const SpiralTensor* a, const SpiralTensor* b);   /* csrc/host/tensor_abi.cpp */
void* spiraltorch_tensor_to_dlpack(const SpiralTensor* t);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_transpose(const SpiralTensor* a);   /* csrc/host/tensor_abi.cpp */
SpiralTensor* spiraltorch_tensor_zeros(size_t rows, size_t cols);   /* csrc/host/tensor_abi.cpp */
const char* spiraltorch_version();   /* csrc/host/tensor_abi.cpp */
int st_cobol_describe(void* handle, const float* values, int len, char** out_summary);   /* csrc/host/cobol_bridge.cpp */
void st_cobol_free_resonator(void* handle);   /* csrc/host/cobol_bridge.cpp */
void st_cobol_free_string(char* ptr);   /* csrc/host/cobol_bridge.cpp */
void* st_cobol_new_resonator(float curvature, float temperature);   /* csrc/host/cobol_bridge.cpp */
int st_host_atomic_write(const char* path, const void* data, int64_t len);   /* csrc/host/host_runtime.cpp */
void* st_host_loader_create(const float* features, const float* targets, int64_t rows, int64_t fcols, int64_t tcols, const int64_t* order, int64_t order_len, int64_t batch, int depth, int drop_last);   /* csrc/host/host_runtime.cpp */
void st_host_loader_destroy(void* h);   /* csrc/host/host_runtime.cpp */
int64_t st_host_loader_next(void* h, float* x, float* y);   /* csrc/host/host_runtime.cpp */
void* st_host_pool_create(int workers);   /* csrc/host/host_runtime.cpp */
void st_host_pool_destroy(void* p);   /* csrc/host/host_runtime.cpp */
void st_host_pool_stats(void* p, uint64_t* out3);   /* csrc/host/host_runtime.cpp */
uint64_t st_host_pool_submit(void* p, st_host_task_fn fn, void* arg);   /* csrc/host/host_runtime.cpp */
int st_host_pool_wait(void* p, uint64_t ticket, int64_t timeout_ms, int* status);   /* csrc/host/host_runtime.cpp */
int st_host_pool_workers(void* p);   /* csrc/host/host_runtime.cpp */
int st_host_rdv_all_reduce_sum(void* s, float* values, int64_t n, int64_t timeout_ms, int64_t* detail);   /* csrc/host/host_runtime.cpp */
uint64_t st_host_rdv_generation(void* s);   /* csrc/host/host_runtime.cpp */
int st_host_rdv_join(const char* group_id, int rank, int world, void** session, int64_t* detail);   /* csrc/host/host_runtime.cpp */
void st_host_rdv_leave(void* s);   /* csrc/host/host_runtime.cpp */
int st_host_rdv_registry_size();   /* csrc/host/host_runtime.cpp */

#ifdef __cplusplus
}
#endif
#endif /* SPIRALTORCH_B200_H */
