// C launch interface of the sm_100a kernels.  Every function enqueues work on
// `stream` and returns 0 or a cudaError_t / negative argument-error code; no
// function here allocates device memory unless its comment says so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

// ---- activation / unary op codes (shared by GEMM epilogues and elementwise kernels)
enum {
  FB_ACT_NONE = 0,
  FB_ACT_RELU = 1,
  FB_ACT_GELU = 2,  // tanh approximation, constants of ferrum-nn/src/activation.rs:254-262
  FB_ACT_SILU = 3,
  FB_ACT_TANH = 4,
  FB_ACT_SIGMOID = 5,
  FB_ACT_LEAKY_RELU = 6,
  FB_ACT_ELU = 7,
  FB_UNARY_NEG = 8,
  FB_UNARY_EXP = 9,
  FB_UNARY_LOG = 10,
  FB_UNARY_SQRT = 11,
  FB_UNARY_ABS = 12,
  FB_UNARY_SIN = 13,
  FB_UNARY_COS = 14,
  FB_UNARY_POW = 15,         // x ** alpha
  FB_UNARY_ADD_SCALAR = 16,  // x + alpha
  FB_UNARY_MUL_SCALAR = 17,  // x * alpha
  FB_UNARY_RSUB_SCALAR = 18, // alpha - x
  FB_UNARY_RDIV_SCALAR = 19, // alpha / x
  FB_UNARY_AFFINE = 20,      // x * alpha + beta   (Normalize / Scale transforms)
  FB_UNARY_CLAMP = 21,       // min(max(x, alpha), beta)
};

enum { FB_BIN_ADD = 0, FB_BIN_SUB = 1, FB_BIN_MUL = 2, FB_BIN_DIV = 3, FB_BIN_POW = 4, FB_BIN_MAX = 5, FB_BIN_MIN = 6 };
enum { FB_RED_SUM = 0, FB_RED_MEAN = 1, FB_RED_MAX = 2, FB_RED_MIN = 3, FB_RED_PROD = 4 };
enum { FB_DT_F32 = 0, FB_DT_BF16 = 3 };  // values follow ferrum-core/src/dtype.rs:31-40
enum { FB_LOSS_MSE = 0, FB_LOSS_BCE = 1, FB_LOSS_L1 = 2, FB_LOSS_SMOOTH_L1 = 3 };

// ---- GEMM -----------------------------------------------------------------
// tcgen05/TMEM bf16 GEMM: out[M,N] = act(A*B^T + bias) (+= out when beta).
// lda/ldb are the row pitches (elements) of the stored matrices: a K-major
// operand is stored [rows=M|N][K], an MN-major operand is stored [rows=K][M|N].
int fb_gemm_bf16_supported(const void* a, const void* b, long long lda, long long ldb);
// out2 (optional, bf16 outputs without accumulate): receives act'(A*B^T + bias) in the layout of out, for
// blocks whose backward would otherwise re-evaluate the activation.
int fb_gemm_bf16(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N, int K,
                 long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_bf16, int act,
                 int beta, int max_ctas, int32_t* status, cudaStream_t stream);
// fp32 operands on the tensor cores as TF32 (tcgen05.mma kind::tf32), fp32 result; lda / ldb multiples of 4.
int fb_gemm_tf32(const float* a, const float* b, float* out, const float* bias, int M, int N, int K, long long lda,
                 long long ldb, long long ldc, int a_mn_major, int b_mn_major, int act, int beta, int max_ctas,
                 int32_t* status, cudaStream_t stream);
int fb_gemm_tf32_2cta(const float* a, const float* b, float* out, const float* bias, int M, int N, int K, long long lda,
                 long long ldb, long long ldc, int a_mn_major, int b_mn_major, int act, int beta, int max_ctas,
                 int32_t* status, cudaStream_t stream);
// CTA-pair variant (tcgen05 cta_group::2; 256 x 256 tiles on two SMs, 256 x 128 for small outputs); same
// arguments.  Returns -3 where clusters of two CTAs cannot be scheduled.  fb_gemm_bf16_2cta_pairs() = resident pairs.
int fb_gemm_bf16_2cta(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N, int K,
                      long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_bf16,
                      int act, int beta, int max_ctas, int32_t* status, cudaStream_t stream);
int fb_gemm_bf16_2cta_pairs(void);
// Timing record of the CTA-pair kernel: 4 x 64-bit words per pair (ns): MMA thread waiting for a drained accumulator,
// waiting for operands, one epilogue warp busy, whole kernel.  NULL switches it off.
void fb_gemm_bf16_2cta_set_profile(unsigned long long* buffer);
// Tiles are walked in groups of `group_m` 256-row blocks x all column blocks (default 8); returns the previous
// value, values < 1 only query.
int fb_gemm_bf16_2cta_set_group_m(int group_m);
// Batched form over batch_outer x batch_inner slices: out[s] = alpha * A[s] * B[s]^T (+= out[s] when beta).
// Each operand carries its own (outer, inner) slice strides in elements, so head-interleaved [B, S, H, D]
// activations are multiplied in place.  Slice strides of A and B must be multiples of 8 elements.
int fb_gemm_bf16_batched(const void* a, const void* b, void* out, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, int batch_outer, int batch_inner, long long sa_outer, long long sa_inner,
                         long long sb_outer, long long sb_inner, long long sc_outer, long long sc_inner,
                         int a_mn_major, int b_mn_major, int out_bf16, int beta, float alpha, int32_t* status,
                         cudaStream_t stream);
// fp32 GEMM of fp32 precision on the tensor cores (three bf16 parts per operand element, gemm/f32_tensor_gemm.cu):
// out[s] = act(alpha * A[s] B[s]^T + bias) (+= when beta), any element strides; s = (outer, inner) batch slice.
int fb_gemm_f32_tensor(const float* a, const float* b, float* out, const float* bias, int M, int N, int K,
                       long long sam, long long sak, long long sbn, long long sbk, long long ldc, int act, int beta,
                       float alpha, int batch_outer, int batch_inner, long long sa_outer, long long sa_inner,
                       long long sb_outer, long long sb_inner, long long sc_outer, long long sc_inner,
                       int32_t* status, cudaStream_t stream);
// The same kernel on bf16 operands of any alignment and strides, one bf16 product per k-block: operands that a TMA map
// cannot describe.  out: bf16 (no accumulation onto it) or fp32.
int fb_gemm_bf16_any(const void* a, const void* b, void* out, const float* bias, int M, int N, int K, long long sam,
                     long long sak, long long sbn, long long sbk, long long ldc, int out_bf16, int act, int beta,
                     int32_t* status, cudaStream_t stream);
// bf16 products of few output tiles: the K splits of a tile meet in a cluster (gemm/splitk_gemm.cu).  Arguments as
// fb_gemm_bf16; tile: 0 = chosen by size, 16 / 32 / 64 = rows of A against 128 rows of B, 192 / 256 = 128 rows of A
// against 64 / 128 rows of B.
int fb_gemm_bf16_splitk_use(int M, int N, int K);  // 1: faster than fb_gemm_bf16 / _2cta for this product
int fb_gemm_bf16_splitk(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N, int K,
                        long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_bf16,
                        int act, int beta, int tile, int32_t* status, cudaStream_t stream);
// The same tiles without the splits: the bits of fb_gemm_bf16.
int fb_gemm_bf16_narrow_use(int M, int N, int K);  // 1: faster than fb_gemm_bf16 for this product
int fb_gemm_bf16_narrow(const void* a, const void* b, void* out, void* out2, const float* bias, int M, int N, int K,
                        long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_bf16,
                        int act, int beta, int tile, int32_t* status, cudaStream_t stream);
// fp32 SIMT GEMM with arbitrary element strides (parity runs, odd shapes):
// out[m,n] = act(sum_k A[m*sam + k*sak] * B[k*sbk + n*sbn] + bias[n]) (+= out when beta).
int fb_gemm_f32_simt(const float* a, const float* b, float* out, const float* bias, int M, int N, int K,
                     long long sam, long long sak, long long sbk, long long sbn, long long ldc, int act, int beta,
                     int batch, long long batch_stride_a, long long batch_stride_b, long long batch_stride_c,
                     cudaStream_t stream);

// ---- elementwise ------------------------------------------------------------
int fb_unary_fwd(const void* x, void* y, long long n, int op, float alpha, float beta, int dtype,
                 cudaStream_t stream);
// dx = dy * f'(.) ; `saved` is x or y depending on the op (see elementwise.cu).
// y = x * (*scalar) with the factor read on the device (fp32 or bf16 data).
int fb_scale_by_device_scalar(const void* x, const float* scalar, void* y, long long n, int dtype,
                              cudaStream_t stream);
int fb_unary_bwd(const void* dy, const void* saved, void* dx, long long n, int op, float alpha, float beta,
                 int dtype, cudaStream_t stream);
// Broadcasting binary op over up to 6 dims; strides in elements, 0 = broadcast.
int fb_binary_fwd(const float* a, const float* b, float* out, int op, int ndim, const long long* shape,
                  const long long* stride_a, const long long* stride_b, cudaStream_t stream);
int fb_cast(const void* src, void* dst, long long n, int src_dtype, int dst_dtype, cudaStream_t stream);
int fb_repack_rows(const void* src0, void* dst0, long long rows0, int cols0, long long pitch0, const void* src1, void* dst1,
                   long long rows1, int cols1, long long pitch1, cudaStream_t stream);
int fb_transpose_2d(const void* src, void* dst, int rows, int cols, int elem_size, cudaStream_t stream);

// ---- reductions: input viewed as [outer, R, inner] --------------------------
// `scratch` (may be NULL) lets the kernel split R over several blocks when there are
// few outputs; fb_reduce_scratch_elems() says how many floats that takes (0 = none).
long long fb_reduce_scratch_elems(long long outer, long long R, long long inner);
int fb_reduce(const float* x, float* out, long long outer, long long R, long long inner, int op, float* scratch,
              long long scratch_elems, cudaStream_t stream);
int fb_arg_reduce(const float* x, long long* idx, float* val, long long outer, long long R, long long inner,
                  int is_max, cudaStream_t stream);
// dx = dy * act'(y) of a ReLU, tanh or sigmoid, and its column sums; -3, nothing launched: these want fb_colsum.
int fb_unary_bwd_colsum(const void* dy, const void* y, void* dx, float* sums, long long rows, long long cols, int op, int dtype,
                        cudaStream_t stream);
// Column sums of a [rows, cols] matrix (fp32 or bf16 in, fp32 out): bias gradients.
int fb_colsum_clusters(long long rows, long long cols, int dtype, int grad, int aligned);  // a query
int fb_colsum(const void* x, float* out, long long rows, long long cols, int dtype, int accumulate,
              cudaStream_t stream);

// ---- normalisation ------------------------------------------------------------
// Where the wide-row kernels (shared-memory ring fed by bulk async copies) report a wait that gave up.
void fb_layernorm_set_status(int32_t* status);
// pre_act: FB_ACT_NONE or FB_ACT_GELU applied to x before normalising (fused block).
int fb_layernorm_fwd(const void* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd,
                     long long rows, int cols, float eps, int pre_act, int dtype, cudaStream_t stream);
// stats = [3][cols]: d_gamma, d_beta, column sum of dx (added to, or written where want_colsum has the bit 2); partial = [nblk][3][cols] workspace.
// act_grad (optional, dtype of x; excludes pre_act): x holds act(z) and act_grad holds act'(z) as written by
// the producing GEMM's epilogue; dx is then the gradient of z.
int fb_layernorm_bwd(const void* dy, const void* x, const void* act_grad, const float* gamma, const float* mean,
                     const float* rstd, void* dx, float* partial, float* stats, long long rows, int cols,
                     int pre_act, int dtype, int nblk, int want_colsum, cudaStream_t stream);
int fb_layernorm_bwd_blocks(long long rows, int cols);
int fb_add_layernorm_fwd(const float* x, const void* r, const float* gamma, const float* beta, float* sum, float* y,
                         float* mean, float* rstd, long long rows, int cols, float eps, int r_dtype, cudaStream_t stream);
int fb_add_layernorm_bwd(const float* dy, const float* sum, const float* gamma, const float* mean, const float* rstd,
                         float* dx, void* dx_low, float* partial, float* stats, long long rows, int cols, int nblk,
                         cudaStream_t stream);
int fb_batchnorm_fwd(const float* x, const float* gamma, const float* beta, float* y, float* save_mean,
                     float* save_rstd, float* running_mean, float* running_var, long long rows, int cols,
                     float eps, float momentum, int training, cudaStream_t stream);
int fb_batchnorm_bwd(const float* dy, const float* x, const float* gamma, const float* save_mean,
                     const float* save_rstd, float* dx, float* dgamma, float* dbeta, long long rows, int cols,
                     cudaStream_t stream);

// ---- softmax / losses -----------------------------------------------------------
int fb_softmax_fwd(const void* x, void* y, long long rows, int cols, int log_mode, int dtype, cudaStream_t stream);
int fb_softmax_bwd(const void* dy, const void* y, void* dx, long long rows, int cols, int log_mode, int dtype,
                   cudaStream_t stream);
// Mean losses (kernels/mean_loss.cu): the scalar scale * sum lands in `loss`; workspace = fb_mean_loss_workspace(n)
// floats.  dlogits (optional, of the logits' type): (softmax - onehot) * scale.  gout: the incoming scalar gradient, read
// on the device.
long long fb_mean_loss_workspace(long long n);
int fb_ce_fwd(const void* logits, const long long* labels, void* dlogits, float* loss, float* workspace, long long rows,
              int cols, float scale, int dtype, cudaStream_t stream);
// a target outside [0, cols) is reported to the status block and makes the loss NaN
int fb_nll_fwd(const void* log_probs, const long long* target, float* loss, float* workspace, long long rows, int cols,
               float scale, int dtype, int32_t* status, cudaStream_t stream);
int fb_nll_bwd(const long long* target, const float* gout, void* dlog_probs, long long rows, int cols, float scale,
               int dtype, cudaStream_t stream);
int fb_loss_mean_fwd(const float* pred, const float* target, float* loss, float* workspace, long long n, int kind,
                     float scale, cudaStream_t stream);
// Gradient of the mean elementwise losses.
int fb_loss_bwd(const float* pred, const float* target, const float* gout, float* dpred, long long n, int kind,
                float scale, cudaStream_t stream);

// ---- secondary layers: recurrent gates, convolution lowering, pooling ---------
// LSTM: pre-activations xi + hh laid out [B, 4H] as (input, forget, cell, output); `gates` receives the
// activated gates for the backward pass.  dh / dc may be NULL (no gradient from that output).
int fb_lstm_gates_fwd(const float* xi, const float* hh, const float* c_prev, float* h_out, float* c_out,
                      float* gates, long long B, int H, cudaStream_t stream);
int fb_lstm_gates_bwd(const float* dh, const float* dc, const float* gates, const float* c_prev, const float* c_out,
                      float* dpre, float* dc_prev, long long B, int H, cudaStream_t stream);
// GRU: xi, hh are [B, 3H] as (reset, update, new); `saved` is [B, 4H] (r, z, n, hn).
int fb_gru_gates_fwd(const float* xi, const float* hh, const float* h_prev, float* h_out, float* saved, long long B,
                     int H, cudaStream_t stream);
int fb_gru_gates_bwd(const float* dh, const float* saved, const float* h_prev, float* dxi, float* dhh,
                     float* dh_prev, long long B, int H, cudaStream_t stream);
// Whole sequences (kernels/rnn_seq.cu), gates = 4 (LSTM) or 3 (GRU): xi [T, B, gates H] input projections, w_t [H,
// gates H] transposed recurrent matrix, hs [T, B, H]; hs_kept (a second hs, so that the first is the caller's) / cs /
// saved / c_last as the backward call reads them (NULL: not kept).  Backward: w [gates H, H]; dxi and, for GRU, dhh [T, B, gates H].  h0, c0 and the incoming gradients may be NULL.
int fb_rnn_seq_supported(int gates, int B, int H);
// The instance that runs: batch rows per cluster (1, 2, 4, 8), + 16: weights in registers, + 32: a full share of them in
// every thread (the unrolled product); 0: not supported.
int fb_rnn_seq_plan(int gates, int B, int H, int backward);
int fb_rnn_seq_fwd(int gates, const float* xi, const float* w_t, const float* bias, const float* h0, const float* c0,
                   float* hs, float* hs_kept, float* cs, float* saved, float* c_last, int T, int B, int H,
                   int32_t* status, cudaStream_t stream);
int fb_rnn_seq_bwd(int gates, const float* w, const float* h0, const float* c0, const float* hs, const float* cs,
                   const float* saved, const float* d_hs, const float* d_c_last, float* dxi, float* dhh, float* dh0,
                   float* dc0, int T, int B, int H, int32_t* status, cudaStream_t stream);
// Window matrix of a convolution: cols[B*Ho*Wo, C*kh*kw] (row pitch ldk elements, fp32 or bf16) and its gradient.
int fb_im2col(const float* x, void* cols, int B, int C, int H, int W, int kh, int kw, int Ho, int Wo, int sh, int sw,
              int ph, int pw, int dh, int dw, long long ldk, int out_dtype, cudaStream_t stream);
int fb_col2im(const float* dcols, float* dx, int B, int C, int H, int W, int kh, int kw, int Ho, int Wo, int sh,
              int sw, int ph, int pw, int dh, int dw, long long ldk, cudaStream_t stream);
// 2-D pooling without padding; op 0 = max (arg receives the winner's offset inside its plane), 1 = average.
int fb_pool2d_fwd(const float* x, float* y, int* arg, int B, int C, int H, int W, int kh, int kw, int Ho, int Wo,
                  int sh, int sw, int op, cudaStream_t stream);
int fb_pool2d_bwd(const float* dy, const int* arg, float* dx, int B, int C, int H, int W, int kh, int kw, int Ho,
                  int Wo, int sh, int sw, int op, cudaStream_t stream);

// ---- dropout / embedding / collate ---------------------------------------------
int fb_dropout_fwd(const void* x, void* y, uint8_t* mask, long long n, float p, unsigned long long seed,
                   unsigned long long offset, int dtype, cudaStream_t stream);
// Graph-capturable dropout: Philox offset = offset + *dev_counter; the counter advances on the stream after the launch.
int fb_dropout_fwd_dyn(const void* x, void* y, uint8_t* mask, long long n, float p, unsigned long long seed,
                       unsigned long long offset, unsigned long long* dev_counter, int dtype, cudaStream_t stream);
int fb_dropout_bwd(const void* dy, const uint8_t* mask, void* dx, long long n, float p, int dtype,
                   cudaStream_t stream);
int fb_embedding_fwd(const float* weight, const long long* idx, void* out, long long n_idx, int dim,
                     long long vocab, long long padding_idx, int out_dtype, int32_t* status, cudaStream_t stream);
// Mean over `seq` consecutive indices: out[b] = mean_s W[idx[b, s]].
int fb_embedding_meanpool_fwd(const float* weight, const long long* idx, void* out, long long batch, int seq,
                              int dim, long long vocab, int out_dtype, cudaStream_t stream);
// dW[idx[i]] += scale * dout[i / group].  Pairs of an index (vocab where it is no row of the table) and its row of dout, i / group,
// sorted by index:
int fb_embedding_pairs(const long long* idx, int32_t* keys, int32_t* rows, long long n, long long vocab, long long group,
                       cudaStream_t stream);
int fb_embedding_bwd_pairs(const void* dout, const int32_t* keys, const int32_t* rows, float* dweight, long long n_idx,
                           int dim, int group, float scale, long long padding_idx, long long vocab, int dtype,
                           cudaStream_t stream);
// The same into a table that holds zeros.
int fb_embedding_bwd_pairs_zeroed(const void* dout, const int32_t* keys, const int32_t* rows, float* dweight, long long n_idx,
                                  int dim, int group, float scale, long long padding_idx, long long vocab, int dtype,
                                  cudaStream_t stream);
// The same for sorted indices of 64 bits and their original positions.
int fb_embedding_bwd_sorted(const void* dout, const long long* sorted_idx, const long long* perm, float* dweight, long long n_idx,
                            int dim, int group, float scale, long long padding_idx, long long vocab, int dtype,
                            cudaStream_t stream);
// Blockwise attention forward (tcgen05, head dimension 64, bf16): out[B, Sq, H, 64] = softmax(scale q k^T) v for
// [B, H, S, 64] views given by element strides; lse (optional) [B, H, Sq].  -2: operand not describable by TMA.
int fb_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int H, int Sq, int Skv,
                     int D, long long q_sb, long long q_sh, long long q_ss, long long k_sb, long long k_sh,
                     long long k_ss, long long v_sb, long long v_sh, long long v_ss, float scale, int causal,
                     int32_t* status, cudaStream_t stream);
// Gradients of the blockwise attention (attention_bwd.cu), D = 64 or 128: out / d_out [B, Sq, H, D] contiguous bf16, lse as
// written by fb_attention_fwd, delta = [B, H, Sq] fp32 scratch filled by the call; dq [B, Sq, H, D], dk / dv [B, Skv, H, D].
int fb_attention_bwd(const void* q, const void* k, const void* v, const void* out, const void* d_out,
                     const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int H, int Sq, int Skv,
                     int D, long long q_sb, long long q_sh, long long q_ss, long long k_sb, long long k_sh, long long k_ss,
                     long long v_sb, long long v_sh, long long v_ss, float scale, int causal, int32_t* status,
                     cudaStream_t stream);
int fb_attention_bwd_map_error(void);
// Stride-1 convolution as an implicit GEMM (gemm/tcgen05_gemm.cu) over NHWC bf16 operands with channel counts padded
// to multiples of 8, its weight gradient, and the layout changes from / to NCHW fp32 (kernels/conv_layout.cu).
int fb_conv_igemm(const void* x, const void* w, void* y, const float* bias, int B, int H, int W, int Cp, int O, int kh,
                  int kw, int ph, int pw, int dh, int dw, long long ldy, int out_bf16, int32_t* status,
                  cudaStream_t stream);
// With an activation, a mask (bf16, laid out like y: results count where it is above zero) or an fp32 y that is added to.
int fb_conv_igemm_epilogue(const void* x, const void* w, void* y, const float* bias, const void* mask, int B, int H, int W,
                           int Cp, int O, int kh, int kw, int ph, int pw, int dh, int dw, long long ldy, int out_bf16, int act,
                           int beta, int32_t* status, cudaStream_t stream);
int fb_conv_wgrad_splits(int B, int Ho, int Wo, int O, int Cp, int taps);
int fb_conv_wgrad(const void* dy, const void* x, float* out, int B, int H, int W, int Cp, int O, int Op, int kh, int kw,
                  int ph, int pw, int dh, int dw, int32_t* status, cudaStream_t stream);
// A convolution of any stride becomes one of stride 1 by a space-to-depth arrangement (conv_layout.cu).
int fb_conv_pack_input(const float* x, const float* mask, void* z, int B, int C, int H, int W, int sh, int sw, int eh,
                       int ew, int ph, int pw, int Hz, int Wz, long long ld, cudaStream_t stream);
// The same of a gradient behind a ReLU whose mask is bytes (fb_nhwc_to_nchw_masks); stride 1, no padding.
int fb_conv_pack_masked(const float* x, const unsigned char* mask, void* z, int B, int C, int H, int W, long long ld,
                        cudaStream_t stream);
int fb_conv_pack_filters(const float* w, void* out, int O, int C, int kh, int kw, int sh, int sw, int eh, int ew, int pitch,
                         int dgrad, cudaStream_t stream);
int fb_conv_fold_wgrad(const float* part, float* dw, int splits, int O, int C, int kh, int kw, int sh, int sw, int eh,
                       int ew, int pitch, cudaStream_t stream);
int fb_s2d_nhwc_to_nchw_f32(const float* z, float* x, int B, int C, int H, int W, int sh, int sw, int eh, int ew, int ph,
                            int pw, int Hz, int Wz, long long ld, cudaStream_t stream);
int fb_s2d_nhwc_to_nchw_add(const float* z, const float* add, float* x, int B, int C, int H, int W, int sh, int sw, int eh, int ew,
                            int ph, int pw, int Hz, int Wz, long long ld, cudaStream_t stream);
int fb_nhwc_to_nchw_f32(const float* x, const float* add, float* y, int B, int C, long long P, long long ld, int relu,
                        cudaStream_t stream);
// add counts where add_mask is set; mask is set where y is above zero (both optional, bytes).
int fb_nhwc_to_nchw_masks(const float* x, const float* add, const unsigned char* add_mask, float* y, unsigned char* mask, int B,
                          int C, long long P, long long ld, int relu, cudaStream_t stream);
int fb_gather_rows(const void* src, const long long* idx, void* dst, long long n_idx, long long row_bytes,
                   long long n_rows, int32_t* status, cudaStream_t stream);

// ---- optimizers (multi-tensor; chunk tables built on the host) -------------------
typedef struct {
  float lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2, grad_scale;
} fb_adam_hparams;
typedef struct {
  float lr, momentum, weight_decay, grad_scale;
  int nesterov, first_step;
} fb_sgd_hparams;
int fb_adam_flat(float* p, const float* g, float* m, float* v, void* shadow, long long n,
                 fb_adam_hparams h, cudaStream_t stream);
int fb_sgd_flat(float* p, const float* g, float* buf, void* shadow, long long n, fb_sgd_hparams h,
                cudaStream_t stream);
// Pointer-table variants: tensors[i] described by ptrs (device arrays of length ntensors).
int fb_adam_multi(float* const* p, const float* const* g, float* const* m, float* const* v,
                  void* const* shadow, const long long* sizes, int ntensors, fb_adam_hparams h,
                  cudaStream_t stream);
int fb_sgd_multi(float* const* p, const float* const* g, float* const* buf, void* const* shadow,
                 const long long* sizes, int ntensors, fb_sgd_hparams h, cudaStream_t stream);
// Graph-capturable forms: the step-dependent factors are device scalars dyn = {lr, bias_corr1, bias_corr2,
// beta1^t, beta2^t, t} (initialise to {lr, 0, 0, 1, 1, 0}); fb_optim_advance moves them one step on the stream
// before the update launches, so a captured step replays correctly.  SGD only reads dyn[0] (lr).
int fb_optim_advance(float* dyn, float beta1, float beta2, cudaStream_t stream);
int fb_adam_multi_dyn(float* const* p, const float* const* g, float* const* m, float* const* v,
                      void* const* shadow, const long long* sizes, int ntensors, fb_adam_hparams h,
                      const float* dyn, cudaStream_t stream);
int fb_sgd_multi_dyn(float* const* p, const float* const* g, float* const* buf, void* const* shadow,
                     const long long* sizes, int ntensors, fb_sgd_hparams h, const float* dyn, cudaStream_t stream);

// ---- AMP helpers -----------------------------------------------------------------
int fb_unscale_check(float* const* g, const long long* sizes, int ntensors, float inv_scale, float* found_inf,
                     cudaStream_t stream);
int fb_sumsq_multi(const float* const* g, const long long* sizes, int ntensors, float* out, cudaStream_t stream);
int fb_scale_multi(float* const* g, const long long* sizes, int ntensors, const float* total_sumsq,
                   float max_norm, float clip_value, int mode, cudaStream_t stream);

#ifdef __cplusplus
}
#endif
