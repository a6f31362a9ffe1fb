// Public convolution / GEMM entry points.  Each picks the kernel family for the shape: the
// tcgen05 tensor-core kernels when the shape meets their alignment rules, otherwise the
// general CUDA-core kernels.  Both families run on the GPU; there is no host fallback.
#include "common.cuh"
#include "kernels.h"

namespace {

// Scratch of the two-term products for one direction, 0 where they do not take it.  Their channel counts are those that fit no
// block of 32, whatever else keeps the TF32 kernels from a call (a small or an unaligned tensor: CUDA cores).  The size that a
// caller is told and the choice of the kernel both rest on this number, so that the choice never depends on how much
// scratch more than that the caller happens to pass.
long long split_scratch_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction) {
  if (direction == 1 ? cout % 32 == 0 && cin % 4 == 0 : cin % 32 == 0 && cout % 4 == 0) return 0;
  return mtb_split_workspace_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, direction);
}

}  // namespace

MTB_API long long mtb_conv2d_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  // no such convolution: the call that the scratch is for says so
  if (n <= 0 || cin <= 0 || cout <= 0 || kh <= 0 || kw <= 0 || sh <= 0 || sw <= 0 || !mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw)) return 0;
  long long a = mtb_conv2d_wgrad_simt_workspace_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  long long b = mtb_tc_conv2d_workspace_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  for (int direction = 0; direction < 3; ++direction) {
    const long long c = split_scratch_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, direction);
    if (c > b) b = c;
  }
  return a > b ? a : b;
}

namespace {

// Whether the two-term products take this convolution: they need the scratch (a caller without it gets the CUDA-core kernels).
bool split_takes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction, const void* workspace,
                 long long workspace_bytes) {
  if (!workspace || !mtb_aligned16(workspace) || n <= 0 || cin <= 0 || cout <= 0 || kh <= 0 || kw <= 0 || sh <= 0 || sw <= 0 || ph < 0 || pw < 0 ||
      !mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw))
    return false;
  const long long need = split_scratch_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, direction);
  return need > 0 && workspace_bytes >= need;
}

// Forward of the shapes that the TF32 kernels do not take.
int forward_fp32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt, const float* bias,
                 float* y, int relu, void* workspace, long long workspace_bytes, void* stream) {
  const int* guard = nullptr;
  int guards = 0;
  if (!(x && wt && y && split_takes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, 0, workspace, workspace_bytes)))
    return mtb_conv2d_forward_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, nullptr, nullptr, stream, nullptr, 0);
  const MtbScratchTurn turn;
  if (int rc = mtb_split_conv2d_forward_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, (cudaStream_t)stream, &guard, &guards))
    return rc;
  return mtb_conv2d_forward_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, nullptr, nullptr, stream, guard, guards);
}

int dgrad_fp32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy, const float* wt, float* dx,
               void* workspace, long long workspace_bytes, void* stream) {
  const int* guard = nullptr;
  int guards = 0;
  if (!(dy && wt && dx && split_takes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, 1, workspace, workspace_bytes)))
    return mtb_conv2d_dgrad_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, stream, nullptr, 0);
  const MtbScratchTurn turn;
  if (int rc = mtb_split_conv2d_dgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, workspace, (cudaStream_t)stream, &guard, &guards)) return rc;
  return mtb_conv2d_dgrad_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, stream, guard, guards);
}

}  // namespace

// workspace (may be NULL): scratch of mtb_conv2d_workspace_bytes() for the weight gradient, and for the operands of channel counts
// that fit no block of 32 (tc_split.cuh); without it forward and data gradient of those run on the CUDA cores.
MTB_API int mtb_conv2d_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                   const float* wt, const float* bias, float* y, int relu, void* workspace, long long workspace_bytes,
                                   void* stream) {
  if (mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, y))
    return mtb_tc_conv2d_forward_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, workspace_bytes, stream);
  return forward_fp32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, workspace_bytes, stream);
}

// Forward convolution that also prepares the batch statistics of its output for a BatchNorm layer
// that follows (the statistics pass of BatchNorm re-reads the whole activation otherwise).  stats:
// room for mtb_conv2d_stats_max_rows() x 3 x cout floats; *stats_rows (HOST) receives the number of
// partial rows [row][3][cout] = (count, mean, M2) written, to be passed to
// mtb_batch_norm2d_forward_prestats_f32, or 0 when this shape's kernel does not produce them (the
// caller then runs the ordinary BatchNorm forward).
MTB_API int mtb_conv2d_stats_max_rows() { return 4 * mtb_sm_count(); }

MTB_API int mtb_conv2d_forward_stats_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                         const float* wt, const float* bias, float* y, int relu, float* stats, int* stats_rows, void* workspace,
                                         long long workspace_bytes, void* stream) {
  MTB_REQUIRE(stats && stats_rows, "conv2d_forward_stats: stats buffer and row counter are required");
  *stats_rows = 0;
  if (mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, y))
    return mtb_tc_conv2d_forward_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, workspace_bytes, stream, stats,
                                     stats_rows);
  return forward_fp32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, workspace_bytes, stream);
}

// Inference: y = relu?(batch_norm(conv(x)) + residual), BatchNorm with running statistics, in one launch.  The epilogue applies
// the BatchNorm kernels' own expression to the value it would have stored, so the bits are those of the separate
// operators; what goes is the write and the read of the convolution's output and two launches.
MTB_API int mtb_conv2d_bn_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                      const float* wt, const float* bias, const float* gamma, const float* beta, const float* running_mean,
                                      const float* running_var, double eps, const float* residual, int relu, float* y, void* workspace,
                                      long long workspace_bytes, void* stream) {
  MTB_REQUIRE(running_mean && running_var, "conv2d_bn_forward: running statistics are required");
  MTB_REQUIRE(!residual || relu, "conv2d_bn_forward: an addition goes with a ReLU");
  const MtbBnEval bn{running_mean, running_var, gamma, beta, (float)eps};
  if (mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, y) && (!residual || mtb_aligned16(residual)))
    return mtb_tc_conv2d_forward_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, workspace, workspace_bytes, stream, nullptr,
                                     nullptr, &bn, residual);
  if (split_takes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, 0, workspace, workspace_bytes)) {
    if (int rc = forward_fp32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, 0, workspace, workspace_bytes, stream)) return rc;
    const long long rows = (long long)n * ((h + 2 * ph - kh) / sh + 1) * ((w + 2 * pw - kw) / sw + 1);
    return mtb_bn_eval_apply(y, y, rows, cout, bn, residual, relu, (cudaStream_t)stream);
  }
  return mtb_conv2d_forward_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, &bn, residual, stream);
}

// Inference: y = max_pool(max(0, batch_norm(conv(x)))) over 2 x 2 windows of stride 2, in one launch, where mtb_conv2d_bn_pool_takes answers 1:
// the convolutions that the small tiles of the CUDA-core family take (also on tensors off 16 bytes, so that the answer follows from
// the shape alone).  The bits, and the tie mask, are those of the separate operators.
// mtb_conv2d_bn_pool_scratch_bytes answers both questions of a forward pass in one call: -1 where the pool goes along, else the scratch that
// mtb_conv2d_bn_forward_f32 reads (0: none).
MTB_API long long mtb_conv2d_bn_pool_scratch_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  const float* al = reinterpret_cast<const float*>(uintptr_t(256));
  if (n <= 0 || cin <= 0 || cout <= 0 || kh <= 0 || kw <= 0 || sh <= 0 || sw <= 0 || ph < 0 || pw < 0 || !mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw)) return 0;
  const long long scratch = split_scratch_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, 0);
  if (scratch > 0 || mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al)) return scratch;
  return mtb_conv2d_bn_pool_simt_takes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout) ? -1 : 0;
}

MTB_API int mtb_conv2d_bn_pool_takes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  return mtb_conv2d_bn_pool_scratch_bytes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout) < 0 ? 1 : 0;
}

MTB_API int mtb_conv2d_bn_pool_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                           const float* wt, const float* bias, const float* gamma, const float* beta, const float* running_mean,
                                           const float* running_var, double eps, float* y, unsigned short* mask, void* stream) {
  MTB_REQUIRE(running_mean && running_var, "conv2d_bn_pool_forward: running statistics are required");
  return mtb_conv2d_bn_pool_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, MtbBnEval{running_mean, running_var, gamma, beta, (float)eps}, y, mask,
                                 stream);
}

MTB_API int mtb_conv2d_dgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                 const float* wt, float* dx, void* workspace, long long workspace_bytes, void* stream) {
  if (mtb_tc_conv2d_dgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx))
    return mtb_tc_conv2d_dgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, nullptr, dx, workspace, workspace_bytes, stream);
  return dgrad_fp32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, workspace, workspace_bytes, stream);
}

// dx = dgrad(dy, wt) + addend: the data gradient added to a gradient the same tensor already received
// from another consumer (residual connections).  On the row-staged tensor-core path the sum happens
// in the epilogue, which saves one pass over dx and one launch; elsewhere it is dgrad followed by an
// add.  addend has the shape of dx and must not alias it, except where
// mtb_conv2d_dgrad_accumulates_in_place answers 1: there addend == dx means dx += data gradient.
MTB_API int mtb_conv2d_dgrad_add_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                     const float* wt, const float* addend, float* dx, void* workspace, long long workspace_bytes, void* stream) {
  MTB_REQUIRE(addend, "conv2d_dgrad_add: addend must be given");
  if (addend == dx) {  // accumulate in place: only where mtb_conv2d_dgrad_accumulates_in_place says so
    MTB_REQUIRE(mtb_tc_conv2d_dgrad_in_place(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx),
                "conv2d_dgrad_add: this shape cannot accumulate in place (addend must not alias dx)");
    return mtb_tc_conv2d_dgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, addend, dx, workspace, workspace_bytes, stream);
  }
  if (mtb_tc_conv2d_dgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx))
    return mtb_tc_conv2d_dgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, addend, dx, workspace, workspace_bytes, stream);
  int rc = dgrad_fp32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, workspace, workspace_bytes, stream);
  if (rc) return rc;
  return mtb_add_f32(dx, addend, dx, (long long)n * h * w * cin, 1.0f, stream);
}

// 1 when mtb_conv2d_dgrad_add_f32 may be called with addend == dx for this convolution (dx += data gradient,
// nothing else touched) and that is its cheaper form; 0 otherwise.  Host code only.
MTB_API int mtb_conv2d_dgrad_accumulates_in_place(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout,
                                                  const float* dy, const float* wt, const float* dx) {
  return mtb_tc_conv2d_dgrad_in_place(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx) ? 1 : 0;
}

MTB_API int mtb_conv2d_wgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                 const float* dy, float* dw, void* workspace, long long workspace_bytes, void* stream) {
  const MtbScratchTurn turn;
  if (mtb_tc_conv2d_wgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, dy, dw))
    return mtb_tc_conv2d_wgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, dy, dw, workspace, workspace_bytes, stream);
  const int* guard = nullptr;
  int guards = 0;
  if (x && dy && dw && split_takes(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, 2, workspace, workspace_bytes))
    if (int rc = mtb_split_conv2d_wgrad_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, dy, dw, workspace, (cudaStream_t)stream, &guard, &guards)) return rc;
  return mtb_conv2d_wgrad_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, dy, dw, workspace, workspace_bytes, stream, guard, guards);
}

MTB_API int mtb_gemm_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu, float* c,
                         void* stream) {
  if (mtb_tc_gemm_supported(m, n, k, a, trans_a, b, trans_b, c))
    return mtb_tc_gemm_f32(m, n, k, a, trans_a, b, trans_b, bias, relu, c, stream);
  return mtb_gemm_simt_f32(m, n, k, a, trans_a, b, trans_b, bias, relu, c, stream);
}

// y = max(0, x w^T + bias) for x [m,k], w [n,k], and, with pre != NULL, pre = x w^T + bias: a Linear layer and the ReLU behind it
// in one launch, with what the ReLU's backward masks by.
MTB_API int mtb_linear_relu_f32(int m, int n, int k, const float* x, const float* w, const float* bias, float* pre, float* y, void* stream) {
  if (mtb_tc_gemm_supported(m, n, k, x, 0, w, 1, y)) return mtb_tc_gemm_f32(m, n, k, x, 0, w, 1, bias, 1, y, stream, pre);
  return mtb_gemm_simt(m, n, k, x, 0, w, 1, bias, 1, y, stream, pre);
}
