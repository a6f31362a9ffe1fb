// Internal declarations shared between the entry-point file and the kernel families.
#pragma once
#include "common.cuh"

// general CUDA-core family (gemm_simt.cu, conv_simt.cu)
MTB_API int mtb_conv2d_forward_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                        const float* wt, const float* bias, float* y, int relu, void* stream);
// the same, followed by BatchNorm with running statistics and an optional addition before the ReLU
int mtb_conv2d_forward_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                            const float* bias, float* y, int relu, const MtbBnEval* bn_eval, const float* residual, void* stream,
                            const int* guard = nullptr, int guards = 0);
// guard: device words (guards of them); unless one is set nothing is done
int mtb_conv2d_dgrad_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy, const float* wt, float* dx,
                          void* stream, const int* guard, int guards);
int mtb_conv2d_wgrad_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* dy, float* dw,
                          void* workspace, long long workspace_bytes, void* stream, const int* guard, int guards);
// the same for a small convolution, followed by a ReLU and a 2 x 2 max-pool of stride 2 (mask: its tie mask)
bool mtb_conv2d_bn_pool_simt_takes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout);
int mtb_conv2d_bn_pool_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                            const float* bias, const MtbBnEval& bn, float* y, unsigned short* mask, void* stream);
// y = relu?(batch_norm(x) + residual) over [rows, c] with running statistics; x == y is allowed (batch_norm.cu)
int mtb_bn_eval_apply(const float* x, float* y, long long rows, int c, const MtbBnEval& bn, const float* residual, int relu, cudaStream_t st);
MTB_API int mtb_conv2d_dgrad_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                      const float* wt, float* dx, void* stream);
MTB_API long long mtb_conv2d_wgrad_simt_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout);
MTB_API int mtb_conv2d_wgrad_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                      const float* dy, float* dw, void* workspace, long long workspace_bytes, void* stream);
MTB_API int mtb_gemm_simt_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu,
                              float* c, void* stream);
// pre (may be NULL; neither operand transposed in memory): the result before the ReLU
int mtb_gemm_simt(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu, float* c, void* stream,
                  float* pre);

// tcgen05 tensor-core family (tc_*.cu)
long long mtb_tc_conv2d_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout);
bool mtb_tc_conv2d_forward_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                     const float* wt, const float* y);
int mtb_tc_conv2d_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                              const float* wt, const float* bias, float* y, int relu, void* workspace, long long workspace_bytes, void* stream,
                              float* stats = nullptr, int* stats_rows = nullptr, const MtbBnEval* bn_eval = nullptr,
                              const float* residual = nullptr);
bool mtb_tc_conv2d_dgrad_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                   const float* wt, const float* dx);
bool mtb_tc_conv2d_dgrad_in_place(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                  const float* wt, const float* dx);
int mtb_tc_conv2d_dgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                            const float* wt, const float* addend, float* dx, void* workspace, long long workspace_bytes, void* stream);
MTB_API int mtb_add_f32(const float* x, const float* y, float* z, long long n, float alpha, void* stream);
bool mtb_tc_conv2d_wgrad_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                   const float* dy, const float* dw);
int mtb_tc_conv2d_wgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                            const float* dy, float* dw, void* workspace, long long workspace_bytes, void* stream);
bool mtb_tc_gemm_supported(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* c);
int mtb_tc_gemm_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu, float* c,
                    void* stream, float* pre = nullptr);

double mtb_conv2d_simt_us(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction);

// FP32 accuracy on the tensor cores for channel counts of any size: operands as sums of two TF32 numbers (tc_split.cuh).
// direction: 0 forward, 1 data gradient, 2 weight gradient.  0 bytes: not taken.
long long mtb_split_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction);
int mtb_split_conv2d_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                                 const float* bias, float* y, int relu, void* workspace, cudaStream_t st, const int** guard, int* guards);
int mtb_split_conv2d_dgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy, const float* wt,
                               float* dx, void* workspace, cudaStream_t st, const int** guard, int* guards);
int mtb_split_conv2d_wgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* dy,
                               float* dw, void* workspace, cudaStream_t st, const int** guard, int* guards);
