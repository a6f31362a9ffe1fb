// Dense matrix products on the CUDA cores (FP32): `mm` / Linear shapes whose pitches or sizes the tensor-core GEMM does
// not take.  See simt_tile.cuh for the kernel.
#include "kernels.h"
#include "simt_tile.cuh"

namespace {
using namespace simt;

template <int VEC>
int dense(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const Out& o, float* pre, cudaStream_t st) {
  const Choice c = choose(m, n, k, 1, 1);
  const NoTable none;
  const DenseK ak{a, k}, bk{b, k};
  const DenseR ar{a, m}, br{b, n};
  if (!trans_a && trans_b) return launch<DenseK, VEC, DenseK, VEC>(c, ak, bk, o, none, 1, m, n, k, st, "gemm_simt", Extra{nullptr, 0, pre});
  if (!trans_a) return launch<DenseK, VEC, DenseR, VEC>(c, ak, br, o, none, 1, m, n, k, st, "gemm_simt");
  if (trans_b) return launch<DenseR, VEC, DenseK, VEC>(c, ar, bk, o, none, 1, m, n, k, st, "gemm_simt");
  return launch<DenseR, VEC, DenseR, VEC>(c, ar, br, o, none, 1, m, n, k, st, "gemm_simt");
}

// C[M,N] = A^T B for A stored [K][M] with M <= 16 and B [K][N]: the weight gradient of a Linear layer with few outputs
// (dW[10][512] = dY^T X).  A CTA owns 32 columns and two rows; its 8 warps take every eighth k, in order, and the 8 partial
// sums are added in warp order.  Bound by the latency of the loads along k, so 32 steps of them are issued ahead of the
// FMAs, and rows are spread over CTAs (one row alone took 27 us, the compiler then issues no loads ahead): with two rows and
// 32 steps instead of four and 16, 10 x 512, K = 512: 10.2 -> 4.1 us; 1 x 500, K = 1000: 18.7 -> 6.1; 1 x 500, K = 8000: 137 -> 35.
__global__ void __launch_bounds__(256) gemm_few_rows_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ c,
                                                             int M, int N, int K) {
  mtb_launch_dependents();
  mtb_wait_prior();
  constexpr int R = 2, AHEAD = 32;
  __shared__ float part[8][R][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 32 + lane, m0 = blockIdx.y * R;
  float acc[R] = {};
  if (col < N) {
    for (int k0 = warp; k0 < K; k0 += 8 * AHEAD) {
      float bv[AHEAD], av[AHEAD][R];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int k = k0 + 8 * u;
        bv[u] = k < K ? __ldg(b + (long long)k * N + col) : 0.f;
#pragma unroll
        for (int m = 0; m < R; ++m) av[u][m] = k < K && m0 + m < M ? __ldg(a + (long long)k * M + m0 + m) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (k0 + 8 * u < K) {
#pragma unroll
          for (int m = 0; m < R; ++m) acc[m] = fmaf(av[u][m], bv[u], acc[m]);
        }
    }
  }
#pragma unroll
  for (int m = 0; m < R; ++m) part[warp][m][lane] = acc[m];
  __syncthreads();
  if (warp < R && m0 + warp < M && col < N) {
    float t = part[0][warp][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += part[w][warp][lane];
    c[(long long)(m0 + warp) * N + col] = t;
  }
}

}  // namespace

// C[M,N] = op(A) * op(B) (+ bias[N]) (relu). A is [M,K] (trans_a == 0) or [K,M]; B is [K,N]
// (trans_b == 0) or [N,K]; all row-major and dense.
MTB_API int mtb_gemm_simt_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu,
                              float* c, void* stream) {
  return mtb_gemm_simt(m, n, k, a, trans_a, b, trans_b, bias, relu, c, stream, nullptr);
}

int mtb_gemm_simt(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu, float* c, void* stream,
                  float* pre) {
  MTB_REQUIRE(a && b && c && m > 0 && n > 0 && k > 0, "gemm: bad arguments");
  if (trans_a && !trans_b && m <= 16 && !bias && !relu) {
    MTB_LAUNCH(gemm_few_rows_kernel, dim3(mtb_div_up(n, 32), mtb_div_up(m, 2)), 256, 0, (cudaStream_t)stream, a, b, c, m, n, k);
    MTB_LAUNCH_CHECK("gemm_few_rows_kernel");
    return MTB_OK;
  }
  Out o{};
  o.out = c; o.ld = n; o.bias = bias; o.relu = relu;
  // four neighbours of each operand in one load: along k for [rows][K] operands, along the row for [K][rows] ones
  const bool vec = mtb_aligned16(a) && mtb_aligned16(b) && (trans_a ? m : k) % 4 == 0 && (trans_b ? k : n) % 4 == 0;
  return vec ? dense<4>(m, n, k, a, trans_a, b, trans_b, o, pre, (cudaStream_t)stream)
             : dense<1>(m, n, k, a, trans_a, b, trans_b, o, pre, (cudaStream_t)stream);
}
