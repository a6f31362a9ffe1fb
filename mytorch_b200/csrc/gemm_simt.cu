// Dense matrix products on the CUDA cores (FP32): `mm` / Linear shapes whose pitches or sizes the tensor-core GEMM does
// not take.  See simt_tile.cuh for the kernel.
#include "simt_tile.cuh"

namespace {
using namespace simt;

template <int VEC>
int dense(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const Out& o, cudaStream_t st) {
  const Choice c = choose(m, n, k, 1, 1);
  const NoTable none;
  const DenseK ak{a, k}, bk{b, k};
  const DenseR ar{a, m}, br{b, n};
  if (!trans_a && trans_b) return launch<DenseK, VEC, DenseK, VEC>(c, ak, bk, o, none, 1, m, n, k, st, "gemm_simt");
  if (!trans_a) return launch<DenseK, VEC, DenseR, VEC>(c, ak, br, o, none, 1, m, n, k, st, "gemm_simt");
  if (trans_b) return launch<DenseR, VEC, DenseK, VEC>(c, ar, bk, o, none, 1, m, n, k, st, "gemm_simt");
  return launch<DenseR, VEC, DenseR, VEC>(c, ar, br, o, none, 1, m, n, k, st, "gemm_simt");
}

}  // namespace

// C[M,N] = op(A) * op(B) (+ bias[N]) (relu). A is [M,K] (trans_a == 0) or [K,M]; B is [K,N]
// (trans_b == 0) or [N,K]; all row-major and dense.
MTB_API int mtb_gemm_simt_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu,
                              float* c, void* stream) {
  MTB_REQUIRE(a && b && c && m > 0 && n > 0 && k > 0, "gemm: bad arguments");
  Out o{};
  o.out = c; o.ld = n; o.bias = bias; o.relu = relu;
  // four neighbours of each operand in one load: along k for [rows][K] operands, along the row for [K][rows] ones
  const bool vec = mtb_aligned16(a) && mtb_aligned16(b) && (trans_a ? m : k) % 4 == 0 && (trans_b ? k : n) % 4 == 0;
  return vec ? dense<4>(m, n, k, a, trans_a, b, trans_b, o, (cudaStream_t)stream)
             : dense<1>(m, n, k, a, trans_a, b, trans_b, o, (cudaStream_t)stream);
}
