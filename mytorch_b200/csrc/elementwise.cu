// Bandwidth kernels with no cross-element dependency: fill, copy, cast, ReLU, add, bias add,
// generic strided copy / broadcast binary ops, NCHW<->NHWC layout changes.
// All are grid-stride loops over float4 where alignment allows; grids are capped at a
// multiple of the SM count.
#include "common.cuh"

namespace {

constexpr int kThreads = 256;

template <class F>
__global__ void __launch_bounds__(kThreads) map1_kernel(float* out, const float* a, long long n4, long long n, F f) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = i; v < n4; v += stride) {
    float4 x = ld4(a + 4 * v);
    float4 r = make_float4(f(x.x), f(x.y), f(x.z), f(x.w));
    st4(out + 4 * v, r);
  }
  for (long long t = 4 * n4 + i; t < n; t += stride) out[t] = f(a[t]);
}

template <class F>
__global__ void __launch_bounds__(kThreads) map2_kernel(float* out, const float* a, const float* b,
                                                         long long n4, long long n, F f) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = i; v < n4; v += stride) {
    float4 x = ld4(a + 4 * v), y = ld4(b + 4 * v);
    st4(out + 4 * v, make_float4(f(x.x, y.x), f(x.y, y.y), f(x.z, y.z), f(x.w, y.w)));
  }
  for (long long t = 4 * n4 + i; t < n; t += stride) out[t] = f(a[t], b[t]);
}

struct ReluF { __device__ float operator()(float x) const { return fmaxf(x, 0.f); } };
// Gradient is blocked only for x < 0 (the CPU reference passes it at x == 0).
struct ReluBwdF { __device__ float operator()(float dy, float x) const { return x < 0.f ? 0.f : dy; } };
struct AxpyF { float alpha; __device__ float operator()(float x, float y) const { return x + y * alpha; } };
struct AddReluF { __device__ float operator()(float x, float y) const { return fmaxf(x + y, 0.f); } };
struct MulF { __device__ float operator()(float x, float y) const { return x * y; } };
struct ScaleF { float s; __device__ float operator()(float x) const { return x * s; } };
struct CopyF { __device__ float operator()(float x) const { return x; } };

// g = (x + y < 0) ? 0 : dy — backward of max(0, x + y); the sum is recomputed from the two
// forward inputs (bit-identical to the forward's), and a sum of exactly 0 passes the gradient.
__global__ void __launch_bounds__(kThreads) add_relu_bwd_kernel(float* g, const float* dy, const float* x, const float* y, long long n4, long long n) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = i; v < n4; v += stride) {
    float4 d = ld4(dy + 4 * v), a = ld4(x + 4 * v), b = ld4(y + 4 * v);
    d.x = (a.x + b.x < 0.f) ? 0.f : d.x;
    d.y = (a.y + b.y < 0.f) ? 0.f : d.y;
    d.z = (a.z + b.z < 0.f) ? 0.f : d.z;
    d.w = (a.w + b.w < 0.f) ? 0.f : d.w;
    st4(g + 4 * v, d);
  }
  for (long long t = 4 * n4 + i; t < n; t += stride) g[t] = (x[t] + y[t] < 0.f) ? 0.f : dy[t];
}

template <class F>
int launch_map1(float* out, const float* a, long long n, F f, cudaStream_t s, const char* name) {
  if (n == 0) return MTB_OK;
  bool vec = mtb_aligned16(out) && mtb_aligned16(a);
  long long n4 = vec ? n / 4 : 0;
  int grid = mtb_stream_grid(vec ? (n4 > 0 ? n4 : 1) : n, kThreads);
  MTB_LAUNCH(map1_kernel<F>, grid, kThreads, 0, s, out, a, n4, n, f);
  MTB_LAUNCH_CHECK(name);
  return MTB_OK;
}

template <class F>
int launch_map2(float* out, const float* a, const float* b, long long n, F f, cudaStream_t s, const char* name) {
  if (n == 0) return MTB_OK;
  bool vec = mtb_aligned16(out) && mtb_aligned16(a) && mtb_aligned16(b);
  long long n4 = vec ? n / 4 : 0;
  int grid = mtb_stream_grid(vec ? (n4 > 0 ? n4 : 1) : n, kThreads);
  MTB_LAUNCH(map2_kernel<F>, grid, kThreads, 0, s, out, a, b, n4, n, f);
  MTB_LAUNCH_CHECK(name);
  return MTB_OK;
}

// y[r, c] = x[r, c] + alpha * bias[c]; cols % 4 == 0 fast path.
__global__ void __launch_bounds__(kThreads) bias_rows_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ bias,
                                                              long long n, int cols, float alpha) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = i; t < n; t += stride) y[t] = x[t] + alpha * bias[t % cols];
}

__global__ void __launch_bounds__(kThreads) fill_kernel(float* out, long long n4, long long n, float v) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  float4 v4 = make_float4(v, v, v, v);
  for (long long k = i; k < n4; k += stride) st4(out + 4 * k, v4);
  for (long long t = 4 * n4 + i; t < n; t += stride) out[t] = v;
}

struct Strides6 {
  int ndim;
  long long shape[6];
  long long a[6];
  long long b[6];
  long long o[6];
};

template <int OP>
__global__ void __launch_bounds__(kThreads) strided_binary_kernel(float* __restrict__ out, const float* __restrict__ a, const float* __restrict__ b,
                                                                   long long n, Strides6 s, float alpha) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = i; t < n; t += stride) {
    long long r = t, oa = 0, ob = 0, oo = 0;
    for (int d = s.ndim - 1; d >= 0; --d) {
      long long c = r % s.shape[d];
      r /= s.shape[d];
      oa += c * s.a[d];
      ob += c * s.b[d];
      oo += c * s.o[d];
    }
    float x = a[oa];
    float y = (OP == 5) ? 0.f : b[ob];
    float v;
    if (OP == 0) v = x + alpha * y;
    else if (OP == 1) v = x - alpha * y;
    else if (OP == 2) v = x * y;
    else if (OP == 3) v = x / y;
    else if (OP == 4) v = powf(x, y);
    else if (OP == 6) v = y * powf(x, y - 1.f);   // d(x^y)/dx
    else if (OP == 7) v = powf(x, y) * logf(x);   // d(x^y)/dy
    else v = x * alpha;  // OP == 5: strided copy (alpha 1) / scaled broadcast
    out[oo] = v;
  }
}

// NCHW -> NHWC through a shared-memory tile transpose of the [C, HW] plane of each image.
__global__ void __launch_bounds__(256) transpose_planes_kernel(float* __restrict__ dst, const float* __restrict__ src, int rows, int cols) {
  mtb_launch_dependents();
  mtb_wait_prior();
  // src: [batch][rows][cols] -> dst: [batch][cols][rows]
  __shared__ float tile[32][33];
  const float* s = src + (long long)blockIdx.z * rows * cols;
  float* d = dst + (long long)blockIdx.z * rows * cols;
  int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    int r = r0 + j, c = c0 + threadIdx.x;
    if (r < rows && c < cols) tile[j][threadIdx.x] = s[(long long)r * cols + c];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    int c = c0 + j, r = r0 + threadIdx.x;
    if (r < rows && c < cols) d[(long long)c * rows + r] = tile[threadIdx.x][j];
  }
}

__global__ void cast_i32_i64_kernel(long long* out, const int* in, long long n) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = in[i];
}
__global__ void cast_i64_f32_kernel(float* out, const long long* in, long long n) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = (float)in[i];
}
__global__ void cast_f32_i64_kernel(long long* out, const float* in, long long n) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = (long long)in[i];
}

__global__ void cast_i8_f32_kernel(float* out, const signed char* in, long long n) {
  mtb_launch_dependents();
  mtb_wait_prior();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = (float)in[i];
}

int transpose_planes(float* dst, const float* src, int batch, int rows, int cols, cudaStream_t s) {
  if ((long long)batch * rows * cols == 0) return MTB_OK;
  MTB_REQUIRE(batch <= 65535 * 1, "layout change: batch %d exceeds grid.z", batch);
  dim3 grid(mtb_div_up(cols, 32), mtb_div_up(rows, 32), batch), block(32, 8);
  MTB_REQUIRE(grid.y <= 65535, "layout change: too many rows");
  MTB_LAUNCH(transpose_planes_kernel, grid, block, 0, s, dst, src, rows, cols);
  MTB_LAUNCH_CHECK("transpose_planes_kernel");
  return MTB_OK;
}

// dst[r][c] = c < c_src ? src[r][c] : 0 for c < c_dst: widen a [rows, c_src] matrix with zero
// columns (c_dst > c_src) or keep its first c_dst columns (c_dst < c_src), in one pass.
__global__ void __launch_bounds__(256) resize_channels_kernel(const float* __restrict__ src, float* __restrict__ dst, long long rows, int c_src, int c_dst) {
  mtb_launch_dependents();
  mtb_wait_prior();
  const long long total = rows * c_dst;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / c_dst;
    const int c = (int)(i - r * c_dst);
    dst[i] = c < c_src ? src[r * c_src + c] : 0.f;
  }
}

// out[n][oh][ow][32]: the first k_h * KW * C entries of a pixel are the input pixels its filter rows see, as one run of
// (kh, kw, c); the rest is zero.  A thread writes four entries (16 bytes; eight threads write a pixel's 128 bytes).
// Bound by those writes: the input is C / 32 of their size and its re-reads hit L1.
struct PatchRuns {
  int N, C, H, W, KH, KW, SH, SW, PH, PW, OH, OW;
};
// ROW: the window is a single filter row (KH = 1), whose entries are neighbours in memory: one address and a range say all.
// AHEAD: pixels of a thread whose loads are in flight before it writes the first, four where it has as many (7x7 over 3
// channels of 128 x 224x224: 155 -> 98 us, of which the 411 MB written take 63; one image, a pixel a thread: 3.7 us, 4.6 with
// three that are not there).  Whole windows did not gain from loads ahead (3x3 over 3 channels of 512 x 32x32: 32 us, 34).
template <bool ROW, int AHEAD>
__global__ void __launch_bounds__(256) pack_patches_kernel(const float* __restrict__ x, float4* __restrict__ out, PatchRuns d, unsigned pixels) {
  mtb_launch_dependents();
  mtb_wait_prior();
  // A thread always writes the same four entries of a pixel, so where they lie in the filter is worked out once; a CTA walks
  // 32 neighbouring pixels at a time.
  const int run = d.KW * d.C, used = d.KH * run;
  const unsigned part = threadIdx.x & 7u;
  int dh[4], dw[4], dc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = (int)part * 4 + q, kh = k / run, r = k - kh * run;
    dh[q] = k < used ? kh - d.PH : -(1 << 28);  // far outside: reads as zero
    dw[q] = r / d.C - d.PW;
    dc[q] = r - r / d.C * d.C;
  }
  const int first = (int)part * 4 - d.PW * d.C, row = d.W * d.C;
  const unsigned step = gridDim.x * 32u;
  for (unsigned pixel = blockIdx.x * 32u + (threadIdx.x >> 3); pixel < pixels; pixel += AHEAD * step) {
    float v[AHEAD][4];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const unsigned px = pixel + u * step;
      const bool in = px < pixels;
      const unsigned ow = px % (unsigned)d.OW, t = px / (unsigned)d.OW;
      const int h0 = (int)(t % (unsigned)d.OH) * d.SH, w0 = (int)ow * d.SW;
      const long long image = (long long)(t / (unsigned)d.OH) * d.H;
      if constexpr (ROW) {
        const int h = h0 - d.PH, j0 = w0 * d.C + first;
        const bool there = in && (unsigned)h < (unsigned)d.H;
        const float* p = x + (image + h) * row + j0;
#pragma unroll
        for (int q = 0; q < 4; ++q) v[u][q] = there && (int)part * 4 + q < used && (unsigned)(j0 + q) < (unsigned)row ? __ldg(p + q) : 0.f;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int h = h0 + dh[q], w = w0 + dw[q];
          v[u][q] = in && (unsigned)h < (unsigned)d.H && (unsigned)w < (unsigned)d.W ? __ldg(x + ((image + h) * d.W + w) * d.C + dc[q]) : 0.f;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const unsigned px = pixel + u * step;
      if (px < pixels) out[(size_t)px * 8 + part] = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    }
  }
}

}  // namespace

// Gathers what a filter of few input channels sees into runs of 32 floats per output pixel: out[N][OH][OW][32] with
// entry (kh * KW + kw) * C + c, zero beyond the edges and from KH * KW * C on (KH * KW * C <= 32).  A convolution with
// few input channels then is one with 32 channels and no window (or, with KH = 1 here, one whose window is a single
// column): a 7x7 filter over 3 channels reads 7 blocks of 32 instead of 49.  No counterpart in the reference.
MTB_API int mtb_pack_patches_f32(int n, int c, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, const float* x, float* out, void* stream) {
  MTB_REQUIRE(x && out && n > 0 && c > 0 && h > 0 && w > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0 && ph >= 0 && pw >= 0, "pack_patches: bad arguments");
  MTB_REQUIRE((long long)kh * kw * c <= 32, "pack_patches: the filter has more than 32 entries");
  MTB_REQUIRE(mtb_window_fits(h, ph, kh) && mtb_window_fits(w, pw, kw), "pack_patches: a %dx%d window is larger than the padded %dx%d input", kh, kw, h, w);
  PatchRuns d{n, c, h, w, kh, kw, sh, sw, ph, pw, (h + 2 * ph - kh) / sh + 1, (w + 2 * pw - kw) / sw + 1};
  MTB_REQUIRE(d.OH > 0 && d.OW > 0 && mtb_aligned16(out), "pack_patches: empty or unaligned output");
  const long long pixels = (long long)n * d.OH * d.OW;
  MTB_REQUIRE(pixels < (1LL << 31), "pack_patches: too many pixels");
  const int grid = mtb_stream_grid(pixels, 32);
  const bool row = kh == 1 && (long long)w * c + 64 < (1LL << 31);
  if (row && pixels >= 4LL * 32 * grid) MTB_LAUNCH(pack_patches_kernel<true, 4>, grid, 256, 0, (cudaStream_t)stream, x, (float4*)out, d, (unsigned)pixels);
  else if (row) MTB_LAUNCH(pack_patches_kernel<true, 1>, grid, 256, 0, (cudaStream_t)stream, x, (float4*)out, d, (unsigned)pixels);
  else MTB_LAUNCH(pack_patches_kernel<false, 1>, grid, 256, 0, (cudaStream_t)stream, x, (float4*)out, d, (unsigned)pixels);
  MTB_LAUNCH_CHECK("pack_patches_kernel");
  return MTB_OK;
}

// Copy a row-major [rows, c_src] matrix into [rows, c_dst]: extra columns are zero, surplus columns are
// dropped.  Pads the 1- or 3-channel image stem (and its filter) to one 32-channel block for the
// tensor-core convolution and cuts the weight gradient back; no counterpart in the reference.
MTB_API int mtb_resize_channels_f32(const float* src, float* dst, long long rows, int c_src, int c_dst, void* stream) {
  MTB_REQUIRE(src && dst && rows > 0 && c_src > 0 && c_dst > 0, "resize_channels: bad arguments");
  MTB_LAUNCH(resize_channels_kernel, mtb_stream_grid(rows * c_dst, kThreads), kThreads, 0, (cudaStream_t)stream, src, dst, rows, c_src, c_dst);
  MTB_LAUNCH_CHECK("resize_channels_kernel");
  return MTB_OK;
}

MTB_API int mtb_fill_f32(float* x, long long n, float value, void* stream) {
  MTB_REQUIRE(n >= 0 && (x || n == 0), "fill: bad arguments");
  if (n == 0) return MTB_OK;
  long long n4 = mtb_aligned16(x) ? n / 4 : 0;
  MTB_LAUNCH(fill_kernel, mtb_stream_grid(n4 > 0 ? n4 : n, kThreads), kThreads, 0, (cudaStream_t)stream, x, n4, n, value);
  MTB_LAUNCH_CHECK("fill_kernel");
  return MTB_OK;
}

MTB_API int mtb_copy_f32(float* dst, const float* src, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((dst && src) || n == 0), "copy: bad arguments");
  return launch_map1(dst, src, n, CopyF{}, (cudaStream_t)stream, "copy");
}

MTB_API int mtb_scale_f32(float* dst, const float* src, long long n, float scale, void* stream) {
  MTB_REQUIRE(n >= 0 && ((dst && src) || n == 0), "scale: bad arguments");
  return launch_map1(dst, src, n, ScaleF{scale}, (cudaStream_t)stream, "scale");
}

MTB_API int mtb_relu_forward_f32(const float* x, float* y, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((x && y) || n == 0), "relu: bad arguments");
  return launch_map1(y, x, n, ReluF{}, (cudaStream_t)stream, "relu_forward");
}

MTB_API int mtb_relu_backward_f32(const float* dy, const float* x, float* dx, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((x && dy && dx) || n == 0), "relu_backward: bad arguments");
  return launch_map2(dx, dy, x, n, ReluBwdF{}, (cudaStream_t)stream, "relu_backward");
}

// z = x + alpha * y, same number of elements and same physical layout. z may alias x.
MTB_API int mtb_add_f32(const float* x, const float* y, float* z, long long n, float alpha, void* stream) {
  MTB_REQUIRE(n >= 0 && ((x && y && z) || n == 0), "add: bad arguments");
  return launch_map2(z, x, y, n, AxpyF{alpha}, (cudaStream_t)stream, "add");
}

// z = max(0, x + y): residual add and ReLU in one pass.
MTB_API int mtb_add_relu_f32(const float* x, const float* y, float* z, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((x && y && z) || n == 0), "add_relu: bad arguments");
  return launch_map2(z, x, y, n, AddReluF{}, (cudaStream_t)stream, "add_relu");
}

// g = (x + y < 0) ? 0 : dy: the gradient of max(0, x + y) with respect to x and to y.
MTB_API int mtb_add_relu_backward_f32(const float* dy, const float* x, const float* y, float* g, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((dy && x && y && g) || n == 0), "add_relu_backward: bad arguments");
  if (n == 0) return MTB_OK;
  bool vec = mtb_aligned16(dy) && mtb_aligned16(x) && mtb_aligned16(y) && mtb_aligned16(g);
  long long n4 = vec ? n / 4 : 0;
  MTB_LAUNCH(add_relu_bwd_kernel, mtb_stream_grid(vec ? (n4 > 0 ? n4 : 1) : n, kThreads), kThreads, 0, (cudaStream_t)stream, g, dy, x, y, n4, n);
  MTB_LAUNCH_CHECK("add_relu_bwd_kernel");
  return MTB_OK;
}

MTB_API int mtb_mul_f32(const float* x, const float* y, float* z, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((x && y && z) || n == 0), "mul: bad arguments");
  return launch_map2(z, x, y, n, MulF{}, (cudaStream_t)stream, "mul");
}

// y[r, :] = x[r, :] + alpha * bias[:] for a row-major [rows, cols] matrix.
MTB_API int mtb_add_bias_rows_f32(const float* x, const float* bias, float* y, long long rows, int cols, float alpha, void* stream) {
  MTB_REQUIRE(rows >= 0 && cols > 0 && x && bias && y, "add_bias_rows: bad arguments");
  long long n = rows * cols;
  if (n == 0) return MTB_OK;
  MTB_LAUNCH(bias_rows_kernel, mtb_stream_grid(n, kThreads), kThreads, 0, (cudaStream_t)stream, y, x, bias, n, cols, alpha);
  MTB_LAUNCH_CHECK("bias_rows_kernel");
  return MTB_OK;
}

// Generic broadcast binary op over up to 6 logical dimensions. Strides are in elements; a stride
// of 0 broadcasts. op: 0 add (x + alpha*y), 1 sub (x - alpha*y), 2 mul, 3 div, 4 pow, 5 alpha*x (y unused),
// 6 y*x^(y-1) and 7 x^y*ln(x) (the two partial derivatives of pow).
MTB_API int mtb_binary_strided_f32(int op, int ndim, const long long* shape, const long long* x_strides, const long long* y_strides,
                                   const long long* z_strides, const float* x, const float* y, float* z, float alpha, void* stream) {
  MTB_REQUIRE(ndim >= 0 && ndim <= 6 && op >= 0 && op <= 7 && x && z && (y || op == 5), "binary_strided: bad arguments");
  Strides6 s;
  s.ndim = ndim;
  long long n = 1;
  for (int d = 0; d < ndim; ++d) {
    s.shape[d] = shape[d];
    s.a[d] = x_strides[d];
    s.b[d] = (op == 5) ? 0 : y_strides[d];
    s.o[d] = z_strides[d];
    n *= shape[d];
  }
  if (n == 0) return MTB_OK;
  int grid = mtb_stream_grid(n, kThreads);
  cudaStream_t st = (cudaStream_t)stream;
  switch (op) {
    case 0: MTB_LAUNCH(strided_binary_kernel<0>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 1: MTB_LAUNCH(strided_binary_kernel<1>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 2: MTB_LAUNCH(strided_binary_kernel<2>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 3: MTB_LAUNCH(strided_binary_kernel<3>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 4: MTB_LAUNCH(strided_binary_kernel<4>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 6: MTB_LAUNCH(strided_binary_kernel<6>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    case 7: MTB_LAUNCH(strided_binary_kernel<7>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
    default: MTB_LAUNCH(strided_binary_kernel<5>, grid, kThreads, 0, st, z, x, y, n, s, alpha); break;
  }
  MTB_LAUNCH_CHECK("strided_binary_kernel");
  return MTB_OK;
}

// Logical NCHW buffer -> channels-last (NHWC) buffer and back.
MTB_API int mtb_nchw_to_nhwc_f32(const float* src, float* dst, int n, int c, int h, int w, void* stream) {
  MTB_REQUIRE(src && dst && n >= 0 && c > 0 && h > 0 && w > 0, "nchw_to_nhwc: bad arguments");
  return transpose_planes(dst, src, n, c, h * w, (cudaStream_t)stream);
}

MTB_API int mtb_nhwc_to_nchw_f32(const float* src, float* dst, int n, int c, int h, int w, void* stream) {
  MTB_REQUIRE(src && dst && n >= 0 && c > 0 && h > 0 && w > 0, "nhwc_to_nchw: bad arguments");
  return transpose_planes(dst, src, n, h * w, c, (cudaStream_t)stream);
}

// kind: 0 int32->int64, 1 int64->float32, 2 float32->int64.
MTB_API int mtb_cast(int kind, const void* src, void* dst, long long n, void* stream) {
  MTB_REQUIRE(n >= 0 && ((src && dst) || n == 0), "cast: bad arguments");
  if (n == 0) return MTB_OK;
  int grid = mtb_stream_grid(n, kThreads);
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 0) MTB_LAUNCH(cast_i32_i64_kernel, grid, kThreads, 0, st, (long long*)dst, (const int*)src, n);
  else if (kind == 1) MTB_LAUNCH(cast_i64_f32_kernel, grid, kThreads, 0, st, (float*)dst, (const long long*)src, n);
  else if (kind == 2) MTB_LAUNCH(cast_f32_i64_kernel, grid, kThreads, 0, st, (long long*)dst, (const float*)src, n);
  else if (kind == 3) MTB_LAUNCH(cast_i8_f32_kernel, grid, kThreads, 0, st, (float*)dst, (const signed char*)src, n);
  else return mtb_fail(MTB_ERR_UNSUPPORTED, "cast kind %d", kind);
  MTB_LAUNCH_CHECK("cast kernel");
  return MTB_OK;
}
