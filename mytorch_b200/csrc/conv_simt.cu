// Convolution on the CUDA cores (FP32) for the shapes the tensor-core kernels do not take: channel counts that are no
// multiple of 32, activations under 128 KiB.  Forward, data gradient and weight gradient as implicit matrix
// products over channels-last tensors (see simt_tile.cuh for the kernel).
#include "kernels.h"
#include "simt_tile.cuh"

namespace {
using namespace simt;

int conv_dims(ConvDims& d, int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  MTB_REQUIRE(n > 0 && cin > 0 && h > 0 && w > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0 && ph >= 0 && pw >= 0 && cout > 0, "conv2d: bad shape");
  MTB_REQUIRE(mtb_window_fits(h, ph, kh) && mtb_window_fits(w, pw, kw), "conv2d: a %dx%d filter is larger than the padded %dx%d input", kh, kw, h, w);
  d = ConvDims{n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, (h + 2 * ph - kh) / sh + 1, (w + 2 * pw - kw) / sw + 1};
  MTB_REQUIRE(d.OH > 0 && d.OW > 0, "conv2d: empty output");
  constexpr long long limit = (1LL << 31) - 256;  // rows and reduction positions are 31-bit numbers, tiles overshoot
  MTB_REQUIRE((long long)n * d.OH * d.OW < limit && (long long)n * h * w < limit, "conv2d: too many pixels for this kernel");
  MTB_REQUIRE((long long)kh * kw * cin < limit && (long long)kh * kw * cout < limit, "conv2d: filter too large for this kernel");
  return MTB_OK;
}

PatchK patch_k(const float* x, const ConvDims& d) { return PatchK{x, d, FastDiv(d.OW), FastDiv(d.OH), FastDiv(d.Cin), FastDiv(d.KW)}; }
PatchR patch_r(const float* x, const ConvDims& d) { return PatchR{x, d, FastDiv(d.OW), FastDiv(d.OH), FastDiv(d.Cin), FastDiv(d.KW)}; }

// One axis of residue class a: taps a + s*t (t < taps), pixels start + s*i (i < count), tap t of pixel i meets output c0 + i - t.
void class_axis(int a, int size, int k, int s, int pad, int& taps, int& start, int& count, int& c0) {
  taps = a < k ? (k - a + s - 1) / s : 0;
  start = (((a - pad) % s) + s) % s;
  count = start < size ? (size - start + s - 1) / s : 0;
  c0 = (start + pad - a) / s;
}

Choice wgrad_choice(const ConvDims& d) {
  const long long pixels = (long long)d.N * d.OH * d.OW;
  const long long most = (pixels + 255) / 256;  // a slice keeps at least 256 pixels
  return choose(d.Cout, (long long)d.KH * d.KW * d.Cin, pixels, 1, (int)(most < 2 ? 2 : (most > 512 ? 512 : most)));
}

}  // namespace

// What the kernels below are priced at, in us (direction: 0 forward, 1 data gradient, 2 weight gradient).
double mtb_conv2d_simt_us(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction) {
  ConvDims d;
  if (conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout)) return 0.0;
  Choice c;
  if (direction == 0) {
    c = choose((long long)n * d.OH * d.OW, cout, (long long)kh * kw * cin, 1, 1);
  } else if (direction == 1) {
    const int classes = sh * sw < kMaxClasses ? sh * sw : kMaxClasses;
    c = choose(((long long)n * h * w + sh * sw - 1) / (sh * sw), cin, (long long)((kh + sh - 1) / sh) * ((kw + sw - 1) / sw) * cout, classes, 1);
    c.cycles *= (double)sh * sw / classes;
  } else {
    c = wgrad_choice(d);
  }
  // the prices are those of float4 loads; single floats cost about 1.4 times as much (16 images of 40x40, 129 -> 130 channels)
  const bool four = direction == 0 ? cin % 4 == 0 : direction == 1 ? cout % 4 == 0 : cin % 4 == 0 && cout % 4 == 0;
  return c.cycles / 1850.0 * (four ? 1.0 : 1.4);
}

int mtb_conv2d_forward_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                            const float* bias, float* y, int relu, const MtbBnEval* bn_eval, const float* residual, void* stream, const int* guard, int guards) {
  ConvDims d;
  int rc = conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (rc) return rc;
  MTB_REQUIRE(x && wt && y, "conv2d_forward: null pointer");
  const int K = kh * kw * cin, M = n * d.OH * d.OW;
  Out o{};
  o.out = y; o.ld = cout; o.bias = bias; o.relu = relu;
  const Choice c = choose(M, cout, K, 1, 1);
  if (bn_eval) {
    if (tile_info(c.tile).cluster) {  // small tiles: BatchNorm in the store
      o.bn = *bn_eval;
      o.residual = residual;
    } else {
      const int rc2 = mtb_conv2d_forward_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, 0, nullptr, nullptr, stream, nullptr, 0);
      return rc2 ? rc2 : mtb_bn_eval_apply(y, y, M, cout, *bn_eval, residual, relu, (cudaStream_t)stream);
    }
  }
  const Extra extra{guard, guards, nullptr};
  const DenseK filter{wt, K};
  if (cin % 4 == 0 && mtb_aligned16(x) && mtb_aligned16(wt))
    return launch<PatchK, 4, DenseK, 4>(c, patch_k(x, d), filter, o, NoTable{}, 1, M, cout, K, (cudaStream_t)stream, "conv2d_forward_simt", extra);
  return launch<PatchK, 1, DenseK, 1>(c, patch_k(x, d), filter, o, NoTable{}, 1, M, cout, K, (cudaStream_t)stream, "conv2d_forward_simt", extra);
}

namespace {
// Rows of the product whose rows are the pixels of 2 x 2 windows, and the tile and reduction slices of the convolution by itself (all pixels: a last odd line
// or column must not change the order of a sum); false: no window, or a tile that is not a cluster's (large products, which have better kernels
// and a pooling pass of their own).
bool pooled_choice(const ConvDims& d, long long& rows, Choice& c) {
  rows = 4LL * d.N * (d.OH / 2) * (d.OW / 2);
  if (rows == 0) return false;
  c = choose((long long)d.N * d.OH * d.OW, d.Cout, (long long)d.KH * d.KW * d.Cin, 1, 1);
  return tile_info(c.tile).cluster;
}
}  // namespace

bool mtb_conv2d_bn_pool_simt_takes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  ConvDims d;
  long long rows;
  Choice c;
  return !conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout) && pooled_choice(d, rows, c);
}

// y = max_pool(max(0, batch_norm(conv(x)))) over 2 x 2 windows of stride 2, running statistics.  Answering one small image is launches and
// host time: the example's digit classifier takes 6 launches instead of 9, 63 -> 45 us.
int mtb_conv2d_bn_pool_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                            const float* bias, const MtbBnEval& bn, float* y, unsigned short* mask, void* stream) {
  ConvDims d;
  if (int rc = conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout)) return rc;
  MTB_REQUIRE(x && wt && y && mask, "conv2d_bn_pool: null pointer");
  long long rows;
  Choice c;
  if (!pooled_choice(d, rows, c)) return mtb_fail(MTB_ERR_UNSUPPORTED, "conv2d_bn_pool: not a small convolution");
  Out o{};
  o.out = y; o.ld = cout; o.bias = bias; o.bn = bn; o.relu = 1;
  PatchPoolK a;
  static_cast<PatchK&>(a) = patch_k(x, d);
  a.pool_w = FastDiv(d.OW / 2);
  a.pool_h = FastDiv(d.OH / 2);
  const int K = kh * kw * cin, M = (int)rows;
  const DenseK filter{wt, K};
  const PoolExtra extra{mask};
  cudaStream_t st = (cudaStream_t)stream;
  const bool four = cin % 4 == 0 && mtb_aligned16(x) && mtb_aligned16(wt);
#define MTB_POOLED(T_, V_) launch_tile<EXTRA_NONE, T_, PatchPoolK, V_, DenseK, V_, true>(a, filter, o, NoTable{}, 1, M, cout, K, c.slices, st, "conv2d_bn_pool_simt", extra)
  if (c.tile == SM) return four ? MTB_POOLED(TileS, 4) : MTB_POOLED(TileS, 1);
  return four ? MTB_POOLED(TileXS, 4) : MTB_POOLED(TileXS, 1);
#undef MTB_POOLED
}

MTB_API int mtb_conv2d_forward_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                        const float* wt, const float* bias, float* y, int relu, void* stream) {
  return mtb_conv2d_forward_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, relu, nullptr, nullptr, stream, nullptr, 0);
}

MTB_API int mtb_conv2d_dgrad_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                      const float* wt, float* dx, void* stream) {
  return mtb_conv2d_dgrad_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx, stream, nullptr, 0);
}

int mtb_conv2d_dgrad_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy, const float* wt, float* dx,
                          void* stream, const int* guard, int guards) {
  ConvDims d;
  int rc = conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (rc) return rc;
  MTB_REQUIRE(dy && wt && dx, "conv2d_dgrad: null pointer");
  Out o{};
  o.out = dx; o.ld = cin; o.H = h; o.W = w; o.SH = sh; o.SW = sw;
  const Extra extra{guard, guards, nullptr};
  const DgradK a{dy, d, FastDiv(cout), nullptr};
  const DgradR b{wt, d, FastDiv(cout), nullptr};
  const bool va = cout % 4 == 0 && mtb_aligned16(dy), vb = cin % 4 == 0 && mtb_aligned16(wt);
  for (int first = 0; first < sh * sw; first += kMaxClasses) {
    const int classes = sh * sw - first < kMaxClasses ? sh * sw - first : kMaxClasses;
    ClassTable table;
    int rows = 0, K = 0;
    for (int q = 0; q < classes; ++q) {
      DgradClass& t = table.c[q];
      t.a = (first + q) / sw;
      t.b = (first + q) % sw;
      class_axis(t.a, h, kh, sh, ph, t.taps_h, t.start_h, t.count_h, t.c0_h);
      class_axis(t.b, w, kw, sw, pw, t.taps_w, t.start_w, t.count_w, t.c0_w);
      t.div_w = FastDiv(t.count_w > 0 ? t.count_w : 1);
      t.div_h = FastDiv(t.count_h > 0 ? t.count_h : 1);
      t.div_tw = FastDiv(t.taps_w > 0 ? t.taps_w : 1);
      if (n * t.count_h * t.count_w > rows) rows = n * t.count_h * t.count_w;
      if (t.taps_h * t.taps_w * cout > K) K = t.taps_h * t.taps_w * cout;
    }
    if (rows == 0) continue;
    const Choice c = choose(rows, cin, K, classes, 1);
    cudaStream_t st = (cudaStream_t)stream;
    if (va && vb) rc = launch<DgradK, 4, DgradR, 4>(c, a, b, o, table, classes, rows, cin, K, st, "conv2d_dgrad_simt", extra);
    else if (va) rc = launch<DgradK, 4, DgradR, 1>(c, a, b, o, table, classes, rows, cin, K, st, "conv2d_dgrad_simt", extra);
    else if (vb) rc = launch<DgradK, 1, DgradR, 4>(c, a, b, o, table, classes, rows, cin, K, st, "conv2d_dgrad_simt", extra);
    else rc = launch<DgradK, 1, DgradR, 1>(c, a, b, o, table, classes, rows, cin, K, st, "conv2d_dgrad_simt", extra);
    if (rc) return rc;
  }
  return MTB_OK;
}

MTB_API long long mtb_conv2d_wgrad_simt_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  ConvDims d;
  if (conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout)) return -1;
  const int slices = wgrad_choice(d).slices;
  return slices > 1 ? (long long)slices * cout * kh * kw * cin * 4 + 256 : 256;
}

namespace {

// out[i] = sum of the planes, in plane order; eight planes' loads in flight per thread.
__global__ void __launch_bounds__(256) add_planes_kernel(const float* __restrict__ ws, float* __restrict__ out, long long n, int planes) {
  mtb_launch_dependents();
  mtb_wait_prior();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float s = 0.f;
#pragma unroll 8
    for (int z = 0; z < planes; ++z) s += ws[z * n + i];
    out[i] = s;
  }
}

}  // namespace

MTB_API int mtb_conv2d_wgrad_simt_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                      const float* dy, float* dw, void* workspace, long long workspace_bytes, void* stream) {
  return mtb_conv2d_wgrad_simt(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, dy, dw, workspace, workspace_bytes, stream, nullptr, 0);
}

int mtb_conv2d_wgrad_simt(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* dy, float* dw,
                          void* workspace, long long workspace_bytes, void* stream, const int* guard, int guards) {
  ConvDims d;
  int rc = conv_dims(d, n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (rc) return rc;
  MTB_REQUIRE(x && dy && dw, "conv2d_wgrad: null pointer");
  const int K = kh * kw * cin, pixels = n * d.OH * d.OW;
  // guarded: one launch that usually does nothing, so its slices add up in clusters
  const Choice c = guard ? choose(cout, K, pixels, 1, 1) : wgrad_choice(d);
  const long long total = (long long)cout * K;
  cudaStream_t st = (cudaStream_t)stream;
  Out o{};
  o.out = dw; o.ld = K;
  const Extra extra{guard, guards, nullptr};
  if (c.slices > 1 && !guard) {
    MTB_REQUIRE(workspace && workspace_bytes >= c.slices * total * 4, "conv2d_wgrad: workspace too small");
    o.out = (float*)workspace;
    o.split_plane = total;
  }
  const DenseR a{dy, cout};
  const bool va = cout % 4 == 0 && mtb_aligned16(dy), vb = cin % 4 == 0 && mtb_aligned16(x);
  if (va && vb) rc = launch<DenseR, 4, PatchR, 4>(c, a, patch_r(x, d), o, NoTable{}, 1, cout, K, pixels, st, "conv2d_wgrad_simt", extra);
  else if (va) rc = launch<DenseR, 4, PatchR, 1>(c, a, patch_r(x, d), o, NoTable{}, 1, cout, K, pixels, st, "conv2d_wgrad_simt", extra);
  else if (vb) rc = launch<DenseR, 1, PatchR, 4>(c, a, patch_r(x, d), o, NoTable{}, 1, cout, K, pixels, st, "conv2d_wgrad_simt", extra);
  else rc = launch<DenseR, 1, PatchR, 1>(c, a, patch_r(x, d), o, NoTable{}, 1, cout, K, pixels, st, "conv2d_wgrad_simt", extra);
  if (rc || c.slices == 1 || guard) return rc;
  MTB_LAUNCH(add_planes_kernel, mtb_stream_grid(total, 256), 256, 0, st, (const float*)workspace, dw, total, c.slices);
  MTB_LAUNCH_CHECK("add_planes_kernel");
  return MTB_OK;
}
