// BatchNorm2d forward / backward over channels-last activations viewed as a [rows = N*H*W, C]
// matrix.  HBM-bound: forward reads x twice and writes y once (3S), backward reads x and dy
// twice and writes dx once (5S).  Per-channel statistics come from per-CTA Welford-style
// partials (shifted sums, Chan merge) combined in a fixed order by a one-CTA-per-256-channels
// finalise kernel, so results are bit-reproducible.
#include "colreduce.cuh"
#include "kernels.h"
#include <type_traits>

MTB_API long long mtb_batch_norm2d_workspace_bytes(int n, int c, int h, int w);

namespace {

// The order in which a pass walks its rows, in groups of kGroup iterations whose loads are issued (forward all, backward see partial_ahead) before the first value is used or stored.
// All CTAs work on neighbouring groups (grid stride), so that what the L2 holds at the end is one stretch of the tensor, and the pass behind it
// starts there: the normalise pass walks back to front behind a convolution that wrote front to back, the backward's sums do so behind a data
// gradient, and dx then front to back.  Single rows of a contiguous range a CTA -> groups, in these orders: ResNet-50 step at 128 images 18.50 -> 18.08 ms,
// ResNet-18 at 512 5465 -> 5353 us (5406 without the turns), at 128 1882 -> 1851, at 64 (captured) 1270 -> 1246.  rows_per_block > 0: a CTA
// takes that many rows one after the other; the sums do so up to 64 MB, which the L2 holds whole, and keep their order there.  Channels that are no fours
// walk a CTA's rows without any of this: their passes are bound by their instructions (207 channels on 69 x 17x17 with ReLU and pool, forward
// and backward: 114.9 us, the backward in groups 117.6; the forward of 150 channels on 30 x 50x50 40.4 us, in groups 42.3).
constexpr int kGroup = 4;
struct RowWalk {
  long long r, last, step, limit;  // first row of the group, of the last group, from group to group; end of the rows
  bool back;
  __device__ __forceinline__ RowWalk(long long rows, int R, long long rows_per_block, bool back_) {
    const long long group = (long long)kGroup * R;
    back = back_ && rows_per_block == 0;
    r = blockIdx.y * (rows_per_block ? rows_per_block : group);
    step = rows_per_block ? group : group * gridDim.y;
    limit = rows_per_block && r + rows_per_block < rows ? r + rows_per_block : rows;
    last = (rows - 1) / group * group;
  }
  __device__ __forceinline__ bool next(long long& first) {
    if (r >= limit) return false;
    first = back ? last - r : r;
    r += step;
    return true;
  }
};

// ---------------------------------------------------------------- forward: statistics

template <int V>
__global__ void __launch_bounds__(256) bn_stats_partial_kernel(const float* __restrict__ x, long long rows, int C, int L, long long rows_per_block,
                                                                float* __restrict__ partial) {
  mtb_launch_dependents();
  mtb_wait_prior();
  const int lane = threadIdx.x & (L - 1);
  const int rsub = threadIdx.x / L;
  const int R = 256 / L;
  const int cg = blockIdx.x * L + lane;  // column group
  const bool active = cg * V < C;
  long long r0 = blockIdx.y * rows_per_block;
  long long r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;

  float pivot[V], s1[V], s2[V];
  int cnt = 0;
#pragma unroll
  for (int i = 0; i < V; ++i) { pivot[i] = 0.f; s1[i] = 0.f; s2[i] = 0.f; }
  if (active) {
    long long r = r0 + rsub;
    if (r < r1) {
      VecF<V> f = vload<V>(x + r * C + (long long)cg * V);
#pragma unroll
      for (int i = 0; i < V; ++i) pivot[i] = f.v[i];
      cnt = 1;
      r += R;
    }
#pragma unroll 4
    for (; r < r1; r += R) {
      VecF<V> f = vload<V>(x + r * C + (long long)cg * V);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float d = f.v[i] - pivot[i];
        s1[i] += d;
        s2[i] += d * d;
      }
      ++cnt;
    }
  }
  __shared__ float sm_mean[V][256];
  __shared__ float sm_m2[V][256];
  __shared__ int sm_cnt[256];
  float inv = cnt > 0 ? 1.f / (float)cnt : 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    sm_mean[i][threadIdx.x] = pivot[i] + s1[i] * inv;
    sm_m2[i][threadIdx.x] = s2[i] - s1[i] * s1[i] * inv;
  }
  sm_cnt[threadIdx.x] = cnt;
  __syncthreads();
  if (rsub == 0 && active) {
    float n = (float)cnt;
    float mean[V], m2[V];
#pragma unroll
    for (int i = 0; i < V; ++i) { mean[i] = sm_mean[i][lane]; m2[i] = sm_m2[i][lane]; }
    for (int k = 1; k < R; ++k) {
      float nb = (float)sm_cnt[k * L + lane];
      if (nb == 0.f) continue;
      float nt = n + nb;
      float wb = nb / nt;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float d = sm_mean[i][k * L + lane] - mean[i];
        mean[i] += d * wb;
        m2[i] += sm_m2[i][k * L + lane] + d * d * n * wb;
      }
      n = nt;
    }
    float* p = partial + (long long)blockIdx.y * 3 * C + (long long)cg * V;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      p[i] = n;
      p[C + i] = mean[i];
      p[2 * C + i] = m2[i];
    }
  }
}

// Chan's parallel update of (count, mean, M2).  The finalise kernel below combines the per-CTA
// partials with it and writes the batch mean / biased variance, the per-channel scale
// gamma/sqrt(var+eps) used by the normalise pass, and the blended running statistics.
__device__ __forceinline__ void chan_merge(float& n, float& mean, float& m2, float nb, float mb, float qb) {
  if (nb == 0.f) return;
  float nt = n + nb;
  float d = mb - mean;
  float wb = nb / nt;
  mean += d * wb;
  m2 += qb + d * d * n * wb;
  n = nt;
}

__global__ void __launch_bounds__(1024) bn_stats_final_kernel(const float* __restrict__ partial, int P, int C, const float* __restrict__ gamma, float eps,
                                                               float one_minus_m, float m, float* running_mean, float* running_var,
                                                               float* __restrict__ mean_out, float* __restrict__ var_out, float* __restrict__ scale_out) {
  mtb_launch_dependents();
  mtb_wait_prior();
  // 8 channels x 128 partial-groups per CTA.  Group g merges partials g, g+128, ... (all loads are
  // issued before the first merge), then the 128 results are merged pairwise in a fixed tree, so the
  // kernel is a couple of memory round trips long and the result does not depend on scheduling.
  constexpr int G = 128, B = 5;
  const int cx = threadIdx.x & 7, g = threadIdx.x >> 3;
  const int c = blockIdx.x * 8 + cx;
  float n = 0.f, mean = 0.f, m2 = 0.f;
  // what the last step needs is on its way beside the partials: one round trip less in a kernel that is
  // all round trips (and in the backward's; ResNet-18 step captured at 64 images 1379 -> 1344 us, at batch 128 2026 -> 1994)
  const bool last = g == 0 && c < C;
  const float gam = last && gamma ? gamma[c] : 1.f;
  const float rm = last && running_mean ? running_mean[c] : 0.f, rv = last && running_var ? running_var[c] : 0.f;
  if (c < C) {
    for (int p0 = g; p0 < P; p0 += G * B) {
      float v[B][3];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int p = p0 + G * u;
        const float* q = partial + (long long)p * 3 * C + c;
        const bool in = p < P;
        v[u][0] = in ? q[0] : 0.f;
        v[u][1] = in ? q[C] : 0.f;
        v[u][2] = in ? q[2 * C] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u) chan_merge(n, mean, m2, v[u][0], v[u][1], v[u][2]);
    }
  }
  __shared__ float sn[G][9], smean[G][9], sm2[G][9];
  sn[g][cx] = n; smean[g][cx] = mean; sm2[g][cx] = m2;
#pragma unroll
  for (int s = G / 2; s >= 1; s >>= 1) {
    __syncthreads();
    if (g < s) {
      chan_merge(n, mean, m2, sn[g + s][cx], smean[g + s][cx], sm2[g + s][cx]);
      sn[g][cx] = n; smean[g][cx] = mean; sm2[g][cx] = m2;
    }
  }
  if (g != 0 || c >= C) return;
  float mu = mean;
  float var = n > 0.f ? m2 / n : 0.f;
  mean_out[c] = mu;
  var_out[c] = var;
  float rstd = 1.0f / sqrtf(var + eps);
  scale_out[c] = gamma ? gam * rstd : rstd;
  if (running_mean) running_mean[c] = __fadd_rn(__fmul_rn(one_minus_m, rm), __fmul_rn(m, mu));
  if (running_var) running_var[c] = __fadd_rn(__fmul_rn(one_minus_m, rv), __fmul_rn(m, var));
}

// Inference mode: statistics are the running ones.
__global__ void bn_eval_prep_kernel(int C, const float* __restrict__ gamma, float eps, const float* __restrict__ rm, const float* __restrict__ rv,
                                    float* __restrict__ mean_out, float* __restrict__ var_out, float* __restrict__ scale_out) {
  mtb_launch_dependents();
  mtb_wait_prior();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  mean_out[c] = rm[c];
  var_out[c] = rv[c];
  float rstd = 1.0f / sqrtf(rv[c] + eps);
  scale_out[c] = gamma ? gamma[c] * rstd : rstd;
}

// ---------------------------------------------------------------- forward: normalise

// MODE 2 with mask != NULL also writes one byte per four channels, bit i set where the ReLU blocked channel i: backward then
// needs neither the added tensor nor the arithmetic that would decide it again, two passes over a tensor less of eight.
// With var != NULL (running statistics) `scale` holds gamma, or is NULL, and the scale is computed here.
// MODE 0: y = bn(x); 1: y = max(0, bn(x)); 2: y = max(0, bn(x) + res) (res has the shape of x)
template <int V, int MODE>
__global__ void __launch_bounds__(256) bn_normalize_kernel(const float* x, float* y, long long rows, int C, int L, long long rows_per_block, const float* __restrict__ mean,
                                                            const float* __restrict__ scale, const float* __restrict__ beta,
                                                            const float* __restrict__ res, const float* __restrict__ var, float eps,
                                                            unsigned char* __restrict__ mask) {
  mtb_launch_dependents();
  mtb_wait_prior();
  const int lane = threadIdx.x & (L - 1);
  const int rsub = threadIdx.x / L;
  const int R = 256 / L;
  const int cg = blockIdx.x * L + lane;
  if (cg * V >= C) return;
  float mu[V], g[V], b[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    mu[i] = mean[cg * V + i];
    if (var) {
      const float rstd = 1.0f / sqrtf(var[cg * V + i] + eps);
      g[i] = scale ? scale[cg * V + i] * rstd : rstd;
    } else {
      g[i] = scale[cg * V + i];
    }
    b[i] = beta ? beta[cg * V + i] : 0.f;
  }
  // Four rows are loaded before the first is stored: x may be y (an update in place), so the compiler would not do it.  BatchNorm,
  // ReLU and pooling of 256 x 128 x 56 x 56, forward and backward: 1073 -> 1050 us; ResNet-18 step at 512 images 5.84 -> 5.78 ms.
  constexpr int AHEAD = kGroup;
  auto group = [&](long long r, long long limit) {
    const long long off = r * C + (long long)cg * V, step = (long long)R * C;
    VecF<V> f[AHEAD], a[MODE == 2 ? AHEAD : 1];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (r + u * R < limit) {
        f[u] = vload<V>(x + off + u * step);
        if (MODE == 2) a[u] = vload<V>(res + off + u * step);
      }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (r + u * R >= limit) break;
      unsigned negative = 0;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float t = (f[u].v[i] - mu[i]) * g[i] + b[i];
        if (MODE == 2) { t = t + a[u].v[i]; negative |= (t < 0.f ? 1u : 0u) << i; }
        f[u].v[i] = MODE ? fmaxf(t, 0.f) : t;
      }
      vstore<V>(y + off + u * step, f[u]);
      if (MODE == 2 && V == 4 && mask) mask[(off + u * step) / 4] = (unsigned char)negative;
    }
  };
  if (V == 1) {  // see RowWalk
    const long long r0 = blockIdx.y * rows_per_block, r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;
    for (long long r = r0 + rsub; r < r1; r += AHEAD * R) group(r, r1);
  } else {
    RowWalk walk(rows, R, 0, true);
    for (long long r; walk.next(r);) group(r + rsub, walk.limit);
  }
}

// y = max_pool(max(0, bn(x))), four channels of one window a thread, with the pool's tie mask (bit WIN * line + column of every element that equals the
// maximum).  WIN = 2: 2 x 2 windows of stride 2; 3: 3 x 3 windows of stride 2 with a border of one, whose values count as 0.  The normalised tensor is
// neither written nor read (2 x 2: S + S/4 instead of 3S + S/4 of traffic), and a launch goes.  The digit classifier's training step at 64 images,
// bound by the host, with the backward below: 60 launches -> 54, 340 -> 316 us.  64 channels of 128 x 112x112, 3 x 3: 233 -> 140 us.
template <int WIN>
__global__ void __launch_bounds__(256) bn_relu_pool_kernel(const float4* __restrict__ x, float4* __restrict__ y, uint2* __restrict__ mask, PoolDiv cv, PoolDiv ow_,
                                                            PoolDiv oh_, int H, int W, const float* __restrict__ mean, const float* __restrict__ scale,
                                                            const float* __restrict__ beta, unsigned total) {
  mtb_launch_dependents();
  mtb_wait_prior();
  constexpr int PAD = WIN == 3 ? 1 : 0, N = WIN * WIN;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    unsigned cg, ow, oh;
    const unsigned n = oh_.divmod(ow_.divmod(cv.divmod(i, cg), ow), oh);
    const int h0 = 2 * (int)oh - PAD, w0 = 2 * (int)ow - PAD;
    float4 v[N];
    bool in[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {  // all loads before the first comparison
      const int h = h0 + k / WIN, w = w0 + k % WIN;
      in[k] = PAD == 0 || ((unsigned)h < (unsigned)H && (unsigned)w < (unsigned)W);
      if (in[k]) v[k] = __ldg(x + ((size_t)(n * H + h) * W + w) * cv.d + cg);
    }
    const float4 mu = ld4(mean + 4 * cg), g = ld4(scale + 4 * cg), b = beta ? ld4(beta + 4 * cg) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 best = make_float4(0.f, 0.f, 0.f, 0.f);  // nothing behind a ReLU is less
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (in[k]) {
        v[k].x = fmaxf((v[k].x - mu.x) * g.x + b.x, 0.f); v[k].y = fmaxf((v[k].y - mu.y) * g.y + b.y, 0.f);
        v[k].z = fmaxf((v[k].z - mu.z) * g.z + b.z, 0.f); v[k].w = fmaxf((v[k].w - mu.w) * g.w + b.w, 0.f);
      } else {
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      best.x = fmaxf(best.x, v[k].x); best.y = fmaxf(best.y, v[k].y); best.z = fmaxf(best.z, v[k].z); best.w = fmaxf(best.w, v[k].w);
    }
    unsigned m0 = 0, m1 = 0, m2 = 0, m3 = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      m0 |= (v[k].x == best.x ? 1u : 0u) << k; m1 |= (v[k].y == best.y ? 1u : 0u) << k;
      m2 |= (v[k].z == best.z ? 1u : 0u) << k; m3 |= (v[k].w == best.w ? 1u : 0u) << k;
    }
    y[i] = best;
    mask[i] = make_uint2(m0 | (m1 << 16), m2 | (m3 << 16));
  }
}

// ---------------------------------------------------------------- backward

// Rows of a group whose loads are issued together (the order of the rows is the same).  The sums' grid is four CTAs an SM, in which four rows take 74 to 94
// registers: two or three CTAs fit.  Two are as good as four, since the grid is two whole turns of them; three leave a second turn with a third of the CTAs.
// BatchNorm by itself (MODE 0) had three so, and has four in 64 registers with two rows: backward of 60 x 64 x 33x33 17.1 -> 15.6 us, 60 x 132 x 33x33 37.7 ->
// 36.4, 120 x 132 x 28x28 55.6 -> 52.3, 70 x 256 x 55x55 176.2 -> 170.6.  Behind a pool (MODE 4), whose loads are three and not neighbours, both passes are for
// it: 67.8 -> 56.4 on 70 x 64 x 55x55, 242 -> 178 on 70 x 132 x 55x55, 257 -> 194 on 70 x 256 x 55x55.
// With ReLU or addition two rows win 0 to 6 % alone and lose 0.3 to 1.3 % of a ResNet step, where weight gradients want the registers beside them.
constexpr int partial_ahead(int mode) { return mode == 0 || mode == 4 ? 2 : kGroup; }
constexpr int dx_ahead(int mode) { return mode == 4 ? 2 : kGroup; }

// MODE 4: MODE 1 whose upstream gradient goes through a 2 x 2 max-pool of stride 2 first: dy and the tie mask have the shape of its result.  (For
// 3 x 3 windows, up to four a pixel, both passes then wait for their windows: 64 channels of 128 x 112x112 380 and 503 us, against 102 for the
// pool's own backward and 316 for two passes over what it writes.)
struct PooledGradient {
  const unsigned short* mask;
  PoolDiv w, h;
  unsigned OW, OH;
};
struct NotPooled {};
template <int MODE>
using GradientSource = std::conditional_t<MODE == 4, PooledGradient, NotPooled>;
template <int V, int MODE>
__device__ __forceinline__ VecF<V> load_gradient(const float* __restrict__ dy, long long row, int C, int channel, const GradientSource<MODE>& pool) {
  if constexpr (MODE == 4) {
    unsigned w, h;
    const unsigned n = pool.h.divmod(pool.w.divmod((unsigned)row, w), h);
    VecF<V> g;
#pragma unroll
    for (int i = 0; i < V; ++i) g.v[i] = 0.f;
    if (h / 2 < pool.OH && w / 2 < pool.OW) {  // a last odd line or column lies in no window
      const size_t o = ((size_t)(n * pool.OH + h / 2) * pool.OW + w / 2) * C + channel;
      const unsigned bit = 1u << (2 * (h & 1) + (w & 1));
      const uint2 m = *reinterpret_cast<const uint2*>(pool.mask + o);
      const VecF<V> d = vload<V>(dy + o);
      g.v[0] = m.x & bit ? d.v[0] : 0.f;
      g.v[1 % V] = m.x >> 16 & bit ? d.v[1 % V] : 0.f;
      g.v[2 % V] = m.y & bit ? d.v[2 % V] : 0.f;
      g.v[3 % V] = m.y >> 16 & bit ? d.v[3 % V] : 0.f;
    }
    return g;
  } else {
    return vload<V>(dy + row * C + channel);
  }
}

// partial[p][0][c] = sum dy, partial[p][1][c] = sum dy * xhat over the CTA's rows.
// MODE 3: MODE 2 with the mask forward wrote (four channels a byte) instead of the added tensor.
// MODE 1 / 2: the forward output went through max(0, .) (MODE 2: after adding `res`) in the same pass;
// the upstream gradient is first masked where the (recomputed, bit-identical) value was negative.
template <int V, int MODE>
__global__ void __launch_bounds__(256, partial_ahead(MODE) == 2 ? 4 : 0 /* as many as the compiler likes */) bn_bwd_partial_kernel(const float* __restrict__ dy, const float* __restrict__ x, long long rows, int C, int L, long long rows_per_block, const float* __restrict__ mean,
                                                              const float* __restrict__ var, float eps, const float* __restrict__ gamma,
                                                              const float* __restrict__ beta, float* __restrict__ partial,
                                                              const float* __restrict__ res, const unsigned char* __restrict__ mask, const GradientSource<MODE> pool) {
  mtb_launch_dependents();
  mtb_wait_prior();
  const int lane = threadIdx.x & (L - 1);
  const int rsub = threadIdx.x / L;
  const int R = 256 / L;
  const int cg = blockIdx.x * L + lane;
  const bool active = cg * V < C;
  float mu[V], rstd[V], a0[V], a1[V], gs[V], bt[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    a0[i] = 0.f; a1[i] = 0.f;
    mu[i] = active ? mean[cg * V + i] : 0.f;
    rstd[i] = active ? 1.0f / sqrtf(var[cg * V + i] + eps) : 0.f;
    gs[i] = (active && gamma) ? gamma[cg * V + i] * rstd[i] : rstd[i];
    bt[i] = (active && beta) ? beta[cg * V + i] : 0.f;
  }
  auto add = [&](const VecF<V>& g, const VecF<V>& f, const VecF<V>& a, unsigned negative) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float gi = g.v[i];
      if (MODE == 3) {
        if (negative >> i & 1u) gi = 0.f;
      } else if (MODE) {
        float t = (f.v[i] - mu[i]) * gs[i] + bt[i];
        if (MODE == 2) t = t + a.v[i];
        if (t < 0.f) gi = 0.f;
      }
      a0[i] += gi;
      a1[i] += gi * ((f.v[i] - mu[i]) * rstd[i]);
    }
  };
  if (V == 1 && active) {  // see RowWalk
    const long long r0 = blockIdx.y * rows_per_block, r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;
#pragma unroll 4
    for (long long r = r0 + rsub; r < r1; r += R) {
      const long long off = r * C + cg;
      VecF<V> a;
      if (MODE == 2) a = vload<V>(res + off);
      add(load_gradient<V, MODE>(dy, r, C, cg, pool), vload<V>(x + off), a, 0u);
    }
  } else if (active) {
    RowWalk walk(rows, R, rows_per_block, true);
    for (long long r0; walk.next(r0);) {
      constexpr int AHEAD = partial_ahead(MODE);
      r0 += rsub;
#pragma unroll 1
      for (int part = 0; part < kGroup / AHEAD; ++part, r0 += AHEAD * R) {
        VecF<V> g[AHEAD], f[AHEAD], a[MODE == 2 ? AHEAD : 1];
        unsigned negative[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          if (r0 + u * R < walk.limit) {
            const long long off = (r0 + u * R) * C + (long long)cg * V;
            g[u] = load_gradient<V, MODE>(dy, r0 + u * R, C, cg * V, pool);
            f[u] = vload<V>(x + off);
            if (MODE == 2) a[u] = vload<V>(res + off);
            negative[u] = MODE == 3 ? mask[off / 4] : 0u;
          }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          if (r0 + u * R >= walk.limit) break;
          add(g[u], f[u], a[MODE == 2 ? u : 0], negative[u]);
        }
      }
    }
  }
  __shared__ float sm0[V][256];
  __shared__ float sm1[V][256];
#pragma unroll
  for (int i = 0; i < V; ++i) { sm0[i][threadIdx.x] = a0[i]; sm1[i][threadIdx.x] = a1[i]; }
  __syncthreads();
  if (rsub == 0 && active) {
    for (int k = 1; k < R; ++k) {
#pragma unroll
      for (int i = 0; i < V; ++i) { a0[i] += sm0[i][k * L + lane]; a1[i] += sm1[i][k * L + lane]; }
    }
    float* p = partial + (long long)blockIdx.y * 2 * C + (long long)cg * V;
#pragma unroll
    for (int i = 0; i < V; ++i) { p[i] = a0[i]; p[C + i] = a1[i]; }
  }
}

// dbeta = sum dy, dgamma = sum dy*xhat; coefficients for dx = k1 * (dy - k2 - (x - mean) * k3).
// Thirty-two threads per channel, fixed summation order.
__global__ void __launch_bounds__(1024) bn_bwd_final_kernel(const float* __restrict__ partial, int P, int C, const float* __restrict__ gamma,
                                                             const float* __restrict__ var, float eps, float inv_m, float* __restrict__ dgamma,
                                                             float* __restrict__ dbeta, float* __restrict__ coef) {
  mtb_launch_dependents();
  mtb_wait_prior();
  // 8 channels x 128 partial-groups per CTA, loads first, then a fixed pairwise tree (see above).
  constexpr int G = 128, B = 5;
  const int cx = threadIdx.x & 7, g = threadIdx.x >> 3;
  const int c = blockIdx.x * 8 + cx;
  float s0 = 0.f, s1 = 0.f;
  const bool last = g == 0 && c < C;
  const float gm = last && gamma ? gamma[c] : 1.f, variance = last ? var[c] : 1.f;
  if (c < C) {
    for (int p0 = g; p0 < P; p0 += G * B) {
      float v[B][2];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const int p = p0 + G * u;
        const bool in = p < P;
        v[u][0] = in ? partial[(long long)p * 2 * C + c] : 0.f;
        v[u][1] = in ? partial[(long long)p * 2 * C + C + c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < B; ++u) { s0 += v[u][0]; s1 += v[u][1]; }
    }
  }
  __shared__ float t0[G][9], t1[G][9];
  t0[g][cx] = s0; t1[g][cx] = s1;
#pragma unroll
  for (int s = G / 2; s >= 1; s >>= 1) {
    __syncthreads();
    if (g < s) {
      s0 += t0[g + s][cx]; s1 += t1[g + s][cx];
      t0[g][cx] = s0; t1[g][cx] = s1;
    }
  }
  if (g != 0 || c >= C) return;
  float db = s0, dg = s1;
  if (dbeta) dbeta[c] = db;
  if (dgamma) dgamma[c] = dg;
  float rstd = 1.0f / sqrtf(variance + eps);
  coef[c] = gm * rstd;               // k1
  coef[C + c] = db * inv_m;          // k2
  coef[2 * C + c] = rstd * dg * inv_m;  // k3: (x - mean) * k3 = xhat * dgamma / m
}

// MODES 2 and 3 also write the masked upstream gradient, which is the gradient of the added tensor, to dres.  rows_per_block: of single rows (V = 1) alone.
template <int V, int MODE>
__global__ void __launch_bounds__(256) bn_bwd_dx_kernel(const float* __restrict__ dy, const float* __restrict__ x, float* __restrict__ dx,
                                                         long long rows, int C, int L, long long rows_per_block,
                                                         const float* __restrict__ mean, const float* __restrict__ coef,
                                                         const float* __restrict__ beta, const float* __restrict__ res, float* __restrict__ dres,
                                                         const unsigned char* __restrict__ mask, const GradientSource<MODE> pool) {
  mtb_launch_dependents();
  mtb_wait_prior();
  const int lane = threadIdx.x & (L - 1);
  const int rsub = threadIdx.x / L;
  const int R = 256 / L;
  const int cg = blockIdx.x * L + lane;
  if (cg * V >= C) return;
  float mu[V], k1[V], k2[V], k3[V], bt[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    mu[i] = mean[cg * V + i];
    k1[i] = coef[cg * V + i];
    k2[i] = coef[C + cg * V + i];
    k3[i] = coef[2 * C + cg * V + i];
    bt[i] = beta ? beta[cg * V + i] : 0.f;
  }
  auto store = [&](long long off, VecF<V>& g, const VecF<V>& f, const VecF<V>& a, unsigned negative) {
    VecF<V> m;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float gi = g.v[i];
      if (MODE == 3) {
        if (negative >> i & 1u) gi = 0.f;
      } else if (MODE) {
        float t = (f.v[i] - mu[i]) * k1[i] + bt[i];  // k1 = gamma / sigma, the forward's scale
        if (MODE == 2) t = t + a.v[i];
        if (t < 0.f) gi = 0.f;
      }
      m.v[i] = gi;
      g.v[i] = k1[i] * (gi - k2[i] - (f.v[i] - mu[i]) * k3[i]);
    }
    vstore<V>(dx + off, g);
    if (MODE == 2 || MODE == 3) vstore<V>(dres + off, m);
  };
  if (V == 1) {  // see RowWalk
    const long long r0 = blockIdx.y * rows_per_block, r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;
#pragma unroll 4
    for (long long r = r0 + rsub; r < r1; r += R) {
      const long long off = r * C + cg;
      VecF<V> a;
      if (MODE == 2) a = vload<V>(res + off);
      VecF<V> g = load_gradient<V, MODE>(dy, r, C, cg, pool);
      store(off, g, vload<V>(x + off), a, 0u);
    }
    return;
  }
  RowWalk walk(rows, R, 0, false);
  for (long long r0; walk.next(r0);) {
    constexpr int AHEAD = dx_ahead(MODE);
    r0 += rsub;
#pragma unroll 1
    for (int part = 0; part < kGroup / AHEAD; ++part, r0 += AHEAD * R) {
      VecF<V> g[AHEAD], f[AHEAD], a[MODE == 2 ? AHEAD : 1];
      unsigned negative[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        if (r0 + u * R < walk.limit) {
          const long long off = (r0 + u * R) * C + (long long)cg * V;
          g[u] = load_gradient<V, MODE>(dy, r0 + u * R, C, cg * V, pool);
          f[u] = vload<V>(x + off);
          if (MODE == 2) a[u] = vload<V>(res + off);
          negative[u] = MODE == 3 ? mask[off / 4] : 0u;
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        if (r0 + u * R >= walk.limit) break;
        store((r0 + u * R) * C + (long long)cg * V, g[u], f[u], a[MODE == 2 ? u : 0], negative[u]);
      }
    }
  }
}

// A streaming pass wants more CTAs than a reduction (no partial rows to combine afterwards).
ColCfg stream_cfg(long long rows, int C, bool aligned) {
  ColCfg c = mtb_col_cfg(rows, C, aligned);
  long long target = (long long)mtb_sm_count() * 8 / c.col_blocks;
  if (target < 1) target = 1;
  long long min_rows = (long long)c.rows_per_iter * 4;
  long long want = (rows + min_rows - 1) / min_rows;
  if (want < 1) want = 1;
  long long rb = want < target ? want : target;
  long long rpb = (rows + rb - 1) / rb;
  rpb = (rpb + c.rows_per_iter - 1) / c.rows_per_iter * c.rows_per_iter;
  c.rows_per_block = rpb;
  c.row_blocks = (int)((rows + rpb - 1) / rpb);
  return c;
}

// Launch latency shows in chains over small tensors only; over large ones CTAs that wait early keep weight gradients of the
// side stream off the SMs (ResNet-18 at 512 images 0.6 % slower with it, at 128 images 5 % faster).
bool short_chain(long long rows, int c) { return rows * c * 4 <= (64ll << 20); }

int launch_normalize(const float* x, float* y, long long rows, int c, bool aligned, const float* mean, const float* scale, const float* beta,
                     int mode, const float* res, cudaStream_t st, const float* var = nullptr, float eps = 0.f,
                     unsigned char* mask = nullptr) {
  ColCfg s = stream_cfg(rows, c, aligned);
  dim3 grid(s.col_blocks, s.row_blocks);
#define MTB_BN_NORM(V_, M_) MTB_CUDA(mtb_launch_after(short_chain(rows, c), bn_normalize_kernel<V_, M_>, grid, dim3(256), 0, st, x, y, rows, c, s.lanes, s.rows_per_block, mean, scale, beta, res, var, eps, mask))
  if (s.vec == 4) { if (mode == 2) MTB_BN_NORM(4, 2); else if (mode == 1) MTB_BN_NORM(4, 1); else MTB_BN_NORM(4, 0); }
  else { if (mode == 2) MTB_BN_NORM(1, 2); else if (mode == 1) MTB_BN_NORM(1, 1); else MTB_BN_NORM(1, 0); }
#undef MTB_BN_NORM
  MTB_LAUNCH_CHECK("bn_normalize_kernel");
  return MTB_OK;
}

// What 2 x 2 windows of stride 2, and 3 x 3 ones with a border of one, leave of an extent.
int pooled_extent(int size, int window) { return window == 2 ? size / 2 : (size + 1) / 2; }

// mode 0: y = bn(x); 1: y = max(0, bn(x)); 2: y = max(0, bn(x) + res).  stats / stats_rows: batch statistics
// prepared by the producer of x as partial rows (see mtb_conv2d_forward_stats_f32); 0 rows = compute them here.
int bn_forward(int n, int c, int h, int w, const float* x, const float* gamma, const float* beta, double eps, int training, double momentum,
               float* running_mean, float* running_var, float* y, float* mean, float* var, int mode, const float* res, unsigned char* mask,
               const float* stats, int stats_rows, void* workspace, long long workspace_bytes, cudaStream_t st, unsigned short* ties = nullptr, int window = 0) {
  const MtbScratchTurn turn;
  MTB_REQUIRE(n > 0 && c > 0 && h > 0 && w > 0 && x && y && mean && var && workspace, "batch_norm2d_forward: bad arguments");
  MTB_REQUIRE(workspace_bytes >= mtb_batch_norm2d_workspace_bytes(n, c, h, w), "batch_norm2d_forward: workspace too small");
  MTB_REQUIRE(training || (running_mean && running_var), "batch_norm2d_forward: inference needs running statistics");
  MTB_REQUIRE(mode != 2 || res, "batch_norm2d_add_relu_forward: the tensor to add is missing");
  long long rows = (long long)n * h * w;
  bool aligned = mtb_aligned16(x) && mtb_aligned16(y) && (mode != 2 || mtb_aligned16(res));
  MTB_REQUIRE(!mask || (aligned && c % 4 == 0), "batch_norm2d_add_relu_forward: a mask needs four channels a byte and 16-byte alignment");
  float* partial = (float*)workspace;
  float* scale = partial + (long long)mtb_col_max_partials() * 3 * c;
  if (training) {
    int P = stats_rows;
    if (!(stats && stats_rows > 0)) {
      ColCfg cfg = mtb_col_cfg(rows, c, mtb_aligned16(x));
      dim3 grid(cfg.col_blocks, cfg.row_blocks);
      if (cfg.vec == 4) MTB_LAUNCH(bn_stats_partial_kernel<4>, grid, 256, 0, st, x, rows, c, cfg.lanes, cfg.rows_per_block, partial);
      else MTB_LAUNCH(bn_stats_partial_kernel<1>, grid, 256, 0, st, x, rows, c, cfg.lanes, cfg.rows_per_block, partial);
      MTB_LAUNCH_CHECK("bn_stats_partial_kernel");
      stats = partial;
      P = cfg.row_blocks;
    }
    MTB_CUDA(mtb_launch_after(short_chain(rows, c), bn_stats_final_kernel, dim3(mtb_div_up(c, 8)), dim3(1024), 0, st, stats, P, c, gamma, (float)eps, (float)(1.0 - momentum),
                              (float)momentum, running_mean, running_var, mean, var, scale));
    MTB_LAUNCH_CHECK("bn_stats_final_kernel");
  } else {
    MTB_LAUNCH(bn_eval_prep_kernel, mtb_div_up(c, 128), 128, 0, st, c, gamma, (float)eps, running_mean, running_var, mean, var, scale);
    MTB_LAUNCH_CHECK("bn_eval_prep_kernel");
  }
  if (ties) {
    const int oh = pooled_extent(h, window), ow = pooled_extent(w, window);
    const unsigned total = (unsigned)((long long)n * oh * ow * (c / 4));
    const int grid = mtb_stream_grid(total, 256);
#define MTB_BN_POOL(W_) \
  MTB_LAUNCH(bn_relu_pool_kernel<W_>, grid, 256, 0, st, (const float4*)x, (float4*)y, (uint2*)ties, PoolDiv(c / 4), PoolDiv(ow), PoolDiv(oh), h, w, mean, scale, beta, total)
    if (window == 2) MTB_BN_POOL(2); else MTB_BN_POOL(3);
#undef MTB_BN_POOL
    MTB_LAUNCH_CHECK("bn_relu_pool_kernel");
    return MTB_OK;
  }
  return launch_normalize(x, y, rows, c, aligned, mean, scale, beta, mode, res, st, nullptr, 0.f, mask);
}

// dx = gamma/sigma * (g - dbeta/m - xhat * dgamma/m) with g = dy masked by the forward's ReLU (modes 1, 2);
// mode 2 also writes g to dres (the gradient of the added tensor).
int bn_backward(int n, int c, int h, int w, const float* dy, const float* mean, const float* var, const float* x, const float* gamma,
                const float* beta, double eps, int mode, const float* res, const unsigned char* mask, float* dx, float* dres, float* dgamma, float* dbeta, void* workspace,
                long long workspace_bytes, cudaStream_t st, const unsigned short* ties = nullptr) {
  const MtbScratchTurn turn;
  MTB_REQUIRE(n > 0 && c > 0 && h > 0 && w > 0 && dy && mean && var && x && dx && workspace, "batch_norm2d_backward: bad arguments");
  MTB_REQUIRE(workspace_bytes >= mtb_batch_norm2d_workspace_bytes(n, c, h, w), "batch_norm2d_backward: workspace too small");
  MTB_REQUIRE(mode != 2 || ((res || mask) && dres), "batch_norm2d_add_relu_backward: the added tensor (or forward's mask) and its gradient buffer are required");
  long long rows = (long long)n * h * w;
  bool aligned = mtb_aligned16(x) && mtb_aligned16(dy) && mtb_aligned16(dx) && (mode != 2 || (mtb_aligned16(res) && mtb_aligned16(dres)));
  if (mode == 2 && mask) {
    MTB_REQUIRE(aligned && c % 4 == 0, "batch_norm2d_add_relu_backward: a mask needs four channels a byte and 16-byte alignment");
    mode = 3;
  }
  float* partial = (float*)workspace;
  float* coef = partial + (long long)mtb_col_max_partials() * 3 * c;  // 3*C floats fit in the 4*C tail
  ColCfg cfg = mtb_col_cfg(rows, c, aligned);
  dim3 grid(cfg.col_blocks, cfg.row_blocks);
#define MTB_BN_PARTIAL(V_, M_) \
  MTB_LAUNCH(bn_bwd_partial_kernel<V_, M_>, grid, 256, 0, st, dy, x, rows, c, cfg.lanes, short_chain(rows, c) || cfg.vec == 1 ? cfg.rows_per_block : 0, mean, var, (float)eps, gamma, beta, \
             partial, res, mask, GradientSource<M_>{})
  const PooledGradient pooled{ties, PoolDiv(w), PoolDiv(h), (unsigned)(w / 2), (unsigned)(h / 2)};
  if (ties)
    MTB_LAUNCH(bn_bwd_partial_kernel<4, 4>, grid, 256, 0, st, dy, x, rows, c, cfg.lanes, short_chain(rows, c) ? cfg.rows_per_block : 0, mean, var, (float)eps, gamma, beta,
               partial, res, mask, pooled);
  else if (cfg.vec == 4) { if (mode == 3) MTB_BN_PARTIAL(4, 3); else if (mode == 2) MTB_BN_PARTIAL(4, 2); else if (mode == 1) MTB_BN_PARTIAL(4, 1); else MTB_BN_PARTIAL(4, 0); }
  else { if (mode == 2) MTB_BN_PARTIAL(1, 2); else if (mode == 1) MTB_BN_PARTIAL(1, 1); else MTB_BN_PARTIAL(1, 0); }
#undef MTB_BN_PARTIAL
  MTB_LAUNCH_CHECK("bn_bwd_partial_kernel");
  MTB_CUDA(mtb_launch_after(short_chain(rows, c), bn_bwd_final_kernel, dim3(mtb_div_up(c, 8)), dim3(1024), 0, st, partial, cfg.row_blocks, c, gamma, var, (float)eps,
                            (float)(1.0 / (double)rows), dgamma, dbeta, coef));
  MTB_LAUNCH_CHECK("bn_bwd_final_kernel");
  ColCfg s = stream_cfg(rows, c, aligned);
  dim3 g2(s.col_blocks, s.row_blocks);
#define MTB_BN_DX(V_, M_) MTB_CUDA(mtb_launch_after(short_chain(rows, c), bn_bwd_dx_kernel<V_, M_>, g2, dim3(256), 0, st, dy, x, dx, rows, c, s.lanes, s.rows_per_block, mean, coef, beta, res, dres, mask, GradientSource<M_>{}))
  if (ties)
    MTB_CUDA(mtb_launch_after(short_chain(rows, c), bn_bwd_dx_kernel<4, 4>, g2, dim3(256), 0, st, dy, x, dx, rows, c, s.lanes, s.rows_per_block, mean, coef, beta, res, dres, mask, pooled));
  else if (s.vec == 4) { if (mode == 3) MTB_BN_DX(4, 3); else if (mode == 2) MTB_BN_DX(4, 2); else if (mode == 1) MTB_BN_DX(4, 1); else MTB_BN_DX(4, 0); }
  else { if (mode == 2) MTB_BN_DX(1, 2); else if (mode == 1) MTB_BN_DX(1, 1); else MTB_BN_DX(1, 0); }
#undef MTB_BN_DX
  MTB_LAUNCH_CHECK("bn_bwd_dx_kernel");
  return MTB_OK;
}

}  // namespace

int mtb_bn_eval_apply(const float* x, float* y, long long rows, int c, const MtbBnEval& bn, const float* residual, int relu, cudaStream_t st) {
  const bool aligned = mtb_aligned16(x) && mtb_aligned16(y) && mtb_aligned16(residual);
  return launch_normalize(x, y, rows, c, aligned, bn.mean, bn.gamma, bn.beta, residual ? 2 : (relu ? 1 : 0), residual, st, bn.var, bn.eps);
}

// Scratch the forward and backward entry points need, in bytes (an upper bound for the shape).
MTB_API long long mtb_batch_norm2d_workspace_bytes(int n, int c, int h, int w) {
  (void)n; (void)h; (void)w;
  long long floats = (long long)mtb_col_max_partials() * 3 * c + 4LL * c;
  return floats * 4 + 256;
}

// Training: batch statistics (biased variance also goes into running_var). Inference: running
// statistics. x, y are channels-last [N,H,W,C]; mean/var outputs are [C]. gamma/beta/running_*
// may be NULL. relu != 0 applies max(0, .) to y in the same pass.
MTB_API int mtb_batch_norm2d_forward_f32(int n, int c, int h, int w, const float* x, const float* gamma, const float* beta, double eps,
                                         int training, double momentum, float* running_mean, float* running_var, float* y,
                                         float* mean, float* var, int relu, void* workspace, long long workspace_bytes, void* stream) {
  return bn_forward(n, c, h, w, x, gamma, beta, eps, training, momentum, running_mean, running_var, y, mean, var, relu ? 1 : 0, nullptr, nullptr, nullptr, 0,
                    workspace, workspace_bytes, (cudaStream_t)stream);
}

// Training-mode forward whose batch statistics were prepared by the producer of x: `stats` holds
// stats_rows partial rows [row][3][C] of per-channel (count, mean, M2) that together cover every element
// of x exactly once (mtb_conv2d_forward_stats_f32 writes them from the convolution's epilogue).  The
// statistics pass over x is skipped: the partials are merged (fixed order), then x is normalised.
MTB_API int mtb_batch_norm2d_forward_prestats_f32(int n, int c, int h, int w, const float* x, const float* gamma, const float* beta, double eps,
                                                  double momentum, float* running_mean, float* running_var, float* y, float* mean, float* var,
                                                  int relu, const float* stats, int stats_rows, void* workspace, long long workspace_bytes,
                                                  void* stream) {
  MTB_REQUIRE(stats && stats_rows > 0, "batch_norm2d_forward_prestats: no statistics rows");
  return bn_forward(n, c, h, w, x, gamma, beta, eps, 1, momentum, running_mean, running_var, y, mean, var, relu ? 1 : 0, nullptr, nullptr, stats, stats_rows,
                    workspace, workspace_bytes, (cudaStream_t)stream);
}

// y = max(0, batch_norm(x) + residual): the tail of a residual block (BatchNorm, shortcut addition, ReLU) in
// one normalise pass; the BatchNorm output is never stored.  stats / stats_rows as above (NULL / 0: the
// statistics are computed here).  residual has the shape of x.
MTB_API int mtb_batch_norm2d_add_relu_forward_f32(int n, int c, int h, int w, const float* x, const float* residual, const float* gamma,
                                                  const float* beta, double eps, int training, double momentum, float* running_mean,
                                                  float* running_var, float* y, float* mean, float* var, const float* stats, int stats_rows,
                                                  void* workspace, long long workspace_bytes, void* stream) {
  return bn_forward(n, c, h, w, x, gamma, beta, eps, training, momentum, running_mean, running_var, y, mean, var, 2, residual, nullptr, stats,
                    stats_rows, workspace, workspace_bytes, (cudaStream_t)stream);
}

// The same, and the ReLU's mask for the backward below: n*h*w*c/4 bytes, bit i of a byte set where channel i of its four was
// blocked.  c must be a multiple of 4, the tensors 16-byte aligned.
MTB_API int mtb_batch_norm2d_add_relu_forward_masked_f32(int n, int c, int h, int w, const float* x, const float* residual, const float* gamma,
                                                         const float* beta, double eps, int training, double momentum, float* running_mean,
                                                         float* running_var, float* y, float* mean, float* var, unsigned char* mask,
                                                         const float* stats, int stats_rows, void* workspace, long long workspace_bytes,
                                                         void* stream) {
  MTB_REQUIRE(mask, "batch_norm2d_add_relu_forward_masked: no mask buffer");
  return bn_forward(n, c, h, w, x, gamma, beta, eps, training, momentum, running_mean, running_var, y, mean, var, 2, residual, mask, stats, stats_rows,
                    workspace, workspace_bytes, (cudaStream_t)stream);
}

// dx = gamma/sigma * (dy - dbeta/m - xhat * dgamma/m); dgamma, dbeta may be NULL (not affine).
// relu != 0: backward of the fused forward (relu flag set there); dy is masked where the
// normalised value gamma*xhat+beta is negative, which needs beta (NULL = 0).
MTB_API int mtb_batch_norm2d_backward_f32(int n, int c, int h, int w, const float* dy, const float* mean, const float* var, const float* x,
                                          const float* gamma, const float* beta, double eps, int relu, float* dx, float* dgamma,
                                          float* dbeta, void* workspace, long long workspace_bytes, void* stream) {
  return bn_backward(n, c, h, w, dy, mean, var, x, gamma, beta, eps, relu ? 1 : 0, nullptr, nullptr, dx, nullptr, dgamma, dbeta, workspace, workspace_bytes,
                     (cudaStream_t)stream);
}

// Backward of mtb_batch_norm2d_add_relu_forward_f32: the ReLU mask is recomputed from x, the statistics and
// residual with the forward's own expression; dresidual receives the masked upstream gradient (the
// gradient of the added tensor), dx the BatchNorm input gradient.
MTB_API int mtb_batch_norm2d_add_relu_backward_f32(int n, int c, int h, int w, const float* dy, const float* mean, const float* var,
                                                   const float* x, const float* residual, const float* gamma, const float* beta, double eps,
                                                   float* dx, float* dresidual, float* dgamma, float* dbeta, void* workspace,
                                                   long long workspace_bytes, void* stream) {
  return bn_backward(n, c, h, w, dy, mean, var, x, gamma, beta, eps, 2, residual, nullptr, dx, dresidual, dgamma, dbeta, workspace, workspace_bytes,
                     (cudaStream_t)stream);
}

// The same from the mask that forward wrote: the added tensor is not read (5S + S/8 instead of 8S of traffic; 64 channels on
// 512 x 32x32: partial sums and dx 163 -> 131 us).
MTB_API int mtb_batch_norm2d_add_relu_backward_masked_f32(int n, int c, int h, int w, const float* dy, const float* mean, const float* var,
                                                          const float* x, const unsigned char* mask, const float* gamma, const float* beta, double eps,
                                                          float* dx, float* dresidual, float* dgamma, float* dbeta, void* workspace,
                                                          long long workspace_bytes, void* stream) {
  MTB_REQUIRE(mask, "batch_norm2d_add_relu_backward_masked: no mask");
  return bn_backward(n, c, h, w, dy, mean, var, x, gamma, beta, eps, 2, nullptr, mask, dx, dresidual, dgamma, dbeta, workspace, workspace_bytes,
                     (cudaStream_t)stream);
}

namespace {
bool poolable(int n, int c, int h, int w, int window, const void* a, const void* b, const unsigned short* ties) {
  return ties && n > 0 && c > 0 && c % 4 == 0 && h > 1 && w > 1 && (window == 2 || window == 3) && mtb_aligned16(a) && mtb_aligned16(b) &&
         (reinterpret_cast<uintptr_t>(ties) & 7u) == 0 && (long long)n * h * w * c < (1LL << 29);
}
}  // namespace

// BatchNorm, ReLU and a max-pool of stride 2 as one operator (window 2: 2 x 2; 3: 3 x 3 with a border of one): y [n, oh, ow, c] and its tie mask; the
// normalised tensor is never stored.  c a multiple of 4, h and w at least 2, the tensors 16-byte aligned, fewer than 2^29 elements.
// stats / stats_rows as above.  Same bits as the operators one by one.
MTB_API int mtb_batch_norm2d_relu_pool_forward_f32(int n, int c, int h, int w, int window, const float* x, const float* gamma, const float* beta, double eps,
                                                   int training, double momentum, float* running_mean, float* running_var, float* y, float* mean, float* var,
                                                   unsigned short* tiemask, const float* stats, int stats_rows, void* workspace, long long workspace_bytes,
                                                   void* stream) {
  MTB_REQUIRE(poolable(n, c, h, w, window, x, y, tiemask) && mtb_aligned16(beta) && mtb_aligned16(mean) && mtb_aligned16(workspace),
              "batch_norm2d_relu_pool_forward: four channels, whole windows and 16-byte alignment are required");
  return bn_forward(n, c, h, w, x, gamma, beta, eps, training, momentum, running_mean, running_var, y, mean, var, 1, nullptr, nullptr, stats, stats_rows, workspace,
                    workspace_bytes, (cudaStream_t)stream, tiemask, window);
}

// Its backward for 2 x 2 windows: dy and tiemask have the shape of y.
MTB_API int mtb_batch_norm2d_relu_pool_backward_f32(int n, int c, int h, int w, const float* dy, const float* mean, const float* var, const float* x,
                                                    const unsigned short* tiemask, const float* gamma, const float* beta, double eps, float* dx, float* dgamma,
                                                    float* dbeta, void* workspace, long long workspace_bytes, void* stream) {
  MTB_REQUIRE(poolable(n, c, h, w, 2, x, dx, tiemask) && mtb_aligned16(dy),
              "batch_norm2d_relu_pool_backward: four channels, whole windows and 16-byte alignment are required");
  return bn_backward(n, c, h, w, dy, mean, var, x, gamma, beta, eps, 1, nullptr, nullptr, dx, nullptr, dgamma, dbeta, workspace, workspace_bytes,
                     (cudaStream_t)stream, tiemask);
}
