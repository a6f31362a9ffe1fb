// The CUDA-core (FP32 FFMA) matrix product behind the shapes the tensor-core kernels do not take: channel counts
// that fit no 32-channel block, odd matrix sizes, tiny problems.  Results are full FP32 (no TF32 rounding).
//
//   C[i, j] = sum_k A(i, k) * B(j, k)
//
// What bounds it: the FFMA pipe (128 lanes per SM, 74 TFLOP/s at 1.965 GHz), as long as operands arrive.  The
// predecessor of this kernel decoded every operand element with three integer divisions, moved single floats
// and used 4x4 outputs per thread: 6-8 TFLOP/s on a 48 -> 82 channel 3x3 convolution.  Here
//   * a thread owns TM x TN outputs (up to 8 x 16), so a 16-byte shared-memory read feeds 10 to 21 FMAs: a warp's read
//     takes four cycles of the shared-memory pipe whatever it holds, so with 4 x 12 outputs that pipe was 87 % busy
//     and bounded; two products per instruction leave issue slots for the addresses;
//   * operands move as float4 wherever four neighbours are contiguous and aligned (VEC = 4);
//   * rows are decoded once per tile and filter taps advance by addition; where a division remains it is a
//     multiplication by a precomputed reciprocal (FastDiv);
//   * two shared-memory buffers: the next block's global loads are in flight while this one is multiplied;
//   * small problems split the reduction over the CTAs of a cluster, which add their tiles through distributed
//     shared memory in rank order: one launch, no scratch, the same bits every time.
// 48 -> 82 channels, 3x3, 32 images of 37x37, 3.1 GFLOP each: forward 383 -> 110 us, data gradient 585 -> 154 us, weight
// gradient 606 -> 171 us; 4095 x 4095 x 1023: 47 TFLOP/s; one output of a single image (128 -> 32 channels on 7x7):
// 224 -> 10 us.
#pragma once
#include "common.cuh"
#include <cooperative_groups.h>
#include <type_traits>

namespace simt {
namespace cg = cooperative_groups;

constexpr int BK = 16;

// Division by a run-time constant for dividends below 2^31: Granlund & Montgomery's round-up method,
// q = (mulhi(n, m) + n) >> s with s = ceil(log2 d), m = floor(2^32 (2^s - d) / d) + 1.
struct FastDiv {
  unsigned d, m, s;
  FastDiv() = default;
  __host__ explicit FastDiv(int div) : d((unsigned)div), m(0), s(0) {
    while ((1ull << s) < d) ++s;
    m = (unsigned)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
  }
  __device__ __forceinline__ unsigned div(unsigned n) const { return (__umulhi(n, m) + n) >> s; }
  __device__ __forceinline__ unsigned divmod(unsigned n, unsigned& r) const {
    const unsigned q = div(n);
    r = n - q * d;
    return q;
  }
};

struct ConvDims {
  int N, Cin, H, W, KH, KW, SH, SW, PH, PW, Cout, OH, OW;
};

template <int VEC>
struct Vec { float v[VEC]; };
template <int VEC>
__device__ __forceinline__ Vec<VEC> load_vec(const float* p) {
  Vec<VEC> r;
  if constexpr (VEC == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int VEC>
__device__ __forceinline__ Vec<VEC> zero_vec() {
  Vec<VEC> r;
#pragma unroll
  for (int i = 0; i < VEC; ++i) r.v[i] = 0.f;
  return r;
}

// ---------------------------------------------------------------- operands whose neighbours along k are contiguous
//
// Source::Row: what is known about a row once; Source::Pos: a position along k, advanced by addition.

// Row-major [rows][K] matrix.
struct DenseK {
  const float* p;
  long long ld;
  struct Row { const float* p; };
  struct Pos { int k; };
  __device__ __forceinline__ Row row(int i, bool valid, int) const { return Row{valid ? p + i * ld : nullptr}; }
  __device__ __forceinline__ Pos pos(int k, int) const { return Pos{k}; }
  __device__ __forceinline__ void advance(Pos& q, int) const { q.k += BK; }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Row& r, const Pos& q) const { return r.p ? load_vec<VEC>(r.p + q.k) : zero_vec<VEC>(); }
};

// Patch matrix of a channels-last input: row = output pixel (n, oh, ow), k = (kh, kw, ci).
struct PatchK {
  const float* x;
  ConvDims d;
  FastDiv ow, oh, cin, kw;
  struct Row { const float* p; int ih, iw; };
  struct Pos { int kh, kw, ci; };
  __device__ __forceinline__ Row row(int i, bool valid, int) const {
    if (!valid) return Row{nullptr, 0, 0};
    unsigned c, r;
    const unsigned n = oh.divmod(ow.divmod((unsigned)i, c), r);
    return Row{x + (long long)n * d.H * d.W * d.Cin, (int)r * d.SH - d.PH, (int)c * d.SW - d.PW};
  }
  __device__ __forceinline__ Pos pos(int k, int) const {
    unsigned ci, w;
    const unsigned h = kw.divmod(cin.divmod((unsigned)k, ci), w);
    return Pos{(int)h, (int)w, (int)ci};
  }
  __device__ __forceinline__ void advance(Pos& q, int) const {
    q.ci += BK;
    while (q.ci >= d.Cin) {
      q.ci -= d.Cin;
      if (++q.kw == d.KW) { q.kw = 0; ++q.kh; }
    }
  }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Row& r, const Pos& q) const {
    const int h = r.ih + q.kh, w = r.iw + q.kw;
    if (!r.p || (unsigned)h >= (unsigned)d.H || (unsigned)w >= (unsigned)d.W) return zero_vec<VEC>();
    return load_vec<VEC>(r.p + (long long)(h * d.W + w) * d.Cin + q.ci);
  }
};

// The same with the rows in the order in which a 2 x 2 max-pool of stride 2 reads the output pixels: four neighbouring rows are a
// window (row-major), a last odd line or column of pixels belongs to none and is left out.
struct PatchPoolK : PatchK {
  FastDiv pool_w, pool_h;
  __device__ __forceinline__ Row row(int i, bool valid, int) const {
    if (!valid) return Row{nullptr, 0, 0};
    unsigned c, r;
    const unsigned n = pool_h.divmod(pool_w.divmod((unsigned)i >> 2, c), r);
    return Row{x + (long long)n * d.H * d.W * d.Cin, (int)(2 * r + (i >> 1 & 1)) * d.SH - d.PH, (int)(2 * c + (i & 1)) * d.SW - d.PW};
  }
};

// Data gradient.  The input pixels fall into SH*SW residue classes (one per blockIdx.z): pixel (i, j) of class (a, b)
// is (start + s*i, ...) and only meets the taps a + s*t, from output row c0 + i - t: no multiplication is spent on
// taps that cannot reach it.  k = (th, tw, co).
struct DgradClass {
  int taps_h, taps_w, start_h, start_w, count_h, count_w, c0_h, c0_w, a, b;
  FastDiv div_w, div_h, div_tw;  // by count_w, count_h, taps_w
};
constexpr int kMaxClasses = 16;
struct DgradK {
  const float* dy;
  ConvDims d;
  FastDiv cout;
  const DgradClass* cls;  // kernel-parameter table
  struct Row { const float* p; int oh, ow; };
  struct Pos { int th, tw, co; };
  __device__ __forceinline__ Row row(int i, bool valid, int z) const {
    if (!valid) return Row{nullptr, 0, 0};
    unsigned c, r;
    const unsigned n = cls[z].div_h.divmod(cls[z].div_w.divmod((unsigned)i, c), r);
    return Row{dy + (long long)n * d.OH * d.OW * d.Cout, (int)r + cls[z].c0_h, (int)c + cls[z].c0_w};
  }
  __device__ __forceinline__ Pos pos(int k, int z) const {
    unsigned co, w;
    const unsigned h = cls[z].div_tw.divmod(cout.divmod((unsigned)k, co), w);
    return Pos{(int)h, (int)w, (int)co};
  }
  __device__ __forceinline__ void advance(Pos& q, int z) const {
    q.co += BK;
    while (q.co >= d.Cout) {
      q.co -= d.Cout;
      if (++q.tw == cls[z].taps_w) { q.tw = 0; ++q.th; }
    }
  }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Row& r, const Pos& q) const {
    const int h = r.oh - q.th, w = r.ow - q.tw;
    if (!r.p || (unsigned)h >= (unsigned)d.OH || (unsigned)w >= (unsigned)d.OW) return zero_vec<VEC>();
    return load_vec<VEC>(r.p + (long long)(h * d.OW + w) * d.Cout + q.co);
  }
};

// ---------------------------------------------------------------- operands whose neighbours along the row are contiguous
//
// Source::Col: what is known about a row index once; load(col, k) decodes k itself.

// [K][rows] matrix, row pitch ld.
struct DenseR {
  const float* p;
  long long ld;
  struct Col { int i; };
  __device__ __forceinline__ Col col(int i, int) const { return Col{i}; }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Col& c, int k, int) const { return load_vec<VEC>(p + k * ld + c.i); }
};

// Filter W[co][kh][kw][ci] as B of the data gradient: row = ci, k = (th, tw, co) of a residue class.
struct DgradR {
  const float* w;
  ConvDims d;
  FastDiv cout;
  const DgradClass* cls;
  struct Col { int i; };
  __device__ __forceinline__ Col col(int i, int) const { return Col{i}; }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Col& c, int k, int z) const {
    unsigned co, tw;
    const unsigned th = cls[z].div_tw.divmod(cout.divmod((unsigned)k, co), tw);
    const int tap = (cls[z].a + d.SH * (int)th) * d.KW + cls[z].b + d.SW * (int)tw;
    return load_vec<VEC>(w + ((long long)co * (d.KH * d.KW) + tap) * d.Cin + c.i);
  }
};

// Patch matrix as B of the weight gradient: row = (kh, kw, ci), k = output pixel.
struct PatchR {
  const float* x;
  ConvDims d;
  FastDiv ow, oh, cin, kw;
  struct Col { int kh, kw, ci; };
  __device__ __forceinline__ Col col(int i, int) const {
    unsigned ci, w;
    const unsigned h = kw.divmod(cin.divmod((unsigned)i, ci), w);
    return Col{(int)h - d.PH, (int)w - d.PW, (int)ci};
  }
  template <int VEC>
  __device__ __forceinline__ Vec<VEC> load(const Col& c, int k, int) const {
    unsigned ow_, oh_;
    const unsigned n = oh.divmod(ow.divmod((unsigned)k, ow_), oh_);
    const int h = (int)oh_ * d.SH + c.kh, w = (int)ow_ * d.SW + c.kw;
    if ((unsigned)h >= (unsigned)d.H || (unsigned)w >= (unsigned)d.W) return zero_vec<VEC>();
    return load_vec<VEC>(x + (((long long)n * d.H + h) * d.W + w) * d.Cin + c.ci);
  }
};

// ---------------------------------------------------------------- staging: global -> registers -> shared [BK][ROWS + 4]

template <class Source, int ROWS, int THREADS, int VEC>
struct StageK {
  static constexpr int kPerRow = BK / VEC, kTotal = ROWS * kPerRow, kCount = (kTotal + THREADS - 1) / THREADS;
  static_assert(THREADS % kPerRow == 0, "a thread stays on one k offset");
  typename Source::Row rows[kCount];
  typename Source::Pos pos;
  Vec<VEC> regs[kCount];
  int k, k_end, z;
  __device__ __forceinline__ void init(const Source& s, int row0, int nrows, int k0, int k1, int z_, int tid) {
    z = z_;
    k = k0 + (tid % kPerRow) * VEC;
    k_end = k1;
    pos = s.pos(k, z);
#pragma unroll
    for (int i = 0; i < kCount; ++i) {
      const int r = row0 + (tid + i * THREADS) / kPerRow;
      rows[i] = s.row(r, r < nrows && tid + i * THREADS < kTotal, z);
    }
  }
  __device__ __forceinline__ void load(const Source& s) {
#pragma unroll
    for (int i = 0; i < kCount; ++i) regs[i] = k < k_end ? s.template load<VEC>(rows[i], pos) : zero_vec<VEC>();
    k += BK;
    s.advance(pos, z);
  }
  __device__ __forceinline__ void store(float (*sm)[ROWS + 4], int tid) const {
#pragma unroll
    for (int i = 0; i < kCount; ++i) {
      const int v = tid + i * THREADS;
      if (kTotal % THREADS == 0 || v < kTotal) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) sm[(v % kPerRow) * VEC + j][v / kPerRow] = regs[i].v[j];
      }
    }
  }
};

template <class Source, int ROWS, int THREADS, int VEC>
struct StageR {
  static constexpr int kPerK = ROWS / VEC, kTotal = BK * kPerK, kCount = (kTotal + THREADS - 1) / THREADS;
  typename Source::Col cols[kCount];
  Vec<VEC> regs[kCount];
  bool valid[kCount];
  int k, k_end, z;
  __device__ __forceinline__ void init(const Source& s, int row0, int nrows, int k0, int k1, int z_, int tid) {
    z = z_;
    k = k0;
    k_end = k1;
#pragma unroll
    for (int i = 0; i < kCount; ++i) {
      const int v = tid + i * THREADS, r = row0 + (v % kPerK) * VEC;
      valid[i] = r < nrows && v < kTotal;
      cols[i] = s.col(valid[i] ? r : 0, z);
    }
  }
  __device__ __forceinline__ void load(const Source& s) {
#pragma unroll
    for (int i = 0; i < kCount; ++i) {
      const int kk = k + ((int)threadIdx.x + i * THREADS) / kPerK;
      regs[i] = valid[i] && kk < k_end ? s.template load<VEC>(cols[i], kk, z) : zero_vec<VEC>();
    }
    k += BK;
  }
  __device__ __forceinline__ void store(float (*sm)[ROWS + 4], int tid) const {
#pragma unroll
    for (int i = 0; i < kCount; ++i) {
      const int v = tid + i * THREADS;
      if (kTotal % THREADS == 0 || v < kTotal) {
        float* p = &sm[v / kPerK][(v % kPerK) * VEC];
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(regs[i].v[0], regs[i].v[1], regs[i].v[2], regs[i].v[3]);
        else *p = regs[i].v[0];
      }
    }
  }
};

template <class Source> struct IsK { static constexpr bool value = false; };
template <> struct IsK<DenseK> { static constexpr bool value = true; };
template <> struct IsK<PatchK> { static constexpr bool value = true; };
template <> struct IsK<PatchPoolK> { static constexpr bool value = true; };
template <> struct IsK<DgradK> { static constexpr bool value = true; };
template <class Source, int ROWS, int THREADS, int VEC>
using Stage = std::conditional_t<IsK<Source>::value, StageK<Source, ROWS, THREADS, VEC>, StageR<Source, ROWS, THREADS, VEC>>;

// ---------------------------------------------------------------- results

struct Out {
  float* out;
  long long ld;
  const float* bias;
  MtbBnEval bn;              // mean != NULL: BatchNorm with running statistics after the bias (cluster kernels only)
  const float* residual;     // laid out like out: added before the ReLU (cluster kernels only)
  int relu;
  long long split_plane;     // > 0: every slice of the reduction writes its own plane of partials
  const DgradClass* cls;     // data gradient: row -> pixel of the residue class
  int H, W, SH, SW;
};

// What few launches need beside the product, in instantiations of their own and as their last parameter: as members of Out, tested
// in every kernel, the two took small convolutions and products 2 to 10 % (128 -> 32 channels 3x3 on one 7x7 image 8.75 -> 9.6 us).
enum { EXTRA_NONE, EXTRA_GUARD, EXTRA_PRE };
struct Extra {
  const int* guard;  // convolutions only; not NULL: nothing is done unless one of these words is set
  int guards;
  float* pre;        // dense products of two operands along k only; not NULL: laid out like out, takes the value before the ReLU
};
struct NoExtra {};
struct PoolExtra {  // with PatchPoolK
  unsigned short* mask;  // per result, bit 2 * line + column of every pixel of the window that equals the maximum
};
template <int EXTRA>
using ExtraOf = std::conditional_t<EXTRA == EXTRA_NONE, NoExtra, Extra>;

__device__ __forceinline__ float* out_row(const Out& o, int i, int z) {
  long long r = i;
  if (o.cls) {
    unsigned c, h;
    const unsigned n = o.cls[z].div_h.divmod(o.cls[z].div_w.divmod((unsigned)i, c), h);
    r = ((long long)n * o.H + o.cls[z].start_h + o.SH * (int)h) * o.W + o.cls[z].start_w + o.SW * (int)c;
  }
  return o.out + r * o.ld;
}

__device__ __forceinline__ float bn_eval_value(const MtbBnEval& bn, int c, float v) {
  const float rstd = 1.0f / sqrtf(bn.var[c] + bn.eps);
  const float scale = bn.gamma ? bn.gamma[c] * rstd : rstd, beta = bn.beta ? bn.beta[c] : 0.f;
  return (v - bn.mean[c]) * scale + beta;
}

// TAIL: with BatchNorm and the residual of Out (the cluster kernels, whose store is one loop)
template <bool TAIL, int EXTRA>
__device__ __forceinline__ void store4(const Out& o, const ExtraOf<EXTRA>& extra, float* row, int j, int N, bool vec, float4 v) {
  float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (o.bias && j + q < N) t[q] += o.bias[j + q];
    if constexpr (TAIL) {
      if (o.bn.mean && j + q < N) t[q] = bn_eval_value(o.bn, j + q, t[q]);
      if (o.residual && j + q < N) t[q] += o.residual[row - o.out + j + q];
    }
    if constexpr (EXTRA == EXTRA_PRE) {
      if (j + q < N) extra.pre[row - o.out + j + q] = t[q];
    }
    if (o.relu) t[q] = fmaxf(t[q], 0.f);
  }
  if (vec && j + 3 < N) {
    *reinterpret_cast<float4*>(row + j) = make_float4(t[0], t[1], t[2], t[3]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (j + q < N) row[j + q] = t[q];
  }
}

// ---------------------------------------------------------------- the kernel

template <int BM_, int BN_, int TM_, int TN_, int MIN_CTAS>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, THREADS = (BM_ / TM_) * (BN_ / TN_), kMinCtas = MIN_CTAS;
};

// Two FMAs in one instruction (the same rounding as two fmaf).  One scalar FFMA per lane and cycle is also all a
// scheduler can issue, so every address or shared-memory instruction of the loop would cost an FMA; packed, half of
// the issue slots are free for them.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

struct ClassTable { DgradClass c[kMaxClasses]; };
struct NoTable {};
template <class SA>
using TableOf = std::conditional_t<std::is_same_v<SA, DgradK>, ClassTable, NoTable>;

// blockIdx.z = class * slices + slice.  CLUSTER: the slices of a tile form a cluster and add up at the end;
// otherwise slices > 1 only with planes of partials (Out::split_plane).
template <class SA, int EXTRA>
using LastParam = std::conditional_t<std::is_same_v<SA, PatchPoolK>, PoolExtra, ExtraOf<EXTRA>>;

template <class T, class SA, int VA, class SB, int VB, bool CLUSTER, int EXTRA>
__global__ void __launch_bounds__(T::THREADS, T::kMinCtas) gemm_kernel(SA sa, SB sb, Out o, const __grid_constant__ TableOf<SA> table, int M, int N, int K,
                                                          int slices, int k_per_slice, const LastParam<SA, EXTRA> extra) {
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, THREADS = T::THREADS;
  constexpr int GM = TM / 4, GN = TN / 4;  // a thread's rows and columns come in groups of four, spread over the tile
  __shared__ float As[2][BK][BM + 4];
  __shared__ float Bs[2][BK][BN + 4];
  mtb_launch_dependents();
  mtb_wait_prior();
  if constexpr (EXTRA == EXTRA_GUARD) {
    int any = 0;
    for (int i = 0; i < extra.guards; ++i) any |= extra.guard[i];
    if (!any) return;
  }
  const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int z = blockIdx.z / slices, slice = blockIdx.z - z * slices;
  if constexpr (std::is_same_v<SA, DgradK>) {  // every residue class has its own rows and reduction
    sa.cls = sb.cls = o.cls = table.c;
    M = table.c[z].count_h * table.c[z].count_w * sa.d.N;
    K = table.c[z].taps_h * table.c[z].taps_w * sa.d.Cout;
    if (m0 >= M) return;  // the whole cluster: its CTAs share the tile and the class
    k_per_slice = ((K + slices - 1) / slices + BK - 1) / BK * BK;
  }
  const int k0 = slice * k_per_slice, k1 = k0 + k_per_slice < K ? k0 + k_per_slice : K;
  Stage<SA, BM, THREADS, VA> a;
  Stage<SB, BN, THREADS, VB> b;
  a.init(sa, m0, M, k0, k1, z, tid);
  b.init(sb, n0, N, k0, k1, z, tid);
  unsigned long long acc2[TM][TN / 2];  // column pairs
#pragma unroll
  for (int p = 0; p < TM; ++p)
#pragma unroll
    for (int q = 0; q < TN / 2; ++q) acc2[p][q] = 0ull;

  a.load(sa);
  b.load(sb);
  a.store(As[0], tid);
  b.store(Bs[0], tid);
  __syncthreads();
  int buf = 0;
  for (int kb = k0; kb < k1; kb += BK) {
    const bool more = kb + BK < k1;
    if (more) { a.load(sa); b.load(sb); }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float fa[TM];
      unsigned long long fb[TN / 2];
#pragma unroll
      for (int g = 0; g < GM; ++g) {
        const float4 t = *reinterpret_cast<const float4*>(&As[buf][kk][g * (BM / GM) + ty * 4]);
        fa[4 * g] = t.x; fa[4 * g + 1] = t.y; fa[4 * g + 2] = t.z; fa[4 * g + 3] = t.w;
      }
#pragma unroll
      for (int g = 0; g < GN; ++g) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][g * (BN / GN) + tx * 4]);
        fb[2 * g] = t.x; fb[2 * g + 1] = t.y;
      }
#pragma unroll
      for (int p = 0; p < TM; ++p) {
        const unsigned long long dup = pack2(fa[p], fa[p]);
#pragma unroll
        for (int q = 0; q < TN / 2; ++q) fma2(acc2[p][q], dup, fb[q]);
      }
    }
    if (more) {
      a.store(As[buf ^ 1], tid);
      b.store(Bs[buf ^ 1], tid);
    }
    __syncthreads();
    buf ^= 1;
  }

  auto four = [&](int p, int g) {
    const float2 u = unpack2(acc2[p][2 * g]), v = unpack2(acc2[p][2 * g + 1]);
    return make_float4(u.x, u.y, v.x, v.y);
  };
  const bool vec = (o.ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(o.out) & 15u) == 0) && (o.split_plane % 4 == 0);
  if constexpr (CLUSTER) {
    // every CTA leaves its tile in shared memory; CTA r then finishes the rows r, r + size, ... of the tile
    __shared__ alignas(16) float tile[BM][BN];
    cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
    for (int p = 0; p < TM; ++p)
#pragma unroll
      for (int g = 0; g < GN; ++g)
        *reinterpret_cast<float4*>(&tile[(p / 4) * (BM / GM) + ty * 4 + (p % 4)][g * (BN / GN) + tx * 4]) = four(p, g);
    cluster.sync();
    const int size = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    constexpr int kVecs = BN / 4;
    if constexpr (std::is_same_v<SA, PatchPoolK>) {  // CTA r finishes the windows r, r + size, ...: bias, BatchNorm and ReLU of four rows, their maximum
      for (int e = tid; e < (BM / 4 / size) * kVecs; e += THREADS) {
        const int u = (e / kVecs) * size + rank, c = (e % kVecs) * 4;
        if (m0 + 4 * u >= M) continue;
        float best[4];
        unsigned ties[4] = {0u, 0u, 0u, 0u};
        for (int w = 0; w < 4; ++w) {
          float4 s = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&tile[4 * u + w][c], 0));
          for (int q = 1; q < size; ++q) {
            const float4 t = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&tile[4 * u + w][c], q));
            s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
          }
          const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (n0 + c + q >= N) continue;
            float t = v[q];
            if (o.bias) t += o.bias[n0 + c + q];
            t = fmaxf(bn_eval_value(o.bn, n0 + c + q, t), 0.f);
            if (w == 0 || t > best[q]) { best[q] = t; ties[q] = 1u << w; }
            else if (t == best[q]) ties[q] |= 1u << w;
          }
        }
        const long long at = (long long)(m0 / 4 + u) * o.ld + n0 + c;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (n0 + c + q < N) { o.out[at + q] = best[q]; extra.mask[at + q] = (unsigned short)ties[q]; }
      }
    } else {
      for (int e = tid; e < (BM / size) * kVecs; e += THREADS) {
        const int r = (e / kVecs) * size + rank, c = (e % kVecs) * 4;
        float4 s = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&tile[r][c], 0));
        for (int q = 1; q < size; ++q) {  // rank order: the same sum every time
          const float4 t = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&tile[r][c], q));
          s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
        }
        if (m0 + r < M) store4<std::is_same_v<SA, PatchK>, EXTRA>(o, extra, out_row(o, m0 + r, z), n0 + c, N, vec, s);
      }
    }
    cluster.sync();  // nobody leaves while its tile is being read
  } else {
#pragma unroll
    for (int p = 0; p < TM; ++p) {
      const int i = m0 + (p / 4) * (BM / GM) + ty * 4 + (p % 4);
      if (i >= M) continue;
      float* row = out_row(o, i, z) + slice * o.split_plane;
#pragma unroll
      for (int g = 0; g < GN; ++g)
        store4<false, EXTRA>(o, extra, row, n0 + g * (BN / GN) + tx * 4, N, vec, four(p, g));
    }
  }
}

// ---------------------------------------------------------------- host: which tile, how many slices
//
// A block of BK = 16 of one CTA costs its multiplications plus about 500 cycles of load latency when nothing else on
// the SM hides it; with other CTAs beside it the FFMA pipe bounds, at `eff` of its rate.  A launch is priced as CTAs per
// SM x blocks x the slower of the two (plus the cluster's exchange, or the pass over the planes) and the cheapest is taken.
struct Choice { int tile, slices; double cycles; };
enum { XL = 0, L = 1, MD = 2, SM = 3, XS = 4, kTiles = 5 };
struct TileInfo { int bm, bn, occ; double eff; bool cluster; };
inline const TileInfo& tile_info(int t) {
  static const TileInfo info[kTiles] = {{128, 128, 2, 0.68, false}, {128, 96, 2, 0.62, false}, {128, 64, 3, 0.58, false}, {64, 64, 4, 0.50, true},
                                        {64, 32, 6, 0.42, true}};
  return info[t];
}

// rows x cols outputs with a reduction of k, `classes` such problems in one launch; max_planes > 1: the reduction may be
// split into that many planes of partials that a second launch adds (long reductions with few outputs).
inline Choice choose(long long rows, long long cols, long long k, int classes, int max_planes) {
  static const int kSlices[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512};
  const double sms = mtb_sm_count();
  Choice best{SM, 1, 1e300};
  for (int t = 0; t < kTiles; ++t) {
    const TileInfo& info = tile_info(t);
    const double tiles = (double)((rows + info.bm - 1) / info.bm) * (double)((cols + info.bn - 1) / info.bn) * classes;
    const double mul = info.bm * info.bn * BK / 128.0;
    const int most = max_planes > 1 ? max_planes : (info.cluster ? 8 : 1);
    for (int s : kSlices) {
      if (s > most || (s > 1 && k / s < 2 * BK)) break;
      if (max_planes <= 1 && (s & (s - 1))) continue;  // a cluster's CTAs share the rows of a tile evenly
      const double ctas = tiles * s, blocks = (double)((k + s - 1) / s + BK - 1) / BK;
      const double per_sm = ctas / sms;
      // all CTAs resident at once: the fullest SM decides; more than that: they follow one another, half a tile of tail
      const double queue = per_sm <= info.occ ? (double)(long long)(per_sm + 0.999999) : per_sm + 0.5;
      const double beside = queue < info.occ ? queue : info.occ;
      const double alone = (500 + mul) / beside, piped = mul / info.eff;
      double cycles = queue * blocks * (alone > piped ? alone : piped) + 2000;
      if (s > 1) cycles += max_planes > 1 ? 4000 + s * (double)rows * cols * 8 / 2500 : 2500;
      if (cycles < best.cycles) best = Choice{t, s, cycles};
    }
  }
  return best;
}

using TileXL = Tile<128, 128, 8, 16, 2>;
using TileL = Tile<128, 96, 8, 12, 2>;
using TileM = Tile<128, 64, 8, 8, 3>;
using TileS = Tile<64, 64, 8, 4, 4>;
using TileXS = Tile<64, 32, 4, 4, 6>;

template <int EXTRA, class T, class SA, int VA, class SB, int VB, bool CLUSTER>
int launch_tile(const SA& sa, const SB& sb, const Out& o, const TableOf<SA>& table, int classes, int M, int N, int K, int slices, cudaStream_t st,
                const char* name, const std::conditional_t<std::is_same_v<SA, PatchPoolK>, PoolExtra, Extra>& extra) {
  int per = (K + slices - 1) / slices;
  per = (per + BK - 1) / BK * BK;
  if (per < BK) per = BK;
  LastParam<SA, EXTRA> with{};
  if constexpr (EXTRA != EXTRA_NONE || std::is_same_v<SA, PatchPoolK>) with = extra;
  dim3 grid(mtb_div_up(M, T::BM), mtb_div_up(N, T::BN), classes * slices);
  MTB_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "%s: grid too large", name);
  if constexpr (CLUSTER) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(T::THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)slices;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    MTB_CUDA(cudaLaunchKernelEx(&cfg, gemm_kernel<T, SA, VA, SB, VB, true, EXTRA>, sa, sb, o, table, M, N, K, slices, per, with));
  } else {
    MTB_LAUNCH(gemm_kernel<T, SA, VA, SB, VB, false, EXTRA>, grid, T::THREADS, 0, st, sa, sb, o, table, M, N, K, slices, per, with);
  }
  MTB_LAUNCH_CHECK(name);
  return MTB_OK;
}

template <int EXTRA, class SA, int VA, class SB, int VB>
int launch_extra(const Choice& c, const SA& sa, const SB& sb, const Out& o, const TableOf<SA>& table, int classes, int M, int N, int K, cudaStream_t st,
                 const char* name, const Extra& extra) {
  const bool cluster = (c.slices > 1 && o.split_plane == 0) || o.bn.mean;
  switch (c.tile) {
    case XL: return launch_tile<EXTRA, TileXL, SA, VA, SB, VB, false>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
    case L: return launch_tile<EXTRA, TileL, SA, VA, SB, VB, false>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
    case MD: return launch_tile<EXTRA, TileM, SA, VA, SB, VB, false>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
    case SM:
      if (cluster) return launch_tile<EXTRA, TileS, SA, VA, SB, VB, true>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
      return launch_tile<EXTRA, TileS, SA, VA, SB, VB, false>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
    default:
      if (cluster) return launch_tile<EXTRA, TileXS, SA, VA, SB, VB, true>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
      return launch_tile<EXTRA, TileXS, SA, VA, SB, VB, false>(sa, sb, o, table, classes, M, N, K, c.slices, st, name, extra);
  }
}

template <class SA, int VA, class SB, int VB>
int launch(const Choice& c, const SA& sa, const SB& sb, const Out& o, const TableOf<SA>& table, int classes, int M, int N, int K, cudaStream_t st,
           const char* name, const Extra& extra = {}) {
  constexpr bool dense = (std::is_same_v<SA, DenseK> || std::is_same_v<SA, DenseR>) && (std::is_same_v<SB, DenseK> || std::is_same_v<SB, DenseR>);
  if constexpr (!dense) {
    if (extra.guard) return launch_extra<EXTRA_GUARD, SA, VA, SB, VB>(c, sa, sb, o, table, classes, M, N, K, st, name, extra);
  } else if constexpr (std::is_same_v<SA, DenseK> && std::is_same_v<SB, DenseK>) {
    if (extra.pre) return launch_extra<EXTRA_PRE, SA, VA, SB, VB>(c, sa, sb, o, table, classes, M, N, K, st, name, extra);
  }
  return launch_extra<EXTRA_NONE, SA, VA, SB, VB>(c, sa, sb, o, table, classes, M, N, K, st, name, extra);
}

}  // namespace simt
