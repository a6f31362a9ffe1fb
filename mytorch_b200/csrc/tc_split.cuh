// Convolutions over channel counts that fit no 32-channel block, in FP32 accuracy on the tensor cores: every operand is the sum
// of two TF32 numbers, x = hi + lo (hi: x rounded to TF32, lo: what is left, rounded), and
//   x * w = lo * hi' + hi * lo' + hi * hi'    (the term left out is 2^-22 of the product and has no preferred sign).
//
// A pass over the operands writes them as rows of blocks [32 channels hi][32 channels lo], channels padded with zeros, in
// scratch; the products then are those of tc_gemm_kernel and tc_wgrad_kernel (im2col-mode loads, one persistent CTA per SM)
// with three products of K = 32 per reduction block.
//
// Accuracy.  The tensor core truncates its sum at every step, a bias that grows with the number of steps, so a chain of steps
// is one reduction block (the two small products first, then four steps of hi * hi'); the epilogue warps add the chains up in
// registers with FP32 rounding while the next ones run (four accumulators in tensor memory).
//
// Infinities, NaN and magnitudes above 3e38 do not survive the split (inf - inf), and where a whole operand is tiny lo falls
// under the smallest normal number, which the tensor core takes for zero (values of 1e-37: error 3.3e-5 instead of 2.6e-7 on the
// CUDA cores).  The packing pass reports both, the products then do nothing, and the CUDA-core kernel, which is
// enqueued behind and otherwise returns at once, computes the result.
//
// What bounds it: copies into shared memory (a block of 128 x 96 outputs takes 56 KB, 0.63 us at the measured 89 GB/s per SM,
// for 576 cycles of MMAs).
#pragma once
#include <cmath>

namespace {
using namespace tc;

// ------------------------------------------------------------------------------ packing

// dst[row][block]{hi[32], lo[32]} of the matrix element(row, c) = src[row / inner * s_outer + row % inner * s_inner + c * s_c]
struct SplitSide {
  const float* src;
  float* dst;
  long long rows, s_outer, s_inner, s_c;
  int inner, C, blocks, vec;  // vec: four channels in one load
};

constexpr int kSplitPackBlocks = 1024;  // most CTAs of the packing pass, each with its word in `bad`

// A word: what a CTA has seen of the first operand, and three bits higher of the second.  Below 2^-114 lo may be lost, an error
// of 2^-126 at most, which is nothing beside an operand with any value from 2^-96 on.
enum { kSplitRefused = 1, kSplitTiny = 2, kSplitOrdinary = 4 };
__device__ __forceinline__ bool split_refused(int word) {
  return (word & (kSplitRefused | kSplitRefused << 3)) || (word & (kSplitTiny | kSplitOrdinary)) == kSplitTiny ||
         (word >> 3 & (kSplitTiny | kSplitOrdinary)) == kSplitTiny;
}
// The words of all threads of the CTA in *all (shared, zero before; a barrier must follow).
__device__ __forceinline__ void split_gather(int* all, int word) {
  word = __reduce_or_sync(0xffffffffu, word);
  if ((threadIdx.x & 31) == 0 && word) atomicOr(all, word);
}

__global__ void __launch_bounds__(256) split_pack_kernel(const SplitSide a, const SplitSide b, int* __restrict__ bad) {
  __shared__ int all;
  if (threadIdx.x == 0) all = 0;
  __syncthreads();
  mtb_launch_dependents();
  mtb_wait_prior();
  int found = 0;
  const unsigned items_a = (unsigned)(a.rows * a.blocks * 8), items = items_a + (unsigned)(b.rows * b.blocks * 8);  // an item is four channels
  for (unsigned i = blockIdx.x * 256u + threadIdx.x; i < items; i += gridDim.x * 256u) {
    const bool first = i < items_a;
    const SplitSide& s = first ? a : b;
    const unsigned k = first ? i : i - items_a;
    const unsigned groups = (unsigned)s.blocks * 8u, row = k / groups;
    const int g = (int)(k - row * groups), c = g * 4;
    const unsigned outer = s.inner == 1 ? row : row / (unsigned)s.inner;
    const float* src = s.src + outer * s.s_outer + (long long)(row - outer * (unsigned)s.inner) * s.s_inner;
    float v[4];
    if (s.vec && c + 3 < s.C) {
      const float4 t = *reinterpret_cast<const float4*>(src + c);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = c + j < s.C ? src[(c + j) * s.s_c] : 0.f;
    }
    float hi[4], lo[4];
    unsigned most = 0, least = ~0u;  // magnitudes as integers, which order like the numbers; least: of those that are not zero, less one
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned u = __float_as_uint(v[j]) & 0x7fffffffu;
      most = most > u ? most : u;
      least = least < u - 1 ? least : u - 1;
      uint32_t r;
      asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v[j]));
      hi[j] = __uint_as_float(r);
      lo[j] = v[j] - hi[j];
    }
    const int seen = (__uint_as_float(most) <= 3.0e38f ? 0 : kSplitRefused) | (least < (13u << 23) - 1 ? kSplitTiny : 0) | (most >= (31u << 23) ? kSplitOrdinary : 0);
    found |= first ? seen : seen << 3;
    float* d = s.dst + ((long long)row * s.blocks + g / 8) * 64 + (g % 8) * 4;
    st4(d, make_float4(hi[0], hi[1], hi[2], hi[3]));
    st4(d + 32, make_float4(lo[0], lo[1], lo[2], lo[3]));
  }
  split_gather(&all, found);
  __syncthreads();
  if (threadIdx.x == 0) bad[blockIdx.x] = all;
}

// ------------------------------------------------------------------------------ products

struct SplitGemmParams {
  int M, N, num_kb, m_tiles, n_tiles;
  float* out;
  long long ldo;
  const float* bias;
  int relu;
  int OW, OH, SW, SH, PW, PH, KW, KH, cblocks;  // geometry of the im2col'ed tensor, in blocks of 32 channels
  int b_tap[64];                                // first column of a tap in B
  int o_strided, o_Hc, o_Wc, o_H, o_W, o_h0, o_w0, o_sh, o_sw;  // see GemmParams
  const int* bad;
  int n_bad;
  int* any_bad;  // one word for the kernel that follows
};

constexpr int kSplitAcc = 4;  // accumulators in tensor memory

template <int BN>
struct SplitCfg {
  static constexpr uint32_t kA = 2 * 128 * 128, kB = 2 * BN * 128;  // hi and lo of 128 (BN) rows x 32
  static constexpr uint32_t kStageBytes = kA + kB;
  static constexpr int kStages = BN <= 64 ? 4 : 3;
  static constexpr uint32_t kTurn = 8 * 32 * 17 * 4;  // the epilogue warps turn their rows here
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + kTurn + 1024;
  static constexpr uint32_t kTmemCols = BN == 32 ? 128 : BN == 64 ? 256 : 512;
  static constexpr int kCols = BN / 2;  // columns of an epilogue warp
  static_assert(kSmemBytes <= 227 * 1024 && kStages <= 4 && kSplitAcc * BN <= (int)kTmemCols && kTmemCols <= 512);
};

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, float* r) {
  uint32_t v[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
        "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) r[j] = __uint_as_float(v[j]);
}

// What both product kernels share: barriers, tensor memory, the issuing warp, and the sum of a unit's chains.
struct SplitShared {
  uint64_t full[4], empty[4], tfull[kSplitAcc], tempty[kSplitAcc];
  uint32_t tmem_slot;
  int abort_flag;
  int words;  // of the packing pass
};

template <int BN>
__device__ __forceinline__ void split_setup(SplitShared& s, int warp) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < SplitCfg<BN>::kStages; ++i) {
      mbar_init(smem_u32(&s.full[i]), 1);
      mbar_init(smem_u32(&s.empty[i]), 1);
    }
    for (int b = 0; b < kSplitAcc; ++b) {
      mbar_init(smem_u32(&s.tfull[b]), 1);
      mbar_init(smem_u32(&s.tempty[b]), kEpilogueWarps);
    }
    s.abort_flag = 0;
    s.words = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&s.tmem_slot), SplitCfg<BN>::kTmemCols);
    tmem_relinquish();
  }
}

// `chains` chains of 12 MMAs, one per stage, into the accumulators in turn.  MN: both operands MN-major (weight gradient).
template <int BN, bool MN>
__device__ __forceinline__ void split_issue(SplitShared& s, uint32_t smem_base, uint32_t tmem_base, int chains, volatile int* abort_ptr) {
  using C = SplitCfg<BN>;
  constexpr uint32_t idesc = idesc_tf32(128, BN, MN, MN);
  constexpr uint32_t hi_word = MN ? desc_hi_mnmajor() : desc_hi_kmajor();
  constexpr uint32_t step = MN ? (1024u >> 4) : (32u >> 4);                // per 8 of K
  constexpr uint32_t a_lo_off = (MN ? 4096u : C::kA / 2) >> 4, b_lo_off = (MN ? 4096u : C::kB / 2) >> 4;
  // MN-major: blocks of 32 rows lie [hi 4 KB][lo 4 KB] one after the other
  const uint32_t a0 = MN ? desc_lo_mnmajor(smem_base, 8192u) : desc_lo_kmajor(smem_base);
  const uint32_t b0 = MN ? desc_lo_mnmajor(smem_base + C::kA, 8192u) : desc_lo_kmajor(smem_base + C::kA);
  int stage = 0;
  uint32_t phase = 0;
  for (int g = 0; g < chains; ++g) {
    const int buf = g % kSplitAcc;
    const uint32_t use = (uint32_t)(g / kSplitAcc);
    bool ok = mbar_wait(smem_u32(&s.tempty[buf]), (use & 1u) ^ 1u, abort_ptr, 42) && mbar_wait(smem_u32(&s.full[stage]), phase, abort_ptr, 43);
    if (!__all_sync(0xffffffffu, ok)) break;
    tc_fence_after();
    const uint32_t d = tmem_base + buf * BN;
    const uint32_t a = a0 + stage * (C::kStageBytes >> 4), b = b0 + stage * (C::kStageBytes >> 4);
    if (elect_one()) {
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_tf32_words(d, a + a_lo_off + k * step, hi_word, b + k * step, hi_word, idesc, k > 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_tf32_words(d, a + k * step, hi_word, b + b_lo_off + k * step, hi_word, idesc, 1u);
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_tf32_words(d, a + k * step, hi_word, b + k * step, hi_word, idesc, 1u);
      mma_commit(smem_u32(&s.empty[stage]));
      mma_commit(smem_u32(&s.tfull[buf]));
    }
    __syncwarp();
    if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
  }
}

// The sum of `chains` chains (from number g on) of this warp's 32 rows and columns.
template <int BN>
__device__ __forceinline__ bool split_sum(SplitShared& s, uint32_t tmem_base, int quarter, int c_first, int lane, int& g, int chains, volatile int* abort_ptr,
                                          float (&acc)[SplitCfg<BN>::kCols]) {
  constexpr int COLS = SplitCfg<BN>::kCols;
#pragma unroll
  for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
  for (int c = 0; c < chains; ++c, ++g) {
    const int buf = g % kSplitAcc;
    bool ok = lane != 0 || mbar_wait(smem_u32(&s.tfull[buf]), (uint32_t)(g / kSplitAcc) & 1u, abort_ptr, 44);
    if (!__all_sync(0xffffffffu, ok)) return false;
    tc_fence_after();
    float r[COLS];
#pragma unroll
    for (int j = 0; j < COLS; j += 16) tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c_first + j), r + j);
    tmem_ld_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&s.tempty[buf]));
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] += r[j];
  }
  return true;
}

__device__ __forceinline__ void split_teardown(SplitShared& s, uint32_t tmem_base, int warp, uint32_t cols) {
  mtb_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (s.abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies in flight land before shared memory is released
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, cols);
  }
}

template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
split_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const SplitGemmParams p) {
  using C = SplitCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ SplitShared s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  split_setup<BN>(s, warp);
  __syncthreads();
  mtb_wait_prior();
  int word = 0;
  for (int i = threadIdx.x; i < p.n_bad; i += kGemmThreads) word |= p.bad[i];
  split_gather(&s.words, word);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const bool bad = split_refused(s.words);
  if (blockIdx.x == 0 && threadIdx.x == 0) *p.any_bad = bad;
  const uint32_t tmem_base = s.tmem_slot;
  const int tiles = bad ? 0 : p.m_tiles * p.n_tiles;
  volatile int* abort_ptr = &s.abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int m0 = (tile / p.n_tiles) * 128, n0 = (tile % p.n_tiles) * BN;
        const int ow = m0 % p.OW, t = m0 / p.OW;
        const int pix_w = ow * p.SW - p.PW, pix_h = (t % p.OH) * p.SH - p.PH, pix_n = t / p.OH;
        int cb = 0, kw = 0, kh = 0;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&s.empty[stage]), phase ^ 1u, abort_ptr, 41)) { ok = false; break; }
          const uint32_t full = smem_u32(&s.full[stage]), a_dst = smem_base + stage * C::kStageBytes, b_dst = a_dst + C::kA;
          mbar_expect_tx(full, C::kStageBytes);
          tma_load_im2col_4d(a_dst, &mapA, full, cb * 64, pix_w, pix_h, pix_n, (uint16_t)kw, (uint16_t)kh);
          tma_load_im2col_4d(a_dst + C::kA / 2, &mapA, full, cb * 64 + 32, pix_w, pix_h, pix_n, (uint16_t)kw, (uint16_t)kh);
          const int bx = p.b_tap[kh * p.KW + kw] + cb * 64;
          tma_load_2d(b_dst, &mapB, full, bx, n0);
          tma_load_2d(b_dst + C::kB / 2, &mapB, full, bx + 32, n0);
          if (++cb == p.cblocks) {
            cb = 0;
            if (++kw == p.KW) { kw = 0; ++kh; }
          }
          if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    const int mine = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    split_issue<BN, false>(s, smem_base, tmem_base, mine * p.num_kb, abort_ptr);
  } else {
    const int quarter = warp & 3, c_first = warp < 6 ? 0 : C::kCols;
    float* turn = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)) + C::kStages * C::kStageBytes) + (warp - 2) * 32 * 17;
    int g = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int row = (tile / p.n_tiles) * 128 + quarter * 32 + lane, n0 = (tile % p.n_tiles) * BN + c_first;
      float acc[C::kCols];
      if (!split_sum<BN>(s, tmem_base, quarter, c_first, lane, g, p.num_kb, abort_ptr, acc)) break;
      long long orow = row;
      if (p.o_strided && row < p.M) {
        const int j = row % p.o_Wc, t2 = row / p.o_Wc;
        const int i = t2 % p.o_Hc, nn = t2 / p.o_Hc;
        orow = ((long long)nn * p.o_H + p.o_h0 + p.o_sh * i) * p.o_W + p.o_w0 + p.o_sw * j;
      }
      orow = row < p.M ? orow * p.ldo : -1;
      // sixteen columns at a time through shared memory, so that a store instruction writes two runs of 64 bytes
#pragma unroll
      for (int c0 = 0; c0 < C::kCols; c0 += 16) {
        if (n0 + c0 >= p.N) break;  // warp-uniform
#pragma unroll
        for (int j = 0; j < 16; ++j) turn[lane * 17 + j] = acc[c0 + j];
        __syncwarp();
        const int col = n0 + c0 + (lane & 15);
        const float bias = p.bias && col < p.N ? p.bias[col] : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int r = 2 * i + (lane >> 4);
          const long long off = __shfl_sync(0xffffffffu, orow, r);
          float v = turn[r * 17 + (lane & 15)] + bias;
          if (p.relu) v = fmaxf(v, 0.f);
          if (off >= 0 && col < p.N) p.out[off + col] = v;
        }
        __syncwarp();
      }
    }
  }
  split_teardown(s, tmem_base, warp, C::kTmemCols);
}

struct SplitWgradParams {
  int Cin, Cout, chunks, cblocks, m_tiles, n_tiles, splits, kb_total, kb_per_split;  // chunk: a tap's block of 32 channels; kb: 32 pixels
  int OW, OH, SW, SH, PW, PH, KW;
  float* partial;  // [splits][Cout][taps * Cin]
  long long Kw;    // taps * Cin
  const int* bad;
  int n_bad;
  int* any_bad;
};

template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
split_wgrad_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapDY, const SplitWgradParams p) {
  using C = SplitCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ SplitShared s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  split_setup<BN>(s, warp);
  __syncthreads();
  mtb_wait_prior();
  int word = 0;
  for (int i = threadIdx.x; i < p.n_bad; i += kGemmThreads) word |= p.bad[i];
  split_gather(&s.words, word);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const bool bad = split_refused(s.words);
  if (blockIdx.x == 0 && threadIdx.x == 0) *p.any_bad = bad;
  const uint32_t tmem_base = s.tmem_slot;
  const int units = bad ? 0 : p.m_tiles * p.n_tiles * p.splits;
  volatile int* abort_ptr = &s.abort_flag;
  auto range = [&](int unit, int& kb0, int& kb1) {
    kb0 = unit % p.splits * p.kb_per_split;
    kb1 = kb0 + p.kb_per_split < p.kb_total ? kb0 + p.kb_per_split : p.kb_total;
  };

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&mapX);
      prefetch_tensormap(&mapDY);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int tile = unit / p.splits, m_tile = tile / p.n_tiles, n0 = (tile % p.n_tiles) * BN;
        int kb0, kb1;
        range(unit, kb0, kb1);
        const int valid = p.chunks - m_tile * 4 < 4 ? p.chunks - m_tile * 4 : 4;
        int q_c[4], q_kw[4], q_kh[4];
        for (int q = 0; q < 4; ++q) {
          const int chunk = m_tile * 4 + (q < valid ? q : 0), tap = chunk / p.cblocks;
          q_c[q] = (chunk - tap * p.cblocks) * 64;
          q_kh[q] = tap / p.KW;
          q_kw[q] = tap - q_kh[q] * p.KW;
        }
        int m = kb0 * 32;
        int ow = m % p.OW, t = m / p.OW;
        int oh = t % p.OH, img = t / p.OH;
        for (int kb = kb0; kb < kb1; ++kb, m += 32) {
          if (!mbar_wait(smem_u32(&s.empty[stage]), phase ^ 1u, abort_ptr, 45)) { ok = false; break; }
          const uint32_t full = smem_u32(&s.full[stage]), a_dst = smem_base + stage * C::kStageBytes;
          mbar_expect_tx(full, (uint32_t)valid * 8192u + C::kB);
          const int pw = ow * p.SW - p.PW, ph = oh * p.SH - p.PH;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q < valid) {
              tma_load_im2col_4d(a_dst + q * 8192, &mapX, full, q_c[q], pw, ph, img, (uint16_t)q_kw[q], (uint16_t)q_kh[q]);
              tma_load_im2col_4d(a_dst + q * 8192 + 4096, &mapX, full, q_c[q] + 32, pw, ph, img, (uint16_t)q_kw[q], (uint16_t)q_kh[q]);
            }
          tma_load_3d(a_dst + C::kA, &mapDY, full, 0, m, n0 / 16);  // hi and lo blocks of BN / 32 blocks of channels
          if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
          ow += 32;
          while (ow >= p.OW) {
            ow -= p.OW;
            if (++oh == p.OH) { oh = 0; ++img; }
          }
        }
      }
    }
  } else if (warp == 1) {
    int chains = 0;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
      int kb0, kb1;
      range(unit, kb0, kb1);
      chains += kb1 - kb0;
    }
    split_issue<BN, true>(s, smem_base, tmem_base, chains, abort_ptr);
  } else {
    const int quarter = warp & 3, c_first = warp < 6 ? 0 : C::kCols;
    int g = 0;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
      const int tile = unit / p.splits, chunk = tile / p.n_tiles * 4 + quarter, n0 = (tile % p.n_tiles) * BN + c_first;
      int kb0, kb1;
      range(unit, kb0, kb1);
      float acc[C::kCols];
      if (!split_sum<BN>(s, tmem_base, quarter, c_first, lane, g, kb1 - kb0, abort_ptr, acc)) break;
      const int tap = chunk / p.cblocks, ci = (chunk - tap * p.cblocks) * 32 + lane;
      if (chunk < p.chunks && ci < p.Cin) {
        float* out = p.partial + ((long long)(unit % p.splits) * p.Cout + n0) * p.Kw + (long long)tap * p.Cin + ci;
#pragma unroll
        for (int j = 0; j < C::kCols; ++j)
          if (n0 + j < p.Cout) out[j * p.Kw] = acc[j];
      }
      __syncwarp();
    }
  }
  split_teardown(s, tmem_base, warp, C::kTmemCols);
}

// out = sum of the planes in order, or that added to what the images before have left
__global__ void __launch_bounds__(256) split_add_planes_kernel(const float* __restrict__ planes, float* __restrict__ out, long long n, int count, int accumulate,
                                                               const int* __restrict__ any_bad) {
  mtb_launch_dependents();
  mtb_wait_prior();
  if (*any_bad) return;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
    float v = 0.f;
#pragma unroll 8
    for (int z = 0; z < count; ++z) v += planes[z * n + i];
    out[i] = accumulate ? out[i] + v : v;
  }
}

// ------------------------------------------------------------------------------ host

struct SplitGeometry { int n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, oh, ow; };

int split_blocks(int c) { return (c + 31) / 32; }
// Column tile: the fewest bytes copied into shared memory per 128 rows (the rows once per tile, its columns).
int split_bn(int n) {
  auto cost = [n](int bn) { return (n + bn - 1) / bn * (128 + bn); };
  int best = 128;
  for (int bn : {96, 64, 32})
    if (cost(bn) < cost(best)) best = bn;
  return best;
}

constexpr long long kSplitPacked = 64LL << 20;      // packed activations of one operand at a time, which the L2 holds
constexpr long long kSplitMost = 256LL << 20;       // most that one packed image, or the packed filter, may take: scratch is kept, and is not to grow with them
constexpr long long kSplitHeader = 4 * (2 * 1024 + 1024);  // words of the packing pass, then one per group of images

// images per pass
int split_images(const SplitGeometry& q, bool with_x, bool with_dy) {
  const long long x = with_x ? (long long)q.h * q.w * split_blocks(q.cin) * 256 : 0, dy = with_dy ? (long long)q.oh * q.ow * split_blocks(q.cout) * 256 : 0;
  const long long image = x > dy ? x : dy;
  long long k = kSplitPacked / image;
  if (k < 1) k = 1;
  const int passes = (int)((q.n + k - 1) / k);
  return (q.n + passes - 1) / passes;  // equal passes
}
long long split_x_bytes(const SplitGeometry& q, int images) { return (long long)images * q.h * q.w * split_blocks(q.cin) * 256; }
long long split_dy_bytes(const SplitGeometry& q, int images) { return (long long)images * q.oh * q.ow * split_blocks(q.cout) * 256; }

// The filter as forward and data gradient read it; for the weight gradient one plane of sums.
long long split_filter_bytes(const SplitGeometry& q, int direction) {
  const long long taps = (long long)q.kh * q.kw;
  if (direction == 0) return q.cout * taps * split_blocks(q.cin) * 256;
  if (direction == 1) return q.cin * taps * split_blocks(q.cout) * 256;
  return q.cout * taps * q.cin * 4;
}

struct SplitWgradPlan {
  int images, bn, chunks, m_tiles, n_tiles, splits;
  bool whole;  // one group of images in one piece: sums go to dw, not to planes
};
SplitWgradPlan split_wgrad_plan(const SplitGeometry& q) {
  SplitWgradPlan r;
  r.images = split_images(q, true, true);
  r.bn = split_bn(q.cout);
  r.chunks = q.kh * q.kw * split_blocks(q.cin);
  r.m_tiles = (r.chunks + 3) / 4;
  r.n_tiles = (q.cout + r.bn - 1) / r.bn;
  const int kb = (int)(((long long)r.images * q.oh * q.ow + 31) / 32);
  int s = mtb_sm_count() / (r.m_tiles * r.n_tiles);
  if (s > kb / 8) s = kb / 8;
  r.splits = s < 1 ? 1 : s;
  r.whole = r.splits == 1 && r.images >= q.n;
  return r;
}

// What the launches of one direction take, in us.  A reduction block costs what the copy engine takes for its 128-byte rows
// (3.4 cycles each: 128 x 96 blocks 0.83 us, 128 x 64 0.65); a pass over memory that the L2 holds moves about 4.5 TB/s; three
// launches around the products take about 8.
double split_us(const SplitGeometry& q, int direction) {
  auto block_us = [](int bn) { return (256 + 2 * bn) * 0.00184; };
  auto waves = [](double tiles) { return std::ceil(tiles / mtb_sm_count()); };
  const double taps = q.kh * q.kw, in = (double)q.n * q.h * q.w, out = (double)q.n * q.oh * q.ow;
  const double x = in * (4.0 * q.cin + 256.0 * split_blocks(q.cin)), dy = out * (4.0 * q.cout + 256.0 * split_blocks(q.cout));
  if (direction == 2) {
    const SplitWgradPlan r = split_wgrad_plan(q);
    const double passes = std::ceil((double)q.n / r.images), blocks = std::ceil(out / passes / 32 / r.splits);
    const double planes = 8.0 * r.splits * taps * q.cin * q.cout;
    return 8 + (x + dy) / 4.5e6 + passes * (waves((double)r.m_tiles * r.n_tiles * r.splits) * blocks * block_us(r.bn) + planes / 4.5e6 + 6);
  }
  const bool forward = direction == 0;
  const int images = split_images(q, forward, !forward), cols = forward ? q.cout : q.cin, bn = split_bn(cols), classes = forward ? 1 : q.sh * q.sw;
  const double passes = std::ceil((double)q.n / images), rows = (forward ? out : in) / passes / classes;
  const double blocks = (forward ? taps : std::ceil((double)q.kh / q.sh) * std::ceil((double)q.kw / q.sw)) * split_blocks(forward ? q.cin : q.cout);
  const double tile_waves = waves(std::ceil(rows / 128) * ((cols + bn - 1) / bn));
  const double store = rows * cols * 4 / 3e6;  // longer than the products of a short reduction
  const double products = tile_waves * blocks * block_us(bn);
  return 8 + (forward ? x : dy) / 4.5e6 + passes * classes * ((products > store ? products : store) + 4);
}

// Most terms of a sum that are not padding: of an output's window at most h x w taps lie on the image, of an input's window (the
// residue class with the fewest taps) at most oh x ow; a filter entry meets every image at most ceil(h / sh) x ceil(w / sw) times.
long long split_terms(const SplitGeometry& q, int direction) {
  auto least = [](int a, int b) { return a < b ? a : b; };
  auto class_taps = [&](int k, int s, int size) { return least(k / s > 0 ? k / s : 1, size); };
  if (direction == 0) return (long long)least(q.kh, q.h) * least(q.kw, q.w) * q.cin;
  if (direction == 1) return (long long)class_taps(q.kh, q.sh, q.oh) * class_taps(q.kw, q.sw, q.ow) * q.cout;
  return (long long)q.n * least(q.oh, (q.h + q.sh - 1) / q.sh) * least(q.ow, (q.w + q.sw - 1) / q.sw);
}

// Whether the two-term products take a direction: within the copy engine's limits, cheaper than the CUDA-core kernels, and a
// reduction of at least 96.  A sum of fewer terms rounds less in FP32 than the operands do here (relative errors against 64
// bits: 20 terms 8.2e-8 on the CUDA cores, 1.15e-7 here; 27 terms 9.4e-8 and 1.07e-7; 96 terms 1.76e-7 and 1.33e-7; 432 terms
// 3.7e-7 and 1.5e-7; 3600 terms 1.06e-6 and 2.3e-7; weight gradients over 43,808 pixels 6.6e-7 and 2.1e-7).  Of 30 shapes
// of 3 to 512 channels the price took the slower side for none; it left the faster one for seven directions, by 1.8 times at
// most (strided data gradients, few pixels under a wide filter).
bool split_takes(const SplitGeometry& q, int direction) {
  const bool always = getenv("MTB_TC_SPLIT_ALWAYS") != nullptr;  // for tests of small shapes
  // 4e7 products take the CUDA cores about 15 us, less than the launches here; a small network's calls end at this test
  if ((double)q.n * q.oh * q.ow * q.cout * q.cin * q.kh * q.kw < 4e7 && !always) return false;
  if (getenv("MTB_DISABLE_TC") || getenv("MTB_DISABLE_TC_SPLIT")) return false;
  if (q.sh > 8 || q.sw > 8 || q.ph > 64 || q.pw > 64 || q.kh > 32 || q.kw > 32 || q.kh * q.kw > 64) return false;
  if (split_x_bytes(q, q.n) < kMinIm2colBytes || split_dy_bytes(q, q.n) < kMinIm2colBytes) return false;
  if (split_x_bytes(q, 1) > kSplitMost || split_dy_bytes(q, 1) > kSplitMost || split_filter_bytes(q, direction) > kSplitMost) return false;
  if (split_terms(q, direction) < 96 && !always) return false;
  // items of the packing pass are numbered with 32 bits
  const int images = split_images(q, true, true);
  const long long most = (split_x_bytes(q, images) + split_dy_bytes(q, images)) / 32 + (long long)q.kh * q.kw * (q.cin + 32LL) * (q.cout + 32LL);
  if (most >= (1LL << 31) || q.n > 1024LL * images) return false;
  return always || split_us(q, direction) < 0.9 * mtb_conv2d_simt_us(q.n, q.cin, q.h, q.w, q.kh, q.kw, q.sh, q.sw, q.ph, q.pw, q.cout, direction);
}

SplitSide split_rows(const float* src, float* dst, long long rows, int c) {
  return SplitSide{src, dst, rows, c, 0, 1, 1, c, split_blocks(c), c % 4 == 0 && al16(src)};
}

int split_pack(const SplitSide& a, const SplitSide& b, int* bad, int* n_bad, cudaStream_t st) {
  const long long items = a.rows * a.blocks * 8 + b.rows * b.blocks * 8;
  long long blocks = (items + 1023) / 1024;
  if (blocks > kSplitPackBlocks) blocks = kSplitPackBlocks;
  *n_bad = (int)blocks;
  MTB_LAUNCH(split_pack_kernel, dim3((unsigned)blocks), dim3(256), 0, st, a, b, bad);
  MTB_LAUNCH_CHECK("split_pack_kernel");
  return MTB_OK;
}

template <int BN>
int launch_split_gemm(const CUtensorMap& a, const CUtensorMap& b, const SplitGemmParams& p, cudaStream_t st) {
  static unsigned long long configured = 0;
  if (int rc = mtb_opt_in_smem((const void*)split_gemm_kernel<BN>, (int)SplitCfg<BN>::kSmemBytes, &configured)) return rc;
  const int tiles = p.m_tiles * p.n_tiles, grid = tiles < mtb_sm_count() ? tiles : mtb_sm_count();
  MTB_LAUNCH(split_gemm_kernel<BN>, dim3(grid), dim3(kGemmThreads), SplitCfg<BN>::kSmemBytes, st, a, b, p);
  MTB_LAUNCH_CHECK("split_gemm_kernel");
  return MTB_OK;
}
int launch_split_gemm_bn(int bn, const CUtensorMap& a, const CUtensorMap& b, const SplitGemmParams& p, cudaStream_t st) {
  if (bn == 32) return launch_split_gemm<32>(a, b, p, st);
  if (bn == 64) return launch_split_gemm<64>(a, b, p, st);
  if (bn == 96) return launch_split_gemm<96>(a, b, p, st);
  return launch_split_gemm<128>(a, b, p, st);
}
template <int BN>
int launch_split_wgrad(const CUtensorMap& a, const CUtensorMap& b, const SplitWgradParams& p, cudaStream_t st) {
  static unsigned long long configured = 0;
  if (int rc = mtb_opt_in_smem((const void*)split_wgrad_kernel<BN>, (int)SplitCfg<BN>::kSmemBytes, &configured)) return rc;
  const int units = p.m_tiles * p.n_tiles * p.splits, grid = units < mtb_sm_count() ? units : mtb_sm_count();
  MTB_LAUNCH(split_wgrad_kernel<BN>, dim3(grid), dim3(kGemmThreads), SplitCfg<BN>::kSmemBytes, st, a, b, p);
  MTB_LAUNCH_CHECK("split_wgrad_kernel");
  return MTB_OK;
}

SplitGeometry split_geometry(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  return SplitGeometry{n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, (h + 2 * ph - kh) / sh + 1, (w + 2 * pw - kw) / sw + 1};
}

}  // namespace

// Scratch of the two-term products for any of the three directions (0: they do not take this convolution).
long long mtb_split_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction) {
  const SplitGeometry q = split_geometry(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (!split_takes(q, direction)) return 0;
  const long long filter = split_filter_bytes(q, direction);
  if (direction == 0) return kSplitHeader + split_x_bytes(q, split_images(q, true, false)) + filter;
  if (direction == 1) return kSplitHeader + split_dy_bytes(q, split_images(q, false, true)) + filter;
  const SplitWgradPlan r = split_wgrad_plan(q);
  return kSplitHeader + split_x_bytes(q, r.images) + split_dy_bytes(q, r.images) + (r.whole ? 0 : r.splits * filter);
}

// *guard: the words that say whether the operands could not be split (*guards of them; the CUDA-core kernel then does the work).
int mtb_split_conv2d_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* wt,
                                 const float* bias, float* y, int relu, void* workspace, cudaStream_t st, const int** guard, int* guards) {
  const SplitGeometry q = split_geometry(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  const int images = split_images(q, true, false), bn = split_bn(cout), cb = split_blocks(cin), taps = kh * kw;
  int* const bad = (int*)workspace;
  int* const any = bad + 2048;
  float* const xp = (float*)((char*)workspace + kSplitHeader);
  float* const wp = xp + split_x_bytes(q, images) / 4;
  CUtensorMap mapA, mapB;
  int rc = tc::encode_tiled_2d(&mapB, wp, cout, (long long)taps * cb * 64, (long long)taps * cb * 64, 32, bn);
  if (rc) return rc;
  SplitSide ws = split_rows(wt, wp, (long long)cout * taps, cin);
  int pass = 0, n_bad_w = 0;
  for (int first = 0; first < n; first += images, ++pass) {
    const int some = n - first < images ? n - first : images;
    SplitGemmParams p{};
    const SplitSide xs = split_rows(x + (long long)first * h * w * cin, xp, (long long)some * h * w, cin);
    // the filter is packed with the first images, and its words stay
    int* const words = pass ? bad + 1024 : bad;
    if (pass) ws.rows = 0;
    int count = 0;
    if ((rc = split_pack(xs, ws, words, &count, st))) return rc;
    if (!pass) n_bad_w = count;
    p.bad = bad;
    p.n_bad = pass ? 1024 + count : n_bad_w;
    if (!pass && n_bad_w < 1024 && images < n) MTB_CUDA(cudaMemsetAsync(bad + n_bad_w, 0, (1024 - n_bad_w) * 4, st));
    p.any_bad = any + pass;
    if ((rc = tc::encode_im2col_4d(&mapA, xp, some, h, w, cb * 64, -pw, -ph, pw - (kw - 1), ph - (kh - 1), sw, sh, 32, 128))) return rc;
    p.M = some * q.oh * q.ow; p.N = cout; p.num_kb = taps * cb;
    p.m_tiles = (p.M + 127) / 128; p.n_tiles = (cout + bn - 1) / bn;
    p.out = y + (long long)first * q.oh * q.ow * cout; p.ldo = cout; p.bias = bias; p.relu = relu;
    p.OW = q.ow; p.OH = q.oh; p.SW = sw; p.SH = sh; p.PW = pw; p.PH = ph; p.KW = kw; p.KH = kh; p.cblocks = cb;
    for (int t = 0; t < taps; ++t) p.b_tap[t] = t * cb * 64;
    if ((rc = launch_split_gemm_bn(bn, mapA, mapB, p, st))) return rc;
  }
  *guard = any;
  *guards = pass;
  return MTB_OK;
}

// See mtb_tc_conv2d_dgrad_f32 for the residue classes.
int mtb_split_conv2d_dgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy, const float* wt,
                               float* dx, void* workspace, cudaStream_t st, const int** guard, int* guards) {
  const SplitGeometry q = split_geometry(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  const int images = split_images(q, false, true), bn = split_bn(cin), cb = split_blocks(cout), taps = kh * kw;
  int* const bad = (int*)workspace;
  int* const any = bad + 2048;
  float* const dyp = (float*)((char*)workspace + kSplitHeader);
  float* const wp = dyp + split_dy_bytes(q, images) / 4;
  CUtensorMap mapA, mapB;
  int rc = tc::encode_tiled_2d(&mapB, wp, cin, (long long)taps * cb * 64, (long long)taps * cb * 64, 32, bn);
  if (rc) return rc;
  SplitSide ws{wt, wp, (long long)cin * taps, 1, cin, (long long)taps * cin, taps, cout, cb, 0};
  bool need_zero = false;
  for (int a = 0; a < sh; ++a)
    for (int b = 0; b < sw; ++b) {
      const ClassAxis ah = class_axis(a, h, q.oh, kh, sh, ph), aw = class_axis(b, w, q.ow, kw, sw, pw);
      if (ah.count > 0 && aw.count > 0 && (ah.taps == 0 || aw.taps == 0)) need_zero = true;
    }
  if (need_zero) MTB_CUDA(cudaMemsetAsync(dx, 0, (size_t)n * h * w * cin * 4, st));
  int pass = 0, n_bad_w = 0;
  for (int first = 0; first < n; first += images, ++pass) {
    const int some = n - first < images ? n - first : images;
    const SplitSide ds = split_rows(dy + (long long)first * q.oh * q.ow * cout, dyp, (long long)some * q.oh * q.ow, cout);
    int* const words = pass ? bad + 1024 : bad;
    if (pass) ws.rows = 0;
    int count = 0;
    if ((rc = split_pack(ds, ws, words, &count, st))) return rc;
    if (!pass) n_bad_w = count;
    if (!pass && n_bad_w < 1024 && images < n) MTB_CUDA(cudaMemsetAsync(bad + n_bad_w, 0, (1024 - n_bad_w) * 4, st));
    for (int a = 0; a < sh; ++a)
      for (int b = 0; b < sw; ++b) {
        const ClassAxis ah = class_axis(a, h, q.oh, kh, sh, ph), aw = class_axis(b, w, q.ow, kw, sw, pw);
        if (ah.count == 0 || aw.count == 0 || ah.taps == 0 || aw.taps == 0) continue;
        if ((rc = tc::encode_im2col_4d(&mapA, dyp, some, q.oh, q.ow, cb * 64, aw.lower, ah.lower, aw.upper, ah.upper, 1, 1, 32, 128))) return rc;
        SplitGemmParams p{};
        p.bad = bad;
        p.n_bad = pass ? 1024 + count : n_bad_w;
        p.any_bad = any + pass;
        p.M = some * ah.count * aw.count; p.N = cin; p.num_kb = ah.taps * aw.taps * cb;
        p.m_tiles = (p.M + 127) / 128; p.n_tiles = (cin + bn - 1) / bn;
        p.out = dx + (long long)first * h * w * cin; p.ldo = cin;
        p.OW = aw.count; p.OH = ah.count; p.SW = 1; p.SH = 1; p.PW = -aw.lower; p.PH = -ah.lower; p.KW = aw.taps; p.KH = ah.taps; p.cblocks = cb;
        for (int jh = 0; jh < ah.taps; ++jh)
          for (int jw = 0; jw < aw.taps; ++jw) {
            const int fkh = a + sh * (ah.taps - 1 - jh), fkw = b + sw * (aw.taps - 1 - jw);
            p.b_tap[jh * aw.taps + jw] = (fkh * kw + fkw) * cb * 64;
          }
        p.o_strided = sh * sw > 1; p.o_Hc = ah.count; p.o_Wc = aw.count; p.o_H = h; p.o_W = w; p.o_h0 = ah.start; p.o_w0 = aw.start; p.o_sh = sh; p.o_sw = sw;
        if ((rc = launch_split_gemm_bn(bn, mapA, mapB, p, st))) return rc;
      }
  }
  *guard = any;
  *guards = pass;
  return MTB_OK;
}

int mtb_split_conv2d_wgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x, const float* dy,
                               float* dw, void* workspace, cudaStream_t st, const int** guard, int* guards) {
  const SplitGeometry q = split_geometry(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  const SplitWgradPlan r = split_wgrad_plan(q);
  const int xb = split_blocks(cin), yb = split_blocks(cout);
  int* const bad = (int*)workspace;
  int* const any = bad + 2048;
  float* const xp = (float*)((char*)workspace + kSplitHeader);
  float* const dyp = xp + split_x_bytes(q, r.images) / 4;
  float* const planes = dyp + split_dy_bytes(q, r.images) / 4;
  const long long total = (long long)kh * kw * cin * cout;
  int pass = 0;
  for (int first = 0; first < n; first += r.images, ++pass) {
    const int some = n - first < r.images ? n - first : r.images;
    const long long pixels = (long long)some * q.oh * q.ow;
    int count = 0, rc;
    if ((rc = split_pack(split_rows(x + (long long)first * h * w * cin, xp, (long long)some * h * w, cin),
                         split_rows(dy + (long long)first * q.oh * q.ow * cout, dyp, pixels, cout), bad, &count, st)))
      return rc;
    CUtensorMap mapX, mapDY;
    if ((rc = tc::encode_im2col_4d(&mapX, xp, some, h, w, xb * 64, -pw, -ph, pw - (kw - 1), ph - (kh - 1), sw, sh, 32, 32, true))) return rc;
    if ((rc = tc::encode_blocks_3d(&mapDY, dyp, pixels, yb * 64, yb * 64, 32, r.bn / 16))) return rc;
    SplitWgradParams p{};
    p.Cin = cin; p.Cout = cout; p.chunks = r.chunks; p.cblocks = xb; p.m_tiles = r.m_tiles; p.n_tiles = r.n_tiles;
    p.kb_total = (int)((pixels + 31) / 32);
    p.kb_per_split = (p.kb_total + r.splits - 1) / r.splits;
    p.splits = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;
    p.OW = q.ow; p.OH = q.oh; p.SW = sw; p.SH = sh; p.PW = pw; p.PH = ph; p.KW = kw;
    p.partial = r.whole ? dw : planes;
    p.Kw = (long long)kh * kw * cin;
    p.bad = bad; p.n_bad = count; p.any_bad = any + pass;
    if (r.bn == 32) rc = launch_split_wgrad<32>(mapX, mapDY, p, st);
    else if (r.bn == 64) rc = launch_split_wgrad<64>(mapX, mapDY, p, st);
    else if (r.bn == 96) rc = launch_split_wgrad<96>(mapX, mapDY, p, st);
    else rc = launch_split_wgrad<128>(mapX, mapDY, p, st);
    if (rc) return rc;
    if (!r.whole) {
      MTB_LAUNCH(split_add_planes_kernel, dim3(mtb_stream_grid(total, 256)), dim3(256), 0, st, planes, dw, total, p.splits, pass > 0, any + pass);
      MTB_LAUNCH_CHECK("split_add_planes_kernel");
    }
  }
  *guard = any;
  *guards = pass;
  return MTB_OK;
}
