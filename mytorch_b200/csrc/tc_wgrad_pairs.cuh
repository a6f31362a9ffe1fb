// Weight gradient of a 3x3 stride-1 convolution with padding 1 by pairs of SMs: every tap of 64 input and 64 output channels in one MMA.
//
// In the padded linear positions of tc_conv_rows.cuh
//     dW[kh][kw][ci][co] = sum over q of X[q + kw - 1][ci] * dY[q - (kh - 1) * Wp][co].
// Both operands are [position][32 channels] panels in shared memory, read as MN-major operands with the position as the reduction
// index, and a shift by positions is a shift of the descriptor's start: the four 32-wide blocks of A are the X panel shifted by 0..3
// positions (descriptor LBO = one position; the fourth is dropped), the three of B the dY panel shifted by 0..2 image rows (LBO = one
// image row).  A cluster of two CTAs issues MMAs of 256 x 192 together (cta_group::2): CTA r holds channel block r of X, and of dY, which
// is its half of B.  One MMA of K = 8 positions thus covers nine taps x 64 x 64 channels in 96 cycles of two SMs, reading 7 KB in each;
// the row-staged kernel, which shifts X alone, takes 288 cycles of one SM for it, and its operands 128 B per cycle.  Three quarters of
// the work is used.  A stage is R whole image rows (a multiple of 8 positions: the steps of a stage end where it does), so X needs
// no rows around them and dY one on either side.
//
// Against the kernel that was taken before (row-staged, or im2col for few positions), with the addition of the planes, us, cold L2: 512 x 32x32 113.7 -> 80.9, 128 x 32x32 43.9 ->
// 37.9, 128 x 56x56 97.3 -> 66.7, 32 x 56x56 37.9 -> 31.8, 64 -> 48 on 64 x 40x40 37.9 -> 33.8.  (The MMAs of the first take 56 us, its 268 MB of
// operands 41.)  Errors against 64-bit sums over the rounded operands: 8.9e-6 -> 8.8e-6, 1.0e-5 -> 2.5e-6, 1.3e-5 -> 6.7e-6, 8.1e-6 -> 1.9e-6.
//
// Barriers as in tc_conv_taps.cuh.
#pragma once

namespace {
using namespace tc;

constexpr int kWgPairStages = 4;
constexpr int kWgPairCin = 64;              // input channels: two blocks, one a CTA
constexpr uint32_t kWgPairLead = 8 * 128;  // zeros around the X panel, which shifted reads of positions without a gradient reach
constexpr int kWgPairCols = 192;           // of one accumulator; at 256 lies the second

struct WgradPairParams {
  int Wp, Hv, H, W, rows;          // rows: image rows a stage
  int Cout;                        // 33 to 64
  int stages, groups_total, groups_per_split;
  uint32_t x_bytes, stage_bytes;   // X panel with its zeros; X and dY
  float* partial;                  // [splits][9 * 64][Cout]
};

__global__ void __launch_bounds__(kGemmThreads, 1)
tc_wgrad_pairs_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapDY, const WgradPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[kWgPairStages], bar_empty[kWgPairStages], bar_tfull;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int ST = p.stages;

  for (uint32_t i = threadIdx.x; i < (uint32_t)ST * 2u * (kWgPairLead / 16u); i += blockDim.x) {
    const uint32_t side = i / (kWgPairLead / 16u), at = (side >> 1) * p.stage_bytes + (side & 1u) * (p.x_bytes - kWgPairLead) + i % (kWgPairLead / 16u) * 16u;
    *reinterpret_cast<uint4*>(smem_raw + (smem_base - smem_u32(smem_raw)) + at) = make_uint4(0, 0, 0, 0);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWgPairStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 2);  // both CTAs' producers
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_tfull), 1);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  mtb_wait_prior();
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the barriers of both CTAs are ready before either signals the other's
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  volatile int* abort_ptr = &abort_flag;

  const int split = (int)(blockIdx.x >> 1);
  const int ch0 = (int)rank * 32;  // this CTA's block of input channels, and of output channels
  const int g0 = split * p.groups_per_split;
  const int g1 = g0 + p.groups_per_split < p.groups_total ? g0 + p.groups_per_split : p.groups_total;

  const int second = g0 + (g1 - g0 + 1) / 2;  // first group of the second accumulator, if there is one

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA), a lane per image row
    if (lane == 0) {
      prefetch_tensormap(&mapX);
      prefetch_tensormap(&mapDY);
    }
    const uint32_t row_bytes = (uint32_t)p.Wp * 128u;
    const int copies = 2 * p.rows + 2;
    int stage = 0, filled = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int g = g0; g < g1; ++g) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr, 41));
      if (!ok) break;
      if (lane == 0) mbar_expect_tx_cluster(cluster_address(smem_u32(&bar_full[stage]), 0), (uint32_t)copies * row_bytes);
      __syncwarp();
      if (lane < copies) {
        const bool is_x = lane < p.rows;
        const int v = g * p.rows + (is_x ? lane : lane - p.rows - 1);
        const int img = v >= 0 ? v / p.Hv : -1, hrow = v - img * p.Hv;  // separators and images outside [0, N): zeros
        const uint32_t st = smem_base + stage * p.stage_bytes, full = cluster_address(smem_u32(&bar_full[stage]), 0);
        if (is_x) tma_load_4d_pair(st + kWgPairLead + (uint32_t)lane * row_bytes, &mapX, full, ch0, -1, hrow, img);
        else tma_load_4d_pair(st + p.x_bytes + (uint32_t)(lane - p.rows) * row_bytes, &mapDY, full, ch0, -1, hrow, img);
      }
      ++filled;
      if (++stage == ST) { stage = 0; phase ^= 1u; }
    }
    // nobody leaves while the issuing CTA's commits may still arrive here
    if (filled < ST) { stage = 0; phase = 1; }
    for (int s = 0; s < ST && s < filled && ok; ++s) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr, 42));
      if (++stage == ST) { stage = 0; phase ^= 1u; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (first CTA of the pair)
    constexpr uint32_t idesc = idesc_tf32(256, kWgPairCols, 1, 1);
    constexpr uint32_t hi = desc_hi_mnmajor();
    const int steps = p.rows * p.Wp / 8;
    int stage = 0;
    uint32_t phase = 0, acc = 0;
    bool ok = true;
    uint32_t d_tmem = tmem_base;
    for (int g = g0; g < g1 && rank == 0; ++g) {
      // The tensor core truncates at every step, so a chain's error grows with its length: half of the positions go to a second accumulator
      // (512 x 32x32: 1.8e-5 with one, 8.9e-6 in the row-staged kernel's twice as many chains, 8.8e-6 so).
      if (g > g0 && g == second) { d_tmem = tmem_base + 256u; acc = 0u; }
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[stage]), phase, abort_ptr, 43));
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = smem_base + stage * p.stage_bytes;
      // block i of A: X[q - 1 + i], tap kw = i; block j of B: dY[q + (j - 1) * Wp], tap kh = 2 - j
      const uint32_t a_lo = desc_lo_mnmajor(st + kWgPairLead, 128u) - 8u;
      const uint32_t b_lo = desc_lo_mnmajor(st + p.x_bytes, (uint32_t)p.Wp * 128u);
      if (elect_one()) {
#pragma unroll 4
        for (int k = 0; k < steps; ++k) {
          mma_tf32_pair(d_tmem, a_lo + 64u * k, hi, b_lo + 64u * k, hi, idesc, acc);
          acc = 1u;
        }
        mma_commit_pair(smem_u32(&bar_empty[stage]));
      }
      __syncwarp();
      acc = 1u;
      if (++stage == ST) { stage = 0; phase ^= 1u; }
    }
    if (ok && rank == 0 && elect_one()) mma_commit_pair(smem_u32(&bar_tfull));
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (the last eight warps of either CTA): two share a quarter of the rows
    const int quarter = warp & 3, half = (warp - 2) >> 2;  // tap kw; block of 32 output channels
    bool ok = lane != 0 || mbar_wait(smem_u32(&bar_tfull), 0, abort_ptr, 44);
    ok = __all_sync(0xffffffffu, ok);
    const int c0 = 32 * half;
    if (ok && quarter < 3 && c0 < p.Cout) {
      tc_fence_after();
      const bool vec_ok = (p.Cout % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.partial) & 15u) == 0);
      const bool wide_ok = (p.Cout % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.partial) & 31u) == 0);
      float* part = p.partial + (long long)split * 9 * kWgPairCin * p.Cout;
#pragma unroll 1
      for (int j = 0; j < 3; ++j) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 96 + j * 32), r);
        tmem_ld_wait();
        if (second < g1) {
          uint32_t t[32];
          tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + 256u + (uint32_t)(half * 96 + j * 32), t);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 32; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) + __uint_as_float(t[k]));
        }
        float* orow = part + ((long long)((2 - j) * 3 + quarter) * kWgPairCin + ch0 + lane) * p.Cout + c0;
        if (vec_ok && c0 + 32 <= p.Cout) {
#pragma unroll
          for (int k = 0; k < 32; k += 8)
            st_row8(orow + k, make_float4(__uint_as_float(r[k]), __uint_as_float(r[k + 1]), __uint_as_float(r[k + 2]), __uint_as_float(r[k + 3])),
                    make_float4(__uint_as_float(r[k + 4]), __uint_as_float(r[k + 5]), __uint_as_float(r[k + 6]), __uint_as_float(r[k + 7])), wide_ok);
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k)
            if (c0 + k < p.Cout) orow[k] = __uint_as_float(r[k]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  mtb_launch_dependents();  // behind the barrier: see tc_wgrad_kernel
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  cluster_arrive();  // the other CTA reads this one's dY and signals its barriers until here
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

struct WgradPairPlan {
  bool ok;
  int Wp, Hv, rows, stages, groups_total, groups_per_split, splits;
  uint32_t x_bytes, stage_bytes, smem_bytes;
};

WgradPairPlan wgrad_pair_plan(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  WgradPairPlan r{};
  if (kh != 3 || kw != 3 || sh != 1 || sw != 1 || ph != 1 || pw != 1 || cin != kWgPairCin || cout % 4 || cout <= 32 || cout > 64) return r;
  if (getenv("MTB_DISABLE_PAIRCONV") || getenv("MTB_DISABLE_ROWCONV") || getenv("MTB_DISABLE_ROWWGRAD")) return r;  // the latter ask for other kernels
  r.Wp = w + 2;
  r.Hv = h + 1;
  if (r.Wp > 256 || (long long)n * r.Hv * r.Wp > 0x7ff00000LL) return r;
  const int whole = r.Wp % 8 == 0 ? 1 : r.Wp % 4 == 0 ? 2 : r.Wp % 2 == 0 ? 4 : 8;  // image rows that are a multiple of 8 positions
  const uint32_t budget = kTapsMaxSmem - 1024u;
  for (r.rows = 8; r.rows >= whole; r.rows -= whole) {
    r.x_bytes = 2u * kWgPairLead + (uint32_t)(r.rows * r.Wp) * 128u;  // a multiple of 1024: 8 positions
    r.stage_bytes = (r.x_bytes + (uint32_t)((r.rows + 2) * r.Wp) * 128u + 1023u) & ~1023u;
    if (2u * r.stage_bytes <= budget) break;
  }
  if (r.rows < whole) return r;
  r.stages = (int)(budget / r.stage_bytes);
  if (r.stages > kWgPairStages) r.stages = kWgPairStages;
  r.smem_bytes = 1024u + (uint32_t)r.stages * r.stage_bytes;
  if (r.smem_bytes < kPairMinSmem) r.smem_bytes = kPairMinSmem;  // image rows of up to 9 pixels
  const long long image_rows = (long long)n * r.Hv;
  r.groups_total = (int)((image_rows + r.rows - 1) / r.rows);
  int splits = cluster_units(2) / 2;  // a pair each
  if (splits < 1) splits = 1;
  if (splits > r.groups_total) splits = r.groups_total;
  r.groups_per_split = (r.groups_total + splits - 1) / splits;
  r.splits = (r.groups_total + r.groups_per_split - 1) / r.groups_per_split;
  r.ok = true;
  return r;
}

// Whether to take it where its layout fits.  Wider layers are near their best in the im2col kernel (128 -> 128 on 512 x 16x16 81 us and 85, on 128 x
// 28x28 65 and 69).  Few positions a pair do not make up for its planes, one a pair: 1088 positions 27.7 us and 27.6, 840 23.6 and 25.6, 464
// 19.5 and 21.4; 1624 37.9 and 31.8.
bool wgrad_pairs_pay(const WgradPairPlan& r) {
  return r.ok && r.groups_per_split * r.rows * r.Wp >= 1000;
}

int run_wgrad_pairs(const WgradPairPlan& q, int n, int h, int w, int cout, const float* x, const float* dy, float* dw, float* partial, cudaStream_t st) {
  CUtensorMap mapX, mapDY;
  if (int rc = tc::encode_rows_4d(&mapX, x, n, h, w, kWgPairCin, 32, q.Wp, true)) return rc;
  if (int rc = tc::encode_rows_4d(&mapDY, dy, n, h, w, cout, 32, q.Wp, true)) return rc;
  WgradPairParams p{};
  p.Wp = q.Wp; p.Hv = q.Hv; p.H = h; p.W = w; p.rows = q.rows; p.Cout = cout;
  p.stages = q.stages; p.groups_total = q.groups_total; p.groups_per_split = q.groups_per_split;
  p.x_bytes = q.x_bytes; p.stage_bytes = q.stage_bytes; p.partial = partial;
  static unsigned long long configured = 0;
  if (int rc = mtb_opt_in_smem((const void*)tc_wgrad_pairs_kernel, (int)kTapsMaxSmem, &configured)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * q.splits);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = q.smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  MTB_CUDA(cudaLaunchKernelEx(&cfg, tc_wgrad_pairs_kernel, mapX, mapDY, p));
  MTB_LAUNCH_CHECK("tc_wgrad_pairs_kernel");
  const int Kw = 9 * kWgPairCin;
  dim3 rgrid((unsigned)((Kw + 3) / 4), (unsigned)((cout + 31) / 32));
  MTB_LAUNCH(wgrad_reduce_many_kernel, rgrid, dim3(32, 4, 8), 0, st, (const float*)partial, dw, Kw, cout, q.splits);
  MTB_LAUNCH_CHECK("wgrad_reduce_many_kernel");
  return MTB_OK;
}

}  // namespace
