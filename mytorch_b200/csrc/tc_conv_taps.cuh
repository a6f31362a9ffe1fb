// 3x3 stride-1 convolution with padding 1 over up to 128 reduction channels (and its data gradient) by pairs of SMs.
//
// What bounds the row-staged kernel (tc_conv_rows.cuh) on narrow layers is shared memory: a 128 x 64 x 8 MMA reads 6 KB of operands
// in 48 cycles, 128 B per cycle, while it could do its arithmetic in 32, and the copies of the next stage want their share.  Here a
// cluster of two CTAs issues MMAs of 256 rows together (cta_group::2): each holds the pixels of its own 128 rows and HALF of the filter,
// which the tensor cores of both read.  That takes an MMA of 64 columns to 5 KB a SM, and halves what the filter takes: it stays
// resident up to 128 reduction channels (74 KB for 64), also beside the long rows of 56x56 images, for which the row-staged kernel
// streams it.  Beyond that, two forms:
//
//   BESIDE = 1: one accumulator of 64 columns; tap (kh, kw) reads the staged pixels (kh - 1) rows and (kw - 1) pixels away.  5 KB for
//               each of 72 MMAs a tile and 64 reduction channels, about 3,300 cycles.
//   BESIDE = 2: the pixels are read once for TWO taps of a filter row: an MMA of 128 columns computes taps kw = 0 and 1 of the same
//               pixels side by side, D_0[p] and D_1[p]; one of 64 columns adds tap kw = 2, a pixel further, to D_1.  Then
//                   y[p] = D_0[p - 1] + D_1[p],
//               which the epilogue adds up from neighbouring lanes.  11 KB instead of 15 for three taps, 104 cycles: about 2,500 per
//               64 reduction channels; but the epilogue gets longer.
//
// BESIDE = 2 is taken above 64 reduction channels, where a tile's MMAs outlast its epilogue (128 -> 128 on 512 x 16x16, us: plain 74 and
// 66, with addition 76 and 70; 96 -> 96 on 64 x 30x30 31 and 29); up to 64 the epilogue decides (64 -> 64 on 512 x 32x32: plain 72 and
// 70, statistics 73 and 78, with addition 90 and 106).  The form follows from the channels alone, so that a layer's results are the same
// bits with every epilogue.  All three taps side by side (192 columns, 96 cycles) left room for two accumulators only and doubled the
// exchange between lanes: 78 us where the others take 70.
//
// Before (row-staged or im2col kernel, whichever was taken) -> now, us, cold L2: 64 -> 64 on 512 x 32x32 forward with statistics 93 -> 73,
// data gradient 92 -> 72, with addition 126 -> 90; on 128 x 56x56 75 -> 58, 78 -> 57, 124 -> 74; 128 -> 128 on 512 x 16x16 78 -> 67, 85 -> 66, 114 -> 70;
// on 128 x 28x28 74 -> 53, 60 -> 53, 80 -> 55.  268 MB of the first cross HBM in 41 us.
//
// Positions are those of tc_conv_rows.cuh: image rows of Wp = W + 2 pixels, images separated by one row of zeros.  Each stage holds
// the whole image rows that a tile touches, 32 channels; rows are placed so that the tile's first position is always at the same
// offset, since both CTAs read through one descriptor.  Where whole image rows fill at least nine tenths of a tile's 128 rows, a tile
// is whole image rows: fewer rows to copy and smaller stages, so that three fit where two did (128 -> 128 on 128 x 28x28 61 -> 53 us).
//
// One producing warp and eight epilogue warps a CTA, one issuing warp a pair.  The barriers that the issuing CTA waits on live in
// that CTA; the other one's copies and epilogue signal them there, and the issuer's commits arrive in both.  Waits are bounded
// (tc_common.cuh); a CTA that gives up makes the other one's waits run out.
#pragma once

namespace {
using namespace tc;

constexpr int kTapsBufs = 4;         // accumulators in tensor memory
constexpr int kTapsMaxStages = 4;
constexpr int kTapsMaxChunks = 4;    // blocks of 32 reduction channels: up to 128
constexpr uint32_t kTapsGroup = 3u * 32u * 128u;  // one CTA's half of the three taps of a filter row, 32 reduction channels x 64 outputs
constexpr int kTapsThreads = 32 * (2 + 8);  // producer, issuer, eight epilogue warps
constexpr uint32_t kTapsMaxSmem = 227u * 1024u - 4096u;  // what is left beside the kernel's own shared variables
// The least that a kernel by pairs of SMs takes: more than half of an SM's 228 KB (a CTA takes 1 KB beside its own), so that no SM holds CTAs of two of them.
// Allocating tensor memory waits without a limit, and a pair holds what one CTA has got until the other has its own: two pairs of different streams (a data
// gradient and the weight gradient beside it), each with its columns on one of two SMs, would wait for each other for good.
// (The filter and two stages of this kernel are always more.)
constexpr uint32_t kPairMinSmem = 114u * 1024u;

struct TapsParams {
  long long Q;             // positions: N * Hv * Wp
  int Wp, Hv, H, W;
  int cchunks;             // reduction channels / 32
  int N;                   // output channels
  int m_items, n_tiles;    // pairs of tiles, tiles of 64 output channels
  int tile_step, lead;     // positions from one tile to the next; accumulator rows in front of the tile's first result
  int rows;                // whole image rows a tile yields, 0: tiles start anywhere
  int origin;              // where in a stage the position of accumulator row 0 lies
  int stages;
  uint32_t a_stage_bytes;
  float* out;
  const float* bias;
  const float* addend;     // optional [same shape as out]: out = conv + addend
  MtbBnEval bn;            // EPI_BN
  int relu;
  int b_tap_x[9];          // first column of tap j in the weight matrix
  float* stats;            // EPI_STATS: partial rows [((pair / n_tiles) * 2 + CTA of the pair) * 4 + epilogue warp][3][N]
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// One arrival, and the bytes to wait for, on a barrier of another CTA of the cluster.  No scope beyond the default: what is handed over
// lies in tensor memory, ordered by the tcgen05 fences, or was written by the copy engine.  (A release at cluster scope waits for the
// epilogue's stores to global memory.)
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// copies whose barrier may be the other CTA's of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c, int w, int h, int n) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n)
               : "memory");
}
__device__ __forceinline__ void mma_tf32_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "mov.b64 da, {%1, %2};\n"
      "mov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], da, db, %5, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate));
}
// one arrival on the barrier at this offset in both CTAs when every MMA issued so far by this thread has completed
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// eight consecutive floats on a 32-byte boundary: a lane's whole sector in one access, as st_global_v8
__device__ __forceinline__ void ld_global_v8(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
// the four epilogue warps of one half of the columns
__device__ __forceinline__ void epilogue_sync(int half) { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); }
__device__ __forceinline__ bool epilogue_all(int half, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 q, %1, 0;\n"
      "bar.red.and.pred p, %2, 128, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(r)
      : "r"((uint32_t)ok), "r"(1 + half)
      : "memory");
  return r != 0;
}

template <int BESIDE, int BMODE, int EPI>
__global__ void __launch_bounds__(kTapsThreads, 1)
tc_conv_taps_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const TapsParams p) {
  constexpr bool STATS = EPI == EPI_STATS, BNORM = EPI == EPI_BN;
  constexpr int BN = 64, DN = BESIDE * BN;  // output channels, accumulator columns
  extern __shared__ uint8_t smem_raw[];
  __shared__ alignas(16) BnColumns<BNORM ? BN : 4> bn_columns;
  __shared__ alignas(16) float edge[2][2][4][32];  // what the next epilogue warp's first lane needs of this one's last (by half of the columns, tile parity)
  __shared__ uint64_t bar_afull[kTapsMaxStages], bar_aempty[kTapsMaxStages], bar_bfull[kTapsMaxChunks], bar_tfull[kTapsBufs], bar_tempty[kTapsBufs];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t b_base = smem_base + (uint32_t)p.stages * p.a_stage_bytes;
  const int ST = p.stages;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTapsMaxStages; ++s) {
      mbar_init(smem_u32(&bar_afull[s]), 2);  // both CTAs' producers
      mbar_init(smem_u32(&bar_aempty[s]), 1);
    }
    for (int c = 0; c < kTapsMaxChunks; ++c) mbar_init(smem_u32(&bar_bfull[c]), 2);
    for (int b = 0; b < kTapsBufs; ++b) {
      mbar_init(smem_u32(&bar_tfull[b]), 1);
      mbar_init(smem_u32(&bar_tempty[b]), 16);  // both CTAs' epilogue warps
    }
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)(kTapsBufs * DN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  const int n0 = (pair % p.n_tiles) * BN;                            // a pair stays on its output channels
  const int first = pair / p.n_tiles, step = pairs / p.n_tiles;      // items of this pair
  mtb_wait_prior();  // everything above overlaps the end of the kernel before
  if constexpr (BNORM) load_bn_columns<BN>(bn_columns, p.bn, n0, p.N);
  tc_fence_before();
  __syncthreads();
  cluster_arrive();  // the barriers of both CTAs are ready before either signals the other's
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  volatile int* abort_ptr = &abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one per CTA)
    // A lane per copy: a thread that issues them one after the other spends about 100 cycles on each, more than the MMAs of a stage take
    // where image rows are short.
    if (lane == 0) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
    }
    const uint32_t row_bytes = (uint32_t)p.Wp * 128u;
    int as = 0;
    uint32_t aphase = 0;
    int filled = 0;
    bool ok = true;
    for (int item = first; item < p.m_items && ok; item += step) {
      const int q0 = (2 * item + (int)rank) * p.tile_step - p.lead;  // position of accumulator row 0
      const int v0 = q0 >= 0 ? q0 / p.Wp : -1;
      const int col = q0 - v0 * p.Wp;
      const int nr = p.rows ? p.rows + 2 : (col + 128) / p.Wp + 3;  // at most 32 (checked on the host)
      // lane r copies image row v0 - 1 + r; rows h >= H (separators) and images outside [0, N) are filled with zeros by the copy
      const int v = v0 - 1 + lane;
      const int img = v >= 0 ? v / p.Hv : -1;
      const int hrow = v - img * p.Hv;
      for (int cc = 0; cc < p.cchunks; ++cc) {
        if (item == first) {
          // this block of the filter, beside the first tile's rows that it multiplies
          if (lane == 0) mbar_expect_tx_cluster(cluster_address(smem_u32(&bar_bfull[cc]), 0), 3u * kTapsGroup);
          __syncwarp();
          if (lane < 9) {
            const int kh = lane / 3, j = lane % 3;
            const int tap = 3 * kh + (BESIDE == 2 && j < 2 ? (int)rank : j), c0 = n0 + 32 * (BESIDE == 2 && j < 2 ? j : (int)rank);
            const uint32_t dst = b_base + (uint32_t)(3 * cc + kh) * kTapsGroup + (uint32_t)j * 4096u;
            const uint32_t bfull = cluster_address(smem_u32(&bar_bfull[cc]), 0);
            if (BMODE == B_KMAJOR) tma_load_2d_pair(dst, &mapB, bfull, p.b_tap_x[tap] + cc * 32, c0);
            else tma_load_2d_pair(dst, &mapB, bfull, p.b_tap_x[tap] + c0, cc * 32);
          }
        }
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_aempty[as]), aphase ^ 1u, abort_ptr, 31));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx_cluster(cluster_address(smem_u32(&bar_afull[as]), 0), (uint32_t)nr * row_bytes);
        __syncwarp();
        // the tile's first position lies at the same place of every stage, whatever its column
        if (lane < nr)
          tma_load_4d_pair(smem_base + as * p.a_stage_bytes + (uint32_t)(p.origin - p.Wp - col) * 128u + (uint32_t)lane * row_bytes, &mapA,
                           cluster_address(smem_u32(&bar_afull[as]), 0), cc * 32, -1, hrow, img);
        ++filled;
        if (++as == ST) { as = 0; aphase ^= 1u; }
      }
    }
    // nobody leaves while the issuing CTA's commits may still arrive here: the last use of every stage has been released
    if (filled < ST) { as = 0; aphase = 1; }
    for (int s = 0; s < ST && s < filled && ok; ++s) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_aempty[as]), aphase ^ 1u, abort_ptr, 32));
      if (++as == ST) { as = 0; aphase ^= 1u; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (first CTA of the pair)
    // One warp is enough here (two in turn, as in tc_conv_rows.cuh: the same times).
    constexpr uint32_t idesc = idesc_tf32(256, DN, 0, BMODE == B_MNMAJOR ? 1 : 0), idesc_one = idesc_tf32(256, BN, 0, BMODE == B_MNMAJOR ? 1 : 0);
    constexpr uint32_t a_hi = desc_hi_kmajor();
    constexpr uint32_t b_hi = BMODE == B_MNMAJOR ? desc_hi_mnmajor() : desc_hi_kmajor();
    constexpr uint32_t b_step = BMODE == B_MNMAJOR ? (1024u >> 4) : (32u >> 4);
    constexpr uint32_t group_step = kTapsGroup >> 4;
    const uint32_t b_lo0 = BMODE == B_MNMAJOR ? desc_lo_mnmajor(b_base) : desc_lo_kmajor(b_base);
    const uint32_t row_step = (uint32_t)p.Wp * 8u;  // one image row, in 16-byte units
    bool ok = true;
    int as = 0, t = 0;
    uint32_t aphase = 0;
    for (int item = first; ok && rank == 0 && item < p.m_items; item += step, ++t) {
      const int buf = t % kTapsBufs;
      const uint32_t use = (uint32_t)(t / kTapsBufs);
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_tempty[buf]), (use & 1u) ^ 1u, abort_ptr, 33));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * DN;
      for (int cc = 0; cc < p.cchunks && ok; ++cc) {
        ok = __all_sync(0xffffffffu, (t > 0 || mbar_wait(smem_u32(&bar_bfull[cc]), 0, abort_ptr, 35)) &&
                                         mbar_wait(smem_u32(&bar_afull[as]), aphase, abort_ptr, 34));
        if (!ok) break;
        tc_fence_after();
        // filter row kh reads (kh - 1) image rows away from the tile's positions
        const uint32_t a_tile = desc_lo_kmajor(smem_base + as * p.a_stage_bytes) + (uint32_t)(p.origin - p.Wp) * 8u;
        const uint32_t b_cc = b_lo0 + (uint32_t)(3 * cc) * group_step;
        if (elect_one()) {
#pragma unroll
          for (int kh = 0; kh < 3; ++kh)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t a_lo = a_tile + kh * row_step + 2 * k, b_lo = b_cc + kh * group_step + k * b_step;
              const uint32_t more = (kh + k) ? 1u : (uint32_t)(cc > 0);
              if constexpr (BESIDE == 1) {
                mma_tf32_pair(d_tmem, a_lo - 8, a_hi, b_lo, b_hi, idesc_one, more);
                mma_tf32_pair(d_tmem, a_lo, a_hi, b_lo + 256, b_hi, idesc_one, 1u);
                mma_tf32_pair(d_tmem, a_lo + 8, a_hi, b_lo + 512, b_hi, idesc_one, 1u);
              } else {
                mma_tf32_pair(d_tmem, a_lo, a_hi, b_lo, b_hi, idesc, more);
                mma_tf32_pair(d_tmem + BN, a_lo + 8, a_hi, b_lo + 512, b_hi, idesc_one, 1u);
              }
            }
          mma_commit_pair(smem_u32(&bar_aempty[as]));
        }
        __syncwarp();
        if (++as == ST) { as = 0; aphase ^= 1u; }
      }
      if (ok && elect_one()) mma_commit_pair(smem_u32(&bar_tfull[buf]));
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------ epilogue (the last eight warps of either CTA)
    // Two warps share a quarter of the rows, 32 output channels each: half as many shorten the epilogue's chain of waits too little
    // (64 -> 64 on 512 x 32x32, all three taps side by side: 102 us with four warps, 78 with eight).
    const int quarter = warp & 3, half = (warp - 2) >> 2, h0 = 32 * half;
    LaneColMoments moments;
    if constexpr (STATS) moments.reset();
    const int row = quarter * 32 + lane;
    const bool wide = (reinterpret_cast<uintptr_t>(p.out) & 31u) == 0;                                   // 32-byte stores and loads;
    const uintptr_t add_low = p.addend ? reinterpret_cast<uintptr_t>(p.addend) & 31u : 0u;             // 16-byte ones, or single values
    // position -> pixel of this lane's row; padding columns, separator rows and rows that belong to another tile have no output
    auto locate = [&](int item, long long& off) {
      const int q = (2 * item + (int)rank) * p.tile_step - p.lead + row;
      const int v = q >= 0 ? q / p.Wp : 0;
      const int wp = q - v * p.Wp;
      const int img = v / p.Hv;
      const int hrow = v - img * p.Hv;
      off = (((long long)img * p.H + hrow) * p.W + (wp - 1)) * p.N + n0 + h0;
      return item < p.m_items && row >= p.lead && row - p.lead < p.tile_step && q < p.Q && hrow < p.H && wp >= 1 && wp <= p.W;
    };
    auto fetch = [&](float (&to)[STATS ? 1 : 32], long long off, bool valid) {
      if constexpr (!STATS) {
        if (p.addend && valid) {
          const float* from = p.addend + off;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (n0 + h0 + j >= p.N) break;
            if (add_low == 0) {
              ld_global_v8(from + j, to + j);
            } else if ((add_low & 15u) == 0) {
              const float4 a = ld4(from + j), b = ld4(from + j + 4);
              to[j] = a.x; to[j + 1] = a.y; to[j + 2] = a.z; to[j + 3] = a.w;
              to[j + 4] = b.x; to[j + 5] = b.y; to[j + 6] = b.z; to[j + 7] = b.w;
            } else {
#pragma unroll
              for (int k = 0; k < 8; ++k) to[j + k] = from[j + k];
            }
          }
        }
      }
    };
    // What is added is fetched a tile ahead, so that memory's latency is over when it is needed.
    long long ooff, next_off;
    float pre[STATS ? 1 : 32], next_pre[STATS ? 1 : 32];
    bool valid = locate(first, ooff);
    fetch(pre, ooff, valid);
    int t = 0;
    for (int item = first; item < p.m_items; item += step, ++t) {
      const int buf = t % kTapsBufs;
      const uint32_t use = (uint32_t)(t / kTapsBufs);
      const bool next_valid = locate(item + step, next_off);
      fetch(next_pre, next_off, next_valid);
      const bool ok = lane != 0 || mbar_wait(smem_u32(&bar_tfull[buf]), use & 1u, abort_ptr, 36);
      if (!epilogue_all(half, ok)) break;  // all four go on, or none: they meet again below
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * DN + h0);
      uint32_t d[32], side[BESIDE == 2 ? 32 : 1];
      if constexpr (BESIDE == 2) tmem_ld_32x32(t_addr, side);
      tmem_ld_32x32(t_addr + (BESIDE - 1) * BN, d);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_address(smem_u32(&bar_tempty[buf]), 0));
      if constexpr (BESIDE == 2) {
        // lane i needs D_0 of lane i - 1: across the warps' borders through shared memory
        if (lane == 31) {
          float* mine = edge[half][t & 1][quarter];
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(mine + j) = make_uint4(side[j], side[j + 1], side[j + 2], side[j + 3]);
        }
        epilogue_sync(half);
        if (lane == 31) {
          const float* before = edge[half][t & 1][(quarter + 3) & 3];
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const uint4 e = *reinterpret_cast<const uint4*>(before + j);
            side[j] = e.x; side[j + 1] = e.y; side[j + 2] = e.z; side[j + 3] = e.w;
          }
        }
        __syncwarp();
      }
      if constexpr (STATS) {
        if (valid) moments.next_row();
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float o[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          o[j] = __uint_as_float(d[16 * c + j]);
          if constexpr (BESIDE == 2) o[j] += __uint_as_float(__shfl_sync(0xffffffffu, side[16 * c + j], lane + 31));
        }
        const int c0 = 16 * c;
        if (valid && n0 + h0 + c0 < p.N) {
          if constexpr (STATS) moments.add(c0, o);  // of the raw accumulator
          if (p.bias) {
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] += __ldg(p.bias + n0 + h0 + c0 + j);
          }
          if constexpr (BNORM) {
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = (o[j] - bn_columns.mean[h0 + c0 + j]) * bn_columns.scale[h0 + c0 + j] + bn_columns.beta[h0 + c0 + j];
          }
          if constexpr (!STATS) {
            if (p.addend) {
#pragma unroll
              for (int j = 0; j < 16; ++j) o[j] += pre[c0 + j];
            }
          }
          if (p.relu) {
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = fmaxf(o[j], 0.f);
          }
#pragma unroll
          for (int j = 0; j < 16; j += 8)
            st_row8(p.out + ooff + c0 + j, make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]), make_float4(o[j + 4], o[j + 5], o[j + 6], o[j + 7]), wide);
        }
      }
      valid = next_valid;
      ooff = next_off;
      if constexpr (!STATS) {
#pragma unroll
        for (int j = 0; j < 32; ++j) pre[j] = next_pre[j];
      }
    }
    if constexpr (STATS) {
      float* srow = p.stats + (((long long)first * 2 + rank) * 4 + quarter) * 3 * p.N;
      moments.store(srow, p.N, n0 + h0, p.N, p.bias, lane);
    }
  }

  // ------------------------------------------------------------ teardown
  mtb_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let copies in flight land before shared memory is released
  }
  cluster_arrive();  // the other CTA reads this one's filter and signals its barriers until here
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(kTapsBufs * DN)) : "memory");
  }
}

// Whether the kernel takes a shape, its stages and its price.
struct TapsPlan {
  bool ok;
  int beside, Wp, Hv, n_tiles, m_items, pairs, stages, rows, tile_step, lead, origin;
  uint32_t a_stage_bytes, smem_bytes;
  double ns;
};

// Both sides from 64 channels on: with 32 of either nothing is gained (32 -> 64 on 64 x 40x40 20.4 us and 20.5, on 4 x 112x112 16.4 and 16.4, 32 -> 32 on 256 x
// 14x14 14.3 and 14.3).
TapsPlan taps_plan(int n, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int kc, int nout) {
  TapsPlan r{};
  if (kh != 3 || kw != 3 || sh != 1 || sw != 1 || ph != 1 || pw != 1 || kc % 32 || kc < 64 || kc > 32 * kTapsMaxChunks || nout % 16 || nout < 64)
    return r;
  // behind what most layers fail: a look at the environment takes longer than all of that
  if (getenv("MTB_DISABLE_PAIRCONV") || getenv("MTB_DISABLE_ROWCONV") || getenv("MTB_ROWCONV_MIN_ITEMS")) return r;  // the latter ask for other kernels
  r.Wp = w + 2;
  r.Hv = h + 1;
  if (r.Wp > 256 || r.Wp < 6) return r;  // rows the copy engine takes; at most 32 of them in a stage
  const long long Q = (long long)n * r.Hv * r.Wp;
  if (Q > 0x7ff00000LL) return r;  // the kernel indexes positions with 32-bit integers
  const uint32_t filter = (uint32_t)(kc / 32) * 3u * kTapsGroup;
  r.beside = kc <= 64 ? 1 : 2;
  r.rows = 128 / r.Wp;
  if (r.rows * r.Wp * 10 < 128 * 9) r.rows = 0;
  if (r.rows) {
    r.tile_step = r.rows * r.Wp;
    r.origin = r.Wp + 1;  // the image row above, and a position that the first pixel's left tap reads for no result
    r.a_stage_bytes = (uint32_t)(2 * r.Wp + 130) * 128u;
  } else {
    r.lead = r.beside - 1;  // D_0 of the position before
    r.tile_step = 128 - r.lead;
    r.origin = 2 * r.Wp;  // up to a row and its last column above
    r.a_stage_bytes = (uint32_t)(4 * r.Wp + 129) * 128u;
  }
  r.a_stage_bytes = (r.a_stage_bytes + 1023u) & ~1023u;
  const uint32_t fixed = 1024u + filter;
  r.stages = fixed < kTapsMaxSmem ? (int)((kTapsMaxSmem - fixed) / r.a_stage_bytes) : 0;
  if (r.stages > kTapsMaxStages) r.stages = kTapsMaxStages;
  if (r.stages < 2) return r;
  r.smem_bytes = fixed + (uint32_t)r.stages * r.a_stage_bytes;
  r.n_tiles = (nout + 63) / 64;
  r.m_items = (int)((Q + 2 * r.tile_step - 1) / (2 * r.tile_step));
  const int most = cluster_units(2) / 2;
  if (r.n_tiles > most) return r;
  const long long items = (long long)r.m_items * r.n_tiles;
  r.pairs = (int)(items < most ? items : most) / r.n_tiles * r.n_tiles;
  const int per = r.pairs / r.n_tiles;
  const int waves = (r.m_items + per - 1) / per;
  // A price to hold against the other kernels' prices, not a time: launches take 6 us and 0.9 (two taps beside each other: 0.75) to 1.1 us a stage, the other
  // kernels 2 to 3 us more than their prices, and more yet where those are high.  Of 207 shapes of 1 to 34 waves the forward pass so takes this kernel where it
  // is over 3 % slower 6 times plain (two waves of 64 channels, 9.7 us against 8.9; 9 % at most), 28 with statistics (one wave, 0.4 to 0.8 us) and never with
  // running statistics, the data gradient once; it does not where it would be that much faster 12, 15, 21 and 23 times.
  r.ns = 3000.0 + waves * (kc / 32) * 860.0;
  r.ok = true;
  return r;
}

int taps_stats_rows(const TapsPlan& plan) { return plan.pairs / plan.n_tiles * 8; }

template <int BESIDE, int BMODE, int EPI>
int launch_taps_form(const TapsPlan& plan, const CUtensorMap& mapA, const CUtensorMap& mapB, const TapsParams& p, cudaStream_t st) {
  auto kernel = tc_conv_taps_kernel<BESIDE, BMODE, EPI>;
  static unsigned long long configured = 0;
  if (int rc = mtb_opt_in_smem((const void*)kernel, (int)kTapsMaxSmem, &configured)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * plan.pairs);
  cfg.blockDim = dim3(kTapsThreads);
  cfg.dynamicSmemBytes = plan.smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  MTB_CUDA(cudaLaunchKernelEx(&cfg, kernel, mapA, mapB, p));
  MTB_LAUNCH_CHECK("tc_conv_taps_kernel");
  return MTB_OK;
}

template <int BMODE, int EPI>
int launch_taps(const TapsPlan& plan, const CUtensorMap& mapA, const CUtensorMap& mapB, const TapsParams& p, cudaStream_t st) {
  return plan.beside == 1 ? launch_taps_form<1, BMODE, EPI>(plan, mapA, mapB, p, st) : launch_taps_form<2, BMODE, EPI>(plan, mapA, mapB, p, st);
}

// Forward (x, K-major weights [nout][9 kc]) and data gradient (dY, weights in place [kc][9 nout]).
// act: [n, h, w, kc] channels-last; out: [n, h, w, nout].
template <int BMODE>
int run_taps(const TapsPlan& plan, int n, int h, int w, int kc, int nout, const float* act, const float* weights, const float* bias, const float* addend,
             int relu, float* out, cudaStream_t st, float* stats = nullptr, const MtbBnEval* bn_eval = nullptr) {
  CUtensorMap mapA, mapB;
  if (int rc = tc::encode_rows_4d(&mapA, act, n, h, w, kc, 32, plan.Wp)) return rc;
  const long long wrows = BMODE == B_KMAJOR ? nout : kc, wcols = 9LL * (BMODE == B_KMAJOR ? kc : nout);
  if (int rc = tc::encode_tiled_2d(&mapB, weights, wrows, wcols, wcols, 32, 32, BMODE == B_MNMAJOR)) return rc;
  TapsParams p{};
  p.Q = (long long)n * plan.Hv * plan.Wp;
  p.Wp = plan.Wp; p.Hv = plan.Hv; p.H = h; p.W = w;
  p.cchunks = kc / 32; p.N = nout;
  p.m_items = plan.m_items; p.tile_step = plan.tile_step; p.lead = plan.lead; p.rows = plan.rows; p.origin = plan.origin; p.n_tiles = plan.n_tiles; p.stages = plan.stages; p.a_stage_bytes = plan.a_stage_bytes;
  p.out = out; p.bias = bias; p.addend = addend; p.relu = relu; p.stats = stats;
  if (bn_eval) p.bn = *bn_eval;
  // the data gradient is the convolution of dY with the filter rotated by 180 degrees
  for (int tap = 0; tap < 9; ++tap) p.b_tap_x[tap] = BMODE == B_KMAJOR ? tap * kc : (8 - tap) * nout;
  if constexpr (BMODE == B_KMAJOR) {
    if (stats) return launch_taps<BMODE, EPI_STATS>(plan, mapA, mapB, p, st);
    if (bn_eval) return launch_taps<BMODE, EPI_BN>(plan, mapA, mapB, p, st);
  }
  return launch_taps<BMODE, EPI_PLAIN>(plan, mapA, mapB, p, st);
}

}  // namespace
