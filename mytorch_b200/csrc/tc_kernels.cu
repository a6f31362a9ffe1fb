// tcgen05 / TMEM / TMA kernels: TF32 GEMM with FP32 accumulation for Linear layers, and
// implicit-GEMM convolution forward and (stride-1) data gradient over channels-last tensors.
//
// One persistent CTA per SM, 320 threads in three roles:
//   warp 0     TMA producer: one lane fills a ring of shared-memory stages (A tile 128 x 32,
//              B tile BN x 32 fp32, 128-byte swizzle).  The convolution's A operand is never
//              materialised: an im2col-mode tensor map gathers 128 output pixels x 32 channels
//              of one filter tap per load, with zero fill for the padding halo.
//   warp 1     MMA issuer: one lane issues tcgen05.mma kind::tf32 (128 x BN x 8 per instruction),
//              accumulating in TMEM; tcgen05.commit releases stages and publishes finished tiles.
//   warps 2-9  epilogue: tcgen05.ld the accumulator (each warp owns a 32-lane TMEM quarter and half of the
//              columns), add bias / apply ReLU, store rows to global memory.  A short reduction is bound by how many
//              loads and stores these warps have in flight: eight instead of four take the 64 <- 256 channel data
//              gradient with addition on 128 x 56x56 from 291 to 213 us.
// Two TMEM accumulator buffers let the epilogue of tile i overlap the main loop of tile i+1.
// All waits are bounded (tc_common.cuh); a kernel that gives up sets g_tc_status and exits.
#include "tc_common.cuh"
#include "kernels.h"
#include <cudaTypedefs.h>

namespace tc {

static PFN_cuTensorMapEncodeTiled_v12000 g_encode_tiled = nullptr;
static PFN_cuTensorMapEncodeIm2col_v12000 g_encode_im2col = nullptr;

// Element type recorded in the tensor maps.  TFLOAT32 makes the copy engine round every fp32
// value to TF32 on its way into shared memory (measured: max relative error of a K=1024 GEMM
// 2.7e-4, against 7.4e-4 when the raw fp32 bits are handed to the MMA, which then simply drops
// the low 13 mantissa bits).  MTB_TMA_FLOAT32=1 selects the unrounded variant for comparison.
static CUtensorMapDataType tma_dtype() {
  static int mode = -1;
  if (mode < 0) mode = getenv("MTB_TMA_FLOAT32") ? 1 : 0;
  return mode ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_TFLOAT32;
}

static int load_driver_entry_points() {
  if (g_encode_tiled && g_encode_im2col) return MTB_OK;
  cudaDriverEntryPointQueryResult q;
  void* fn = nullptr;
  MTB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
  if (q != cudaDriverEntryPointSuccess || !fn) return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
  g_encode_tiled = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  fn = nullptr;
  MTB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &q));
  if (q != cudaDriverEntryPointSuccess || !fn) return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeIm2col is not available in this driver");
  g_encode_im2col = (PFN_cuTensorMapEncodeIm2col_v12000)fn;
  return MTB_OK;
}

int encode_tiled_2d(CUtensorMap* map, const float* base, long long rows, long long cols, long long pitch_elems, int box_cols, int box_rows,
                    bool mn_major) {
  int rc = load_driver_entry_points();
  if (rc) return rc;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch_elems * 4};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode_tiled(map, tma_dtype(), 2, const_cast<float*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) rows=%lld cols=%lld pitch=%lld box=%dx%d", (int)r, rows, cols, pitch_elems, box_cols, box_rows);
  return MTB_OK;
}

int encode_result_2d(CUtensorMap* map, const float* base, long long rows, long long cols, long long pitch_elems) {
  int rc = load_driver_entry_points();
  if (rc) return rc;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch_elems * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeTiled (result) failed (%d) rows=%lld cols=%lld pitch=%lld", (int)r, rows, cols, pitch_elems);
  return MTB_OK;
}

int encode_blocks_3d(CUtensorMap* map, const float* base, long long rows, long long cols, long long pitch_elems, int box_rows, int blocks) {
  int rc = load_driver_entry_points();
  if (rc) return rc;
  cuuint64_t dims[3] = {32, (cuuint64_t)rows, (cuuint64_t)(cols / 32)};
  cuuint64_t strides[2] = {(cuuint64_t)pitch_elems * 4, 128};
  cuuint32_t box[3] = {32, (cuuint32_t)box_rows, (cuuint32_t)blocks};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = g_encode_tiled(map, tma_dtype(), 3, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeTiled (blocks) failed (%d) rows=%lld cols=%lld pitch=%lld box=%d blocks=%d", (int)r, rows, cols, pitch_elems, box_rows, blocks);
  return MTB_OK;
}

int encode_rows_4d(CUtensorMap* map, const float* base, int n, int h, int w, int c, int channels, int box_w, bool mn_major) {
  int rc = load_driver_entry_points();
  if (rc) return rc;
  cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
  cuuint64_t strides[3] = {(cuuint64_t)c * 4, (cuuint64_t)w * c * 4, (cuuint64_t)h * w * c * 4};
  cuuint32_t box[4] = {(cuuint32_t)channels, (cuuint32_t)box_w, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode_tiled(map, tma_dtype(), 4, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeTiled (rows) failed (%d) n=%d h=%d w=%d c=%d box_w=%d", (int)r, n, h, w, c, box_w);
  return MTB_OK;
}

int encode_im2col_4d(CUtensorMap* map, const float* base, int n, int h, int w, int c, int lower_w, int lower_h, int upper_w, int upper_h,
                     int stride_w, int stride_h, int channels, int pixels, bool mn_major) {
  int rc = load_driver_entry_points();
  if (rc) return rc;
  cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
  cuuint64_t strides[3] = {(cuuint64_t)c * 4, (cuuint64_t)w * c * 4, (cuuint64_t)h * w * c * 4};
  int lower[2] = {lower_w, lower_h};
  int upper[2] = {upper_w, upper_h};
  cuuint32_t estr[4] = {1, (cuuint32_t)stride_w, (cuuint32_t)stride_h, 1};
  CUresult r = g_encode_im2col(map, tma_dtype(), 4, const_cast<float*>(base), dims, strides, lower, upper,
                               (cuuint32_t)channels, (cuuint32_t)pixels, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return mtb_fail(MTB_ERR_CUDA, "cuTensorMapEncodeIm2col failed (%d) n=%d h=%d w=%d c=%d lower=(%d,%d) upper=(%d,%d) stride=(%d,%d)", (int)r, n,
                    h, w, c, lower_w, lower_h, upper_w, upper_h, stride_w, stride_h);
  return MTB_OK;
}

}  // namespace tc

namespace {
using namespace tc;

enum { A_KMAJOR = 0, A_MNMAJOR = 1, A_IM2COL = 2 };
enum { B_KMAJOR = 0, B_MNMAJOR = 1 };

struct GemmParams {
  int M, N;
  int num_kb;  // reduction blocks of 32
  int m_tiles, n_tiles;
  float* out;
  long long ldo;
  const float* bias;
  // optional tensor laid out like `out`: out = result + addend (gradient accumulation).  May be `out` itself: a
  // thread reads the very elements it then writes.
  const float* addend;
  MtbBnEval bn;  // EPI_BN
  int relu;
  // geometry of the im2col'ed tensor (A operand of a convolution)
  int OW, OH, SW, SH, PW, PH, KW, KH, cchunks;
  // MN-major operands through one copy per reduction block (encode_blocks_3d) instead of one per 32 columns
  int a_blocks, b_blocks;
  // B operand addressed per filter tap (data gradient: weights read in place).  When set, the
  // k-block (tap, cc) reads B at inner coordinate b_tap_x[tap] + n0 (+32j), outer cc*32.
  int b_per_tap;
  int b_tap_x[64];
  // Output rows are pixels of a strided sub-grid of an [N, o_H, o_W, ldo] tensor: row
  // (n, i, j) of an o_Hc x o_Wc grid lands on pixel (o_h0 + o_sh*i, o_w0 + o_sw*j).
  int o_strided, o_Hc, o_Wc, o_H, o_W, o_h0, o_w0, o_sh, o_sw;
  // STATS kernels only: partial rows [(blockIdx.x / n_tiles) * 4 + epilogue warp][3][N] of per-column
  // (count, mean, M2) over the output rows this CTA produced (the grid is a multiple of n_tiles, so a
  // CTA always works on the same column tile)
  float* stats;
  // Split reduction (splits > 1): unit u = tile * splits + split works on reduction blocks [split * kb_per_split, ...).  The
  // units of a tile form a cluster.  When its accumulators are complete every unit hands each of the others the columns
  // that one finishes (distributed shared memory), and adds what it received to its own in split order.
  int splits, kb_per_split;
  float* pre;  // EPI_PRE: laid out like `out`, takes the result before the ReLU
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_address(uint32_t smem, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_cluster4(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void st_shared4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float ld_shared1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_shared4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// A stage holds kKB reduction blocks of 32 (each one 128-byte swizzle span per operand row).  One
// producer/consumer hand-over costs the issuing thread 300-400 cycles that do not overlap with MMA
// work, and four MMAs of a narrow tile are only 192-256 cycles of work, so tiles up to 128 wide
// take two blocks (8 MMAs) per stage.
//
// Tiles of 64 x 32 and 32 x 16 are for products with few outputs and a long reduction (the classifier of a small network),
// which have nothing but the rate at which an SM loads its operands (84 GB/s) to go by: A comes in boxes of as many rows as the
// tile has (the MMA's rows behind them read what lies there and are never stored) and a stage takes four blocks or eight.  The sum of an
// output is the same whatever the tile.  64 x 128, K = 9216: 53 us in tiles
// of 128 x 64, 40 in 64 x 32, 35 in 32 x 16 with eight blocks a stage (40 with four: a hand-over costs 350 cycles, a block of four
// MMAs 170); 512 x 512, K = 4000: 26.6 -> 20.5 us in 64 x 32.
template <int BN>
struct Cfg {
  static constexpr int kKB = BN == 16 ? 8 : BN == 32 ? 4 : BN <= 128 ? 2 : 1;
  static constexpr int kStages = BN == 256 ? 4 : (BN == 128 ? 3 : 4);
  static constexpr int kRowsA = BN == 16 ? 32 : BN == 32 ? 64 : 128;  // rows of the tile
  static constexpr int kAccCols = BN < 32 ? 32 : BN;                  // of one accumulator (read in 32 columns)
  static constexpr uint32_t kABytes = kRowsA * 32 * 4;   // one reduction block of A
  static constexpr uint32_t kBBytes = BN * 32 * 4;    // one reduction block of B
  static constexpr uint32_t kStageBytes = kKB * (kABytes + kBBytes);  // [A blocks][B blocks]
  static constexpr uint32_t kTmemCols = 2 * kAccCols;
};

// What the epilogue does beside bias / ReLU / store: nothing, BatchNorm statistics of the output, add a tensor, BatchNorm
// with running statistics (then optionally add a tensor), or store the result before the ReLU too (dense products).
enum { EPI_PLAIN = 0, EPI_STATS = 1, EPI_ADD = 2, EPI_BN = 3, EPI_PRE = 4 };

constexpr int kEpilogueWarps = 8, kGemmThreads = 64 + 32 * kEpilogueWarps;

// Shared memory: the stages, then what the epilogue warps hand to the copy engine, in blocks of 32 rows x 32 columns (128-byte
// swizzle): one block per warp, two where a tensor is added (one arrives while the other is being stored).  Those kernels are
// bound by what the epilogue moves, not by the main loop, and keep fewer stages: what they leave of the SM's shared memory is
// where BatchNorm's partial sums and the weight gradients' reductions of the side stream run beside them (ResNet-50 step, 128
// images, with two stages for additions 19.24 ms, with three 19.36).  Statistics want the depth: 256-wide tiles with four stages
// 19.23 ms, with three 19.33; the 7x7 stem's 64-wide ones 198 us and 204, and 212 with three and a second block per warp.
constexpr uint32_t kOutBlock = 32 * 32 * 4;
template <int BN, int EPI, bool BULK>
struct GemmSmem {
  static constexpr int kOutBlocks = !BULK ? 0 : EPI == EPI_ADD ? 2 : 1;  // per warp
  static constexpr int kStages = !BULK ? Cfg<BN>::kStages : EPI == EPI_ADD ? 2 : EPI == EPI_STATS ? (BN == 128 ? 3 : 4) : (BN == 128 ? 2 : 3);
  static constexpr uint32_t kBytes = kStages * Cfg<BN>::kStageBytes + kEpilogueWarps * kOutBlocks * kOutBlock + 1024;  // + alignment slack
  static_assert(kBytes <= 227 * 1024);
  static_assert((Cfg<BN>::kKB - 1) * Cfg<BN>::kABytes + 128 * 128 <= Cfg<BN>::kStageBytes);  // the MMA reads 128 rows of A, behind the last box of few rows blocks of B
};

// Tensor maps of what the epilogue moves by bulk copies: the result, and what is added to it.
template <int N>
struct BulkMaps {
  CUtensorMap map[N];
};
template <>
struct BulkMaps<0> {};
template <int EPI, bool BULK>
using BulkMapsOf = BulkMaps<!BULK ? 0 : EPI == EPI_ADD ? 2 : 1>;

// SPLIT: GemmParams::splits > 1, a kernel of its own because the exchange takes the registers that the other epilogues need.
// BULK: results (and the addend) move through shared memory by bulk copies, for rows that lie one after the other.  Kernels of
// their own, too: with the depth of the ring a parameter of the launch and two more maps in every launch, those that
// move nothing in bulk took 0.3 to 0.45 us longer (256 -> 256 data gradient on 128 x 8x8 21.85 -> 22.20 us, 512 -> 512
// on 4x4 22.82 -> 23.19, a weight product of 8192 x 2000 x 480 87.4 -> 88.7).
template <int BN, int AMODE, int BMODE, int EPI, bool SPLIT, bool BULK>
__global__ void __launch_bounds__(kGemmThreads, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const GemmParams p,
               const __grid_constant__ BulkMapsOf<EPI, BULK> bulk) {
  static_assert(!BULK || (!SPLIT && BN >= 64 && EPI != EPI_BN && EPI != EPI_PRE));
  using C = Cfg<BN>;
  using Smem = GemmSmem<BN, EPI, BULK>;
  constexpr int STAGES = Smem::kStages;
  constexpr bool STATS = EPI == EPI_STATS, BNORM = EPI == EPI_BN, ADD = EPI == EPI_ADD || BNORM;
  constexpr bool PRE = EPI == EPI_PRE;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[8], bar_empty[8], bar_tfull[2], bar_tempty[2];
  __shared__ uint64_t bar_add[BULK && EPI == EPI_ADD ? kEpilogueWarps : 1][2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ alignas(16) BnColumns<BNORM ? BN : 4> bn_columns;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_tfull[b]), 1);
      mbar_init(smem_u32(&bar_tempty[b]), kEpilogueWarps);  // one arrival per epilogue warp
      if constexpr (BULK && EPI == EPI_ADD)
        for (int w = 0; w < kEpilogueWarps; ++w) mbar_init(smem_u32(&bar_add[w][b]), 1);
    }
    abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  mtb_wait_prior();  // everything above overlaps the end of the kernel before
  if constexpr (BNORM) load_bn_columns<BN>(bn_columns, p.bn, (blockIdx.x / p.splits) % p.n_tiles * BN, p.N);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const int S = SPLIT ? p.splits : 1;
  const int tiles = p.m_tiles * p.n_tiles * S;  // work units: (tile, split) pairs, the splits of a tile adjacent
  volatile int* abort_ptr = &abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < tiles && ok; unit += gridDim.x) {
        const int tile = unit / S, split = unit - tile * S;
        const int kb0 = split * p.kb_per_split;
        const int kb1 = kb0 + p.kb_per_split < p.num_kb ? kb0 + p.kb_per_split : p.num_kb;
        const int m0 = (tile / p.n_tiles) * C::kRowsA, n0 = (tile % p.n_tiles) * BN;
        int pix_w = 0, pix_h = 0, pix_n = 0;
        if (AMODE == A_IM2COL) {
          int ow = m0 % p.OW, t = m0 / p.OW;
          pix_w = ow * p.SW - p.PW;
          pix_h = (t % p.OH) * p.SH - p.PH;
          pix_n = t / p.OH;
        }
        // reduction blocks in (tap, channel-block) order; plain GEMMs have a single "tap"
        int cc = kb0 % p.cchunks, kw = (kb0 / p.cchunks) % p.KW, kh = (kb0 / p.cchunks) / p.KW;
        for (int kb = kb0; kb < kb1 && ok; kb += C::kKB) {
          const int nblk = kb1 - kb < C::kKB ? kb1 - kb : C::kKB;  // the last stage may hold one block
          if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr, 1)) { ok = false; break; }
          const uint32_t full = smem_u32(&bar_full[stage]);
          mbar_expect_tx(full, (uint32_t)nblk * (C::kABytes + C::kBBytes));
          const uint32_t st_base = smem_base + stage * C::kStageBytes;
          for (int h = 0; h < nblk; ++h) {
            const int kbh = kb + h;
            const int tap = kh * p.KW + kw;
            const uint32_t a_dst = st_base + h * C::kABytes, b_dst = st_base + C::kKB * C::kABytes + h * C::kBBytes;
            if (AMODE == A_KMAJOR) {
              tma_load_2d(a_dst, &mapA, full, kbh * 32, m0);
            } else if (AMODE == A_MNMAJOR) {
              if (p.a_blocks) {
                tma_load_3d(a_dst, &mapA, full, 0, kbh * 32, m0 / 32);
              } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) tma_load_2d(a_dst + j * 4096, &mapA, full, m0 + 32 * j, kbh * 32);
              }
            } else {
              tma_load_im2col_4d(a_dst, &mapA, full, cc * 32, pix_w, pix_h, pix_n, (uint16_t)kw, (uint16_t)kh);
            }
            if (BMODE == B_KMAJOR) {
              tma_load_2d(b_dst, &mapB, full, kbh * 32, n0);
            } else {
              int bx = n0, by = kbh * 32;
              if (p.b_per_tap) { bx = p.b_tap_x[tap] + n0; by = cc * 32; }
              if (p.b_blocks) {
                tma_load_3d(b_dst, &mapB, full, 0, by, bx / 32);
              } else {
#pragma unroll
                for (int j = 0; j < BN / 32; ++j) tma_load_2d(b_dst + j * 4096, &mapB, full, bx + 32 * j, by);
              }
            }
            if (++cc == p.cchunks) {
              cc = 0;
              if (++kw == p.KW) { kw = 0; ++kh; }
            }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
    if constexpr (SPLIT) { cluster_arrive(); cluster_wait(); cluster_arrive(); cluster_wait(); }  // see the epilogue
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp runs the loop converged and one elected lane issues (warp-uniform control
    // flow keeps the descriptors in uniform registers: a lane-0 branch around the loop costs
    // about twice as many cycles per tcgen05.mma).
    constexpr uint32_t idesc = idesc_tf32(128, BN, AMODE == A_MNMAJOR ? 1 : 0, BMODE == B_MNMAJOR ? 1 : 0);
    constexpr uint32_t a_hi = AMODE == A_MNMAJOR ? desc_hi_mnmajor() : desc_hi_kmajor();
    constexpr uint32_t b_hi = BMODE == B_MNMAJOR ? desc_hi_mnmajor() : desc_hi_kmajor();
    constexpr uint32_t a_step = AMODE == A_MNMAJOR ? (1024u >> 4) : (32u >> 4);  // per 8 of K, in 16-byte units
    constexpr uint32_t b_step = BMODE == B_MNMAJOR ? (1024u >> 4) : (32u >> 4);
    const uint32_t a_lo0 = AMODE == A_MNMAJOR ? desc_lo_mnmajor(smem_base) : desc_lo_kmajor(smem_base);
    const uint32_t b_lo0 = BMODE == B_MNMAJOR ? desc_lo_mnmajor(smem_base + C::kKB * C::kABytes) : desc_lo_kmajor(smem_base + C::kKB * C::kABytes);
    int stage = 0;
    uint32_t phase = 0;
    int t = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < tiles && ok; unit += gridDim.x, ++t) {
      const int split = unit % S;
      const int kb0 = split * p.kb_per_split;
      const int kb1 = kb0 + p.kb_per_split < p.num_kb ? kb0 + p.kb_per_split : p.num_kb;
      const int buf = t & 1;
      const uint32_t use = (uint32_t)(t >> 1);
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_tempty[buf]), (use & 1u) ^ 1u, abort_ptr, 2));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * C::kAccCols;
      uint32_t acc = 0;
      for (int kb = kb0; kb < kb1; kb += C::kKB) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[stage]), phase, abort_ptr, 3));
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_lo = a_lo0 + stage * (C::kStageBytes >> 4), b_lo = b_lo0 + stage * (C::kStageBytes >> 4);
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < C::kKB; ++h) {
            if (h > 0 && kb + h >= kb1) break;
            const uint32_t a = a_lo + h * (C::kABytes >> 4), b = b_lo + h * (C::kBBytes >> 4);
            mma_tf32_words(d_tmem, a, a_hi, b, b_hi, idesc, h == 0 ? acc : 1u);
            mma_tf32_words(d_tmem, a + a_step, a_hi, b + b_step, b_hi, idesc, 1u);
            mma_tf32_words(d_tmem, a + 2 * a_step, a_hi, b + 2 * b_step, b_hi, idesc, 1u);
            mma_tf32_words(d_tmem, a + 3 * a_step, a_hi, b + 3 * b_step, b_hi, idesc, 1u);
          }
          mma_commit(smem_u32(&bar_empty[stage]));
        }
        __syncwarp();
        acc = 1u;
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (ok && elect_one()) mma_commit(smem_u32(&bar_tfull[buf]));
      __syncwarp();
    }
    if constexpr (SPLIT) { cluster_arrive(); cluster_wait(); cluster_arrive(); cluster_wait(); }  // see the epilogue
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int quarter = warp & 3;
    // columns of the tile this warp finishes: half of the tile, from c_first on, or its share of the columns of its unit
    constexpr int COLS = BN >= 64 ? BN / 2 : 32;
    const int cols_here = BN < 64 && (warp >= 6 || (warp & 3) * 32 >= C::kRowsA) ? 0 : COLS;  // a narrow tile has work for one or two of the warps
    const int rank = SPLIT ? (int)(blockIdx.x % S) : 0, width = BN / S;
    const int c_first = !SPLIT ? (warp < 6 ? 0 : COLS) : rank * width + (width >= 64 && warp >= 6 ? width / 2 : 0);
    const int split_chunks = width >= 64 ? width / 64 : (warp < 6 ? 1 : 0);
    int t = 0;
    const uintptr_t results = reinterpret_cast<uintptr_t>(p.out) | (PRE ? reinterpret_cast<uintptr_t>(p.pre) : 0);
    const bool vec_ok = (p.ldo % 4 == 0) && (((results | reinterpret_cast<uintptr_t>(p.bias)) & 15u) == 0);
    const bool wide_ok = vec_ok && (p.ldo % 8 == 0) && ((results & 31u) == 0);  // 32-byte stores
    // statistics of a split reduction: narrow tiles keep per-lane sums, wide tiles merge per tile
    constexpr bool LANE_SUMS = STATS && SPLIT && BN == 64;
    WarpColStats<(STATS && !LANE_SUMS) ? COLS / 32 : 1> stats;
    LaneColSums<LANE_SUMS ? COLS / 32 : 1> sums;
    if constexpr (LANE_SUMS) sums.reset(); else stats.reset();
    if constexpr (BULK) {
      // Results through shared memory and the copy engine.  A lane holds a row of the accumulator; stored from registers
      // every store instruction touches 32 lines (64 passes through the L1, which was 84 to 96 % busy and bounded every
      // convolution with a short reduction), as blocks of 32 x 32 in shared memory eight conflict-free stores and one copy do.
      // What is to be added arrives the same way, one block ahead.  Statistics read the block by columns: a lane has the 32
      // values of its column in registers, without a single exchange between lanes.
      constexpr int OUT_BLOCKS = Smem::kOutBlocks;
      const int ew = warp - 2;
      const uint32_t blocks = smem_base + STAGES * C::kStageBytes + (uint32_t)(ew * OUT_BLOCKS) * kOutBlock;
      const uint32_t row_base = (uint32_t)lane * 128u, swz = (uint32_t)(lane & 7);
      // blocks of this warp in order: (tile, 32 columns); those outside the matrix are skipped
      auto next_block = [&](int& unit, int& c0) {
        do {
          c0 += 32;
          if (c0 >= COLS) { c0 = 0; unit += gridDim.x; }
        } while (unit < tiles && ((unit / p.n_tiles) * 128 + quarter * 32 >= p.M || (unit % p.n_tiles) * BN + c_first + c0 >= p.N));
      };
      int load_unit = blockIdx.x, load_c0 = -32, loaded = 0;  // the addend's blocks, asked for one ahead
      auto load_addend = [&]() {  // lane 0
        next_block(load_unit, load_c0);
        if (load_unit >= tiles) return;
        const uint32_t bar = smem_u32(&bar_add[ew][loaded & 1]);
        mbar_expect_tx(bar, kOutBlock);
        tma_load_2d(blocks + (uint32_t)(loaded & 1) * kOutBlock, &bulk.map[EPI == EPI_ADD ? 1 : 0], bar, (load_unit % p.n_tiles) * BN + c_first + load_c0,
                    (load_unit / p.n_tiles) * 128 + quarter * 32);
        ++loaded;
      };
      if constexpr (EPI == EPI_ADD) {
        if (lane == 0) load_addend();
      }
      int g = 0;  // blocks handled
      for (int unit = blockIdx.x; unit < tiles; unit += gridDim.x, ++t) {
        const int row0 = (unit / p.n_tiles) * 128 + quarter * 32, n0 = (unit % p.n_tiles) * BN + c_first;
        const int buf = t & 1;
        bool ok = lane != 0 || mbar_wait(smem_u32(&bar_tfull[buf]), (uint32_t)(t >> 1) & 1u, abort_ptr, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const int rows = p.M - row0 < 32 ? p.M - row0 : 32;
#pragma unroll
        for (int c0 = 0; c0 < COLS; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c_first + c0), r);
          const int col0 = n0 + c0;
          const bool inside = rows > 0 && col0 < p.N;  // warp-uniform
          const uint32_t block = blocks + (uint32_t)(OUT_BLOCKS == 2 ? (g & 1) : 0) * kOutBlock;
          float4 add[8];
          if constexpr (EPI == EPI_ADD) {
            if (inside) {
              ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_add[ew][g & 1]), (uint32_t)(g >> 1) & 1u, abort_ptr, 5));
              if (!ok) break;
#pragma unroll
              for (int j = 0; j < 8; ++j) add[j] = ld_shared4(block + row_base + (((uint32_t)j ^ swz) << 4));
              if (lane == 0) {
                bulk_wait_read<0>();  // the block before has been read, its place is free
                load_addend();
              }
            }
          } else {
            if (inside) {
              if (lane == 0) bulk_wait_read<0>();  // the block before has been read
              __syncwarp();
            }
          }
          tmem_ld_wait();
          if (c0 + 32 >= COLS) {  // the accumulator is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[buf]));
          }
          if (!inside) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 v = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
            if (p.bias && col0 + 4 * j < p.N) {  // N % 4 == 0 on this path
              const float4 b = *reinterpret_cast<const float4*>(p.bias + col0 + 4 * j);
              v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
            }
            if constexpr (EPI == EPI_ADD) { v.x += add[j].x; v.y += add[j].y; v.z += add[j].z; v.w += add[j].w; }
            if (p.relu) { v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f); }
            st_shared4(block + row_base + (((uint32_t)j ^ swz) << 4), v);
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&bulk.map[0], block, col0, row0);
            bulk_commit();
          }
          ++g;
          if constexpr (STATS) {
            float o[32];
            const uint32_t column = block + (uint32_t)(lane & 3) * 4u;
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = ld_shared1(column + (uint32_t)k * 128u + (((uint32_t)(lane >> 2) ^ (uint32_t)(k & 7)) << 4));
            stats.add_column(c0 / 32, o, rows);
          }
        }
        if (!ok) break;
        if constexpr (STATS) { if (rows > 0) stats.n += (float)rows; }
      }
      if (lane == 0) bulk_wait_all();
    }
    if constexpr (!BULK) {
    for (int unit = blockIdx.x; unit < tiles; unit += gridDim.x, ++t) {
      const int tile = unit / S;
      const int m0 = (tile / p.n_tiles) * C::kRowsA, n0 = (tile % p.n_tiles) * BN;
      const int col_end = BN >= 32 || n0 + BN > p.N ? p.N : n0 + BN;
      const int buf = t & 1;
      const uint32_t use = (uint32_t)(t >> 1);
      // one lane polls (128 threads spinning on the barrier slow the other roles' barrier traffic down)
      auto wait_for_accumulator = [&]() {
        bool ok = lane != 0 || mbar_wait(smem_u32(&bar_tfull[buf]), use & 1u, abort_ptr, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) tc_fence_after();
        return ok;
      };
      if constexpr (!ADD) {
        if (!SPLIT && !wait_for_accumulator()) break;
      }
      const int row = m0 + quarter * 32 + lane;
      long long orow_index = row;
      if (p.o_strided && row < p.M) {
        const int j = row % p.o_Wc, t2 = row / p.o_Wc;
        const int i = t2 % p.o_Hc, nn = t2 / p.o_Hc;
        orow_index = ((long long)nn * p.o_H + p.o_h0 + p.o_sh * i) * p.o_W + p.o_w0 + p.o_sw * j;
      }
      float* orow = p.out + orow_index * p.ldo;
      const float* arow = ADD && (!BNORM || p.addend) ? p.addend + orow_index * p.ldo : nullptr;
      const bool valid = row < p.M;
      const float cnt = STATS ? (float)__popc(__ballot_sync(0xffffffffu, valid)) : 0.f;
      // r: this lane's row of the finished accumulator, columns c0 .. c0+31 of the warp's half; add: the same columns of the
      // addend, fetched one chunk ahead (a memory round trip per chunk in front of the stores would make the epilogue
      // of a short reduction several times longer than its main loop)
      const bool adds = ADD && arow && valid && vec_ok && n0 + BN <= p.N;
      auto fetch_addend = [&](int c0, float4 (&add)[8]) {
        if (adds) {
#pragma unroll
          for (int j = 0; j < 8; ++j) add[j] = *reinterpret_cast<const float4*>(arow + n0 + c_first + c0 + 4 * j);
        }
      };
      float4 add[8];
      if constexpr (ADD) {
        fetch_addend(0, add);
        if (!SPLIT && !wait_for_accumulator()) break;
      }
      auto finish = [&](int c0, const uint32_t (&r)[32]) {
        const int col0 = n0 + c_first + c0;
        if constexpr (STATS) {
          // the forward convolution that feeds a BatchNorm layer: full column tiles (N % 32 == 0, checked on
          // the host), vector stores, and the per-channel statistics of what is stored
          if (col0 < p.N) {  // warp-uniform
            float o[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __uint_as_float(r[j]) + (p.bias ? __ldg(p.bias + col0 + j) : 0.f);
            if (valid) {
#pragma unroll
              for (int j = 0; j < 32; j += 8)
                st_row8(orow + col0 + j, make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]), make_float4(o[j + 4], o[j + 5], o[j + 6], o[j + 7]), wide_ok);
            }
            if constexpr (LANE_SUMS) {
              if (valid) sums.add_chunk(c0 / 32, r);
            } else {
              if (cnt > 0.f) stats.add_chunk(c0 / 32, o, valid, cnt, lane);
            }
          }
        } else {
          if (valid && col0 < col_end) {
            if (vec_ok && col0 + 32 <= col_end) {
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                float4 v[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const int jj = j + 4 * h;
                  v[h] = make_float4(__uint_as_float(r[jj]), __uint_as_float(r[jj + 1]), __uint_as_float(r[jj + 2]), __uint_as_float(r[jj + 3]));
                  if (p.bias) {
                    const float4 b = *reinterpret_cast<const float4*>(p.bias + col0 + jj);
                    v[h].x += b.x; v[h].y += b.y; v[h].z += b.z; v[h].w += b.w;
                  }
                  if constexpr (BNORM) {
                    const float4 mu = *reinterpret_cast<const float4*>(&bn_columns.mean[c_first + c0 + jj]);
                    const float4 g = *reinterpret_cast<const float4*>(&bn_columns.scale[c_first + c0 + jj]);
                    const float4 b = *reinterpret_cast<const float4*>(&bn_columns.beta[c_first + c0 + jj]);
                    v[h].x = (v[h].x - mu.x) * g.x + b.x; v[h].y = (v[h].y - mu.y) * g.y + b.y;
                    v[h].z = (v[h].z - mu.z) * g.z + b.z; v[h].w = (v[h].w - mu.w) * g.w + b.w;
                  }
                  if (ADD && arow) {
                    const float4 b = adds ? add[jj / 4] : *reinterpret_cast<const float4*>(arow + col0 + jj);
                    v[h].x += b.x; v[h].y += b.y; v[h].z += b.z; v[h].w += b.w;
                  }
                  if constexpr (!PRE) {
                    if (p.relu) { v[h].x = fmaxf(v[h].x, 0.f); v[h].y = fmaxf(v[h].y, 0.f); v[h].z = fmaxf(v[h].z, 0.f); v[h].w = fmaxf(v[h].w, 0.f); }
                  }
                }
                if constexpr (PRE) {
                  st_row8(p.pre + orow_index * p.ldo + col0 + j, v[0], v[1], wide_ok);
                  if (p.relu) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) { v[h].x = fmaxf(v[h].x, 0.f); v[h].y = fmaxf(v[h].y, 0.f); v[h].z = fmaxf(v[h].z, 0.f); v[h].w = fmaxf(v[h].w, 0.f); }
                  }
                }
                st_row8(orow + col0 + j, v[0], v[1], wide_ok);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (col0 + j < col_end) {
                  float v = __uint_as_float(r[j]);
                  if (p.bias) v += p.bias[col0 + j];
                  if constexpr (BNORM) v = (v - bn_columns.mean[c_first + c0 + j]) * bn_columns.scale[c_first + c0 + j] + bn_columns.beta[c_first + c0 + j];
                  if (ADD && arow) v += arow[col0 + j];
                  if constexpr (PRE) p.pre[orow_index * p.ldo + col0 + j] = v;
                  if (p.relu) v = fmaxf(v, 0.f);
                  orow[col0 + j] = v;
                }
              }
            }
          }
        }
      };
      auto release_accumulator = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[buf]));
      };
      auto count_rows = [&]() {
        if constexpr (LANE_SUMS) sums.cnt += valid ? 1.f : 0.f;
        else if constexpr (STATS) stats.n += cnt;
      };
      if constexpr (!SPLIT) {
#pragma unroll 1
        for (int c0 = 0; c0 < cols_here; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * C::kAccCols + c_first + c0), r);
          if constexpr (ADD) {
            float4 next[8];
            if (c0 + 32 < COLS) fetch_addend(c0 + 32, next);
            tmem_ld_wait();
            finish(c0, r);
#pragma unroll
            for (int j = 0; j < 8; ++j) add[j] = next[j];
          } else {
            tmem_ld_wait();
            finish(c0, r);
          }
        }
        release_accumulator();
      } else {
      // Split reduction (one unit per CTA).  The stages are free when every unit of the cluster has its accumulator; received
      // columns lie there as [sender][column / 4][row] float4, so that a warp writes and reads 512 contiguous bytes.  The
      // exchange takes 1.1 to 2 us (64 to 256 columns); through bulk copies instead of stores it took the same.
      const bool complete = wait_for_accumulator();  // a unit that gave up still takes part in the barriers
      cluster_arrive();
      cluster_wait();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN);
      const uint32_t row16 = (uint32_t)(quarter * 32 + lane) * 16u;
#pragma unroll 2
      for (int c0 = warp < 6 ? 0 : 32; c0 < BN; c0 += 64) {  // the two warps of a row quarter take turns: equal shares for every rank
        const int owner = c0 / width;
        if (owner == rank) continue;
        uint32_t r[32];
        tmem_ld_32x32(taddr + (uint32_t)c0, r);
        tmem_ld_wait();
        const uint32_t slot = (uint32_t)((rank < owner ? rank : rank - 1) * (width / 4) + (c0 - owner * width) / 4);
        const uint32_t dst = cluster_address(smem_base + slot * 2048u + row16, (uint32_t)owner);
#pragma unroll
        for (int j = 0; j < 32; j += 4) st_cluster4(dst + (uint32_t)(j / 4) * 2048u, r[j], r[j + 1], r[j + 2], r[j + 3]);
      }
      cluster_arrive();
      cluster_wait();
      auto reduce_chunk = [&](int c, uint32_t (&r)[32]) {
        tmem_ld_32x32(taddr + (uint32_t)(c_first + c * 32), r);
        tmem_ld_wait();
        const uint32_t src = smem_base + (uint32_t)((c_first - rank * width) / 4 + c * 8) * 2048u + row16;
        float acc[32];
        for (int sp = 0; sp < S; ++sp) {  // fixed order: split 0, 1, 2, ...
          const uint32_t q = src + (uint32_t)((sp < rank ? sp : sp - 1) * (width / 4)) * 2048u;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 v = sp == rank ? make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]))
                                        : ld_shared4(q + (uint32_t)(j / 4) * 2048u);
            if (sp == 0) { acc[j] = v.x; acc[j + 1] = v.y; acc[j + 2] = v.z; acc[j + 3] = v.w; }
            else { acc[j] += v.x; acc[j + 1] += v.y; acc[j + 2] += v.z; acc[j + 3] += v.w; }
          }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(acc[j]);
      };
#pragma unroll (STATS ? COLS / 32 : 1)
      for (int c = 0; c < COLS / 32; ++c) {
        if (c >= split_chunks || !complete) break;
        uint32_t r[32];
        if constexpr (ADD) {
          if (c > 0) fetch_addend(c * 32, add);
        }
        reduce_chunk(c, r);
        finish(c * 32, r);
      }
      count_rows();
      if constexpr (STATS) {
        float* row = p.stats + ((long long)(tile / p.n_tiles) * 4 + quarter) * 3 * p.N;
        const int end = n0 + c_first + 32 * split_chunks < p.N ? n0 + c_first + 32 * split_chunks : p.N;
        if constexpr (LANE_SUMS) sums.store(row, p.N, n0 + c_first, end, p.bias, lane);
        else stats.store(row, p.N, n0 + c_first, end, lane);
      }
      }
    }
    }
    if constexpr (STATS && !SPLIT)
      stats.store(p.stats + ((long long)(blockIdx.x / p.n_tiles) * 4 + quarter) * 3 * p.N, p.N, (blockIdx.x % p.n_tiles) * BN + c_first, p.N, lane);
  }

  // ------------------------------------------------------------ teardown
  mtb_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    // give copies that are still in flight time to land before the CTA's shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// From how many reduction blocks on results are stored from registers.  Times through shared memory over times from registers,
// means over 1279 products of 1,000 to 200,000 rows and 32 to 9,216 columns (tiles of 64 / 128 / 256 columns):
//   with addition, one wave of tiles    4 blocks 1.02 / 0.83 / 0.72   8: 1.04 / 0.85 / 0.78   16: 1.00 / 0.87 / 0.88   32: 1.00 / 0.92 / 1.06
//   with addition, more                 4 blocks 0.82 / 0.65 / 0.67   8: 1.00 / 0.78 / 0.77   16: 1.08 / 0.96 / 1.06   32: 1.17 / 1.11 / 1.42
//   plain, one wave                     2 blocks 1.00 / 0.98 / 0.9    4: 1.01 / 0.98 / 0.88    7: 1.03 / 0.99 / 0.88
//   plain, more                         2 blocks 0.95 / 0.86 / 0.79   4: 0.97 / 0.88 / 0.83    7: 1.06 / 1.07 / 0.90
// 512 <- 1024 channels with addition on 32 x 28x28: 54.8 us from registers, 78.2 through shared memory with two stages.  Rows that
// are no whole sectors of 32 bytes are stored 16 bytes at a time from registers (1000 x 500, 4 blocks: 5.8 us, 4.8).
int bulk_limit(int bn, bool adds, bool one_wave, bool whole_sectors) {
  if (bn == 64) return !whole_sectors ? 8 : one_wave ? 0 : adds ? 8 : 5;
  if (adds) return !one_wave ? 16 : bn == 128 ? 40 : 32;
  return bn == 128 && whole_sectors ? 6 : 8;
}

template <int BN, int AMODE, int BMODE, int EPI, bool BULK>
int launch_tc_whole(const CUtensorMap& mapA, const CUtensorMap& mapB, const GemmParams& p, const BulkMapsOf<EPI, BULK>& bulk, cudaStream_t st) {
  auto kernel = tc_gemm_kernel<BN, AMODE, BMODE, EPI, false, BULK>;
  constexpr uint32_t smem = GemmSmem<BN, EPI, BULK>::kBytes;
  static unsigned long long configured = 0;
  if (int rc = mtb_opt_in_smem((const void*)kernel, (int)smem, &configured)) return rc;
  const int tiles = p.m_tiles * p.n_tiles;
  int grid = tiles < mtb_sm_count() ? tiles : mtb_sm_count();
  if (EPI == EPI_STATS || EPI == EPI_BN) grid = grid / p.n_tiles * p.n_tiles;  // every CTA stays on one column tile (see GemmParams::stats)
  MTB_LAUNCH(kernel, dim3(grid), dim3(kGemmThreads), smem, st, mapA, mapB, p, bulk);
  MTB_LAUNCH_CHECK("tc_gemm_kernel");
  return MTB_OK;
}

template <int BN, int AMODE, int BMODE, int EPI = EPI_PLAIN>
int launch_tc(const CUtensorMap& mapA, const CUtensorMap& mapB, const GemmParams& p, cudaStream_t st) {
  if (p.splits > 1) {  // one unit per CTA, the units of a tile a cluster
    if constexpr (AMODE == A_IM2COL) {
      auto kernel = tc_gemm_kernel<BN, AMODE, BMODE, EPI, true, false>;
      constexpr uint32_t smem = GemmSmem<BN, EPI, false>::kBytes;
      static unsigned long long configured = 0;
      if (int rc = mtb_opt_in_smem((const void*)kernel, (int)smem, &configured)) return rc;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(p.m_tiles * p.n_tiles * p.splits);
      cfg.blockDim = dim3(kGemmThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)p.splits;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      MTB_CUDA(cudaLaunchKernelEx(&cfg, kernel, mapA, mapB, p, BulkMaps<0>{}));
      MTB_LAUNCH_CHECK("tc_gemm_kernel");
      return MTB_OK;
    }
    return mtb_fail(MTB_ERR_INVALID, "tc_gemm: only convolutions split the reduction");
  }
  if constexpr (BN >= 64 && EPI != EPI_BN && EPI != EPI_PRE) {
    // Whole rows one after the other, their pitch and start on 16 bytes: what the copy engine asks for.  Everything else (a
    // residue class of a strided data gradient, odd widths) is stored from registers, and so are the results of long reductions,
    // whose stores hide behind the main loop, which wants the stages.
    const bool whole_sectors = p.ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31u) == 0;
    const bool fits = !p.o_strided && p.ldo % 4 == 0 && p.N % 4 == 0 && al16(p.out) && al16(p.bias) && al16(p.addend);
    if (fits && (EPI == EPI_STATS || p.num_kb < bulk_limit(BN, EPI == EPI_ADD, p.m_tiles * p.n_tiles <= mtb_sm_count(), whole_sectors))) {
      BulkMapsOf<EPI, true> bulk;
      if (int rc = tc::encode_result_2d(&bulk.map[0], p.out, p.M, p.N, p.ldo)) return rc;
      if constexpr (EPI == EPI_ADD)
        if (int rc = tc::encode_result_2d(&bulk.map[1], p.addend, p.M, p.N, p.ldo)) return rc;
      return launch_tc_whole<BN, AMODE, BMODE, EPI, true>(mapA, mapB, p, bulk, st);
    }
  }
  if constexpr (EPI == EPI_STATS) return mtb_fail(MTB_ERR_INVALID, "tc_gemm: statistics need whole aligned rows");
  else return launch_tc_whole<BN, AMODE, BMODE, EPI, false>(mapA, mapB, p, {}, st);
}

// Partial-statistics rows the STATS variant writes for a problem of `tiles` tiles in `n_tiles` column tiles.
int stats_rows_for(int tiles, int n_tiles) {
  int grid = tiles < mtb_sm_count() ? tiles : mtb_sm_count();
  return grid / n_tiles * 4;
}

template <int AMODE, int BMODE, int EPI = EPI_PLAIN>
int launch_tc_bn(int bn, const CUtensorMap& mapA, const CUtensorMap& mapB, const GemmParams& p, cudaStream_t st) {
  if constexpr (AMODE == A_KMAJOR && BMODE == B_KMAJOR && (EPI == EPI_PLAIN || EPI == EPI_PRE)) {
    if (bn == 16) return launch_tc<16, AMODE, BMODE, EPI>(mapA, mapB, p, st);
    if (bn == 32) return launch_tc<32, AMODE, BMODE, EPI>(mapA, mapB, p, st);
  }
  if (bn == 64) return launch_tc<64, AMODE, BMODE, EPI>(mapA, mapB, p, st);
  if (bn == 128) return launch_tc<128, AMODE, BMODE, EPI>(mapA, mapB, p, st);
  return launch_tc<256, AMODE, BMODE, EPI>(mapA, mapB, p, st);
}

int pick_bn(int n) { return n <= 64 ? 64 : (n <= 128 ? 128 : 256); }

// Tile width of the row-staged kernels for `rows` output rows: the widest tile (best MMA efficiency) that still
// yields enough tiles to occupy most SMs; small problems (late layers at small batch) fall back
// to narrower tiles so that more CTAs take part.  A rule, not a price (the im2col kernel's width is priced: cheapest_bn);
// row_conv_pays then compares the price of the width it gives.
int pick_bn_for(int n, long long rows) {
  const long long m_tiles = (rows + 127) / 128;
  const int want = mtb_sm_count() * 3 / 4;
  int bn = pick_bn(n);
  while (bn > 64 && m_tiles * ((n + bn - 1) / bn) < want) bn >>= 1;
  return bn;
}

// One reduction block of 32 of a tile of 128 rows, in ns (see im2col_ns).
double kb_ns(int bn, bool mn_major) { return mn_major ? (bn == 64 ? 285 : bn == 128 ? 295 : 405) : (bn == 64 ? 232 : bn == 128 ? 262 : 376); }

// What a launch of the im2col kernel without split takes, in ns: waves x (reduction blocks x the time of one block + about
// 900 ns for filling the pipeline and the first stores).  The block times were measured (weights K-major in forward,
// MN-major in the data gradient; 72 blocks on 64 to 592 images of 8x8): a 64-wide tile is bound by the gather of 128
// pixel rows, a 256-wide one by the MMAs.  `copies` launches of this size share the GPU.
double im2col_ns(int bn, int n, long long rows, int num_kb, bool mn_major, int copies = 1) {
  const long long tiles = ((rows + 127) / 128) * ((n + bn - 1) / bn) * copies, waves = (tiles + mtb_sm_count() - 1) / mtb_sm_count();
  const double block = kb_ns(bn, mn_major);
  const double store = 8.0 * bn;  // a tile's epilogue: longer than the main loop of a short reduction
  return waves * ((num_kb * block > store ? num_kb * block : store) + 900.0) + store;
}

// The tile width with the least time: one more wave costs more than a narrower or wider tile gains (256 -> 256 channels on
// 100 images of 8x8: 200 tiles of 64 columns are two waves, 34 us; 100 tiles of 128 one, 23 us).
int cheapest_bn(int n, long long rows, int num_kb, bool mn_major, int copies = 1) {
  int best = pick_bn(n);
  for (int bn = best >> 1; bn >= 64; bn >>= 1)
    if (im2col_ns(bn, n, rows, num_kb, mn_major, copies) < im2col_ns(best, n, rows, num_kb, mn_major, copies)) best = bn;
  return best;
}

// CTAs of the widest kernel that the GPU holds at once in clusters of `size` (clusters do not span the GPU's partitions, so
// a few SMs stay without).
int cluster_units(int size) {
  static int units[9] = {};
  if (!units[size]) {
    const int sms = mtb_sm_count();
    auto kernel = tc_gemm_kernel<256, A_IM2COL, B_KMAJOR, EPI_PLAIN, true, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms / size * size);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = GemmSmem<256, EPI_PLAIN, false>::kBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmSmem<256, EPI_PLAIN, false>::kBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();  // no GPU (plans are also made without one)
      clusters = sms * 7 / 8 / size;
    }
    units[size] = clusters * size;
  }
  return units[size];
}

// Tile width and reduction split of the im2col kernel.  A layer with few pixels leaves most of the GPU idle on wide tiles and
// spends its time on loading the pixels again for every narrow one (kb_ns: a block of 32 takes 64 columns 232 ns, 256 columns 376),
// so its long reduction is split over a cluster of 2, 4 or 8 CTAs on wide tiles, one unit per CTA, as long as all units fit
// the GPU at once.  Times of a split launch as measured (512 -> 512 channels on 4x4, 16 to 128 images): base (launch, pipeline
// fill, exchange, epilogue) + blocks per unit x block time.  128 images, before -> now: forward 31 -> 22 us, data gradient
// 38.5 -> 23.5 us; 64 images (before: partial sums through global memory) 19.0 -> 15 and 21.4 -> 16.5 us; 256 -> 256 on 8x8,
// 64 images: 18.8 -> 14.5 and 22.6 -> 16 us.  Under 64 blocks the exchange costs what the split gains.  The block times fitted
// to these launches (180 / 200 / 280 ns) are a quarter below kb_ns, which was fitted to launches over larger images; what
// makes the difference was not looked into, so neither set should be used for the other kind of launch.
// `copies` launches of this size share the GPU, of which this one may split.
struct GemmPlan { int bn, splits, kb_per_split; double ns; };

GemmPlan plan_gemm(int n, long long rows, int num_kb, bool mn_major, int force_bn = 0, int copies = 1) {
  const long long m_tiles = (rows + 127) / 128;
  GemmPlan best{force_bn ? force_bn : cheapest_bn(n, rows, num_kb, mn_major, copies), 1, num_kb, 0.0};
  best.ns = im2col_ns(best.bn, n, rows, num_kb, mn_major, copies);
  if (num_kb < 64 || getenv("MTB_DISABLE_SPLITK")) return best;
  for (int bn = force_bn ? force_bn : pick_bn(n); bn >= (force_bn ? force_bn : 64); bn >>= 1)
    for (int s = 2; s <= 8 && bn / s >= 32; s *= 2) {
      if (m_tiles * ((n + bn - 1) / bn) * (s + copies - 1) > cluster_units(s)) continue;
      const int per = (num_kb + s - 1) / s;
      const double ns = (bn == 64 ? 6500 : bn == 128 ? 7700 : 10500) + (double)per * ((bn == 64 ? 180 : bn == 128 ? 200 : 280) + (mn_major ? 40 : 0));
      if (ns < best.ns) best = GemmPlan{bn, s, per, ns};
    }
  return best;
}

// Activations smaller than this stay on the CUDA-core kernels: tiny tensors gain nothing from
// the tensor cores, and im2col tensor maps over very small tensors are avoided altogether.
constexpr long long kMinIm2colBytes = 128 * 1024;

}  // namespace

#include "tc_conv_rows.cuh"
#include "tc_conv_taps.cuh"
#include "tc_wgrad_pairs.cuh"

// ------------------------------------------------------------------------------ host API

// Reads (and clears) the status word the tensor-core kernels set when a bounded wait ran out.
// Synchronises the device.
MTB_API int mtb_tc_status(int* status_out) {
  int h[8] = {0};
  MTB_CUDA(cudaDeviceSynchronize());
  MTB_CUDA(cudaMemcpyFromSymbol(h, g_tc_status, sizeof(h)));
  if (status_out) *status_out = h[0];
  if (h[0] != 0) {
    int z[8] = {0};
    MTB_CUDA(cudaMemcpyToSymbol(g_tc_status, z, sizeof(z)));
  }
  return MTB_OK;
}

// Self-test of the give-up path every tensor-core kernel shares: a CTA allocates tensor memory,
// then one thread waits (with the given limit) on an mbarrier that nothing will ever complete.
// The wait runs out, the waiter records `code` in the status word and raises the CTA's abort flag,
// and the kernel tears down like the real ones: tensor memory is freed, the CTA exits.
namespace {
__global__ void __launch_bounds__(64, 1) tc_wait_selftest_kernel(long long limit_cycles, int code) {
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), 32);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0 && lane == 0) mbar_wait_limit(smem_u32(&bar), 0, &abort_flag, code, limit_cycles);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_slot, 32);
  }
}
}  // namespace

MTB_API int mtb_tc_wait_selftest(long long limit_cycles, int code, void* stream) {
  MTB_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000LL && code != 0, "tc_wait_selftest: limit must be 1..2e8 cycles and code non-zero");
  tc_wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(limit_cycles, code);
  MTB_LAUNCH_CHECK("tc_wait_selftest_kernel");
  return MTB_OK;
}

bool mtb_tc_gemm_supported(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* c) {
  if (getenv("MTB_DISABLE_TC")) return false;
  if (!al16(a) || !al16(b) || !al16(c)) return false;
  if (m < 32 || n < 8 || k < 32) return false;
  if (k % 4) return false;                 // K-major pitches
  if (trans_a && m % 4) return false;      // A stored [K][M]
  if (!trans_b && n % 4) return false;     // B stored [K][N]
  return true;
}

int mtb_tc_gemm_f32(int m, int n, int k, const float* a, int trans_a, const float* b, int trans_b, const float* bias, int relu, float* c,
                    void* stream, float* pre) {
  CUtensorMap mapA, mapB;
  int bn = cheapest_bn(n, m, (k + 31) / 32, !trans_b), rows = 128;
  if (!trans_a && trans_b) {  // see Cfg
    auto narrow_ns = [&](int r, int c, double block, double fixed) {
      const long long tiles = (long long)((m + r - 1) / r) * ((n + c - 1) / c);
      return (tiles + mtb_sm_count() - 1) / mtb_sm_count() * (((k + 31) / 32) * block + fixed);
    };
    double best = im2col_ns(bn, n, m, (k + 31) / 32, false);
    const double wide_32 = narrow_ns(64, 32, 146, 900);  // as calibrated against the tiles of 128 rows
    if ((m <= 64 && wide_32 <= 900 + ((k + 31) / 32) * 146.0) || wide_32 < 0.9 * best) {
      // against 32 x 16: the time of a block is what both take from K = 1024 on; rows that are no whole sectors of 32 bytes cost
      // the 32 columns of this tile 600 ns more
      bn = 32; rows = 64;
      best = narrow_ns(64, 32, 125, n % 8 ? 1500 : 900);
    } else {
      best *= 0.9;
    }
    // Eight blocks a stage fill late: 500 ns more than 64 x 32 before the first MMA, 20 ns a block less from there on.  64 x 128 in one
    // wave, 64 x 32 and 32 x 16: K = 288 4.3 and 5.0 us, 768 6.2 and 6.5, 1024 7.6 and 7.4, 4096 19.5 and 17.4.  Over 1053 products of
    // 32 to 2000 rows, 10 to 2048 columns and K = 32 to 9216 the tile taken is 0.3 % off the fastest of the three, 10 % at most.
    if (narrow_ns(32, 16, 104, 1400) < best) { bn = 16; rows = 32; }
  }
  int rc;
  GemmParams p{};
  p.a_blocks = trans_a && m % 32 == 0;
  p.b_blocks = !trans_b && n % 32 == 0;
  if (!trans_a) rc = tc::encode_tiled_2d(&mapA, a, m, k, k, 32, rows);
  else if (p.a_blocks) rc = tc::encode_blocks_3d(&mapA, a, k, m, m, 32, 4);
  else rc = tc::encode_tiled_2d(&mapA, a, k, m, m, 32, 32, true);
  if (rc) return rc;
  if (trans_b) rc = tc::encode_tiled_2d(&mapB, b, n, k, k, 32, bn);
  else if (p.b_blocks) rc = tc::encode_blocks_3d(&mapB, b, k, n, n, 32, bn / 32);
  else rc = tc::encode_tiled_2d(&mapB, b, k, n, n, 32, 32, true);
  if (rc) return rc;
  p.splits = 1; p.kb_per_split = (k + 31) / 32;
  p.M = m; p.N = n; p.num_kb = (k + 31) / 32;
  p.m_tiles = (m + rows - 1) / rows; p.n_tiles = (n + bn - 1) / bn;
  p.out = c; p.ldo = n; p.bias = bias; p.relu = relu; p.pre = pre;
  p.KH = 1; p.KW = 1; p.cchunks = p.num_kb;
  cudaStream_t st = (cudaStream_t)stream;
  if (!trans_a && trans_b && pre) return launch_tc_bn<A_KMAJOR, B_KMAJOR, EPI_PRE>(bn, mapA, mapB, p, st);
  if (!trans_a && trans_b) return launch_tc_bn<A_KMAJOR, B_KMAJOR>(bn, mapA, mapB, p, st);
  if (!trans_a && !trans_b) return launch_tc_bn<A_KMAJOR, B_MNMAJOR>(bn, mapA, mapB, p, st);
  if (trans_a && trans_b) return launch_tc_bn<A_MNMAJOR, B_KMAJOR>(bn, mapA, mapB, p, st);
  return launch_tc_bn<A_MNMAJOR, B_MNMAJOR>(bn, mapA, mapB, p, st);
}

bool mtb_tc_conv2d_forward_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                     const float* wt, const float* y) {
  if (getenv("MTB_DISABLE_TC")) return false;
  if (!mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw)) return false;  // the other kernels say so
  if (!al16(x) || !al16(wt) || !al16(y)) return false;
  if (cin % 32 || cout % 4) return false;
  if (sh > 8 || sw > 8 || ph > 100 || pw > 100 || kh > 32 || kw > 32) return false;
  if ((long long)n * h * w * cin * 4 < kMinIm2colBytes) return false;
  return true;
}

namespace {
// The kernel by pairs of SMs for a forward pass or (mn_major) a data gradient, and what the launch takes without it.  One price for all epilogues, without
// the shared memory that some reserve in the other kernels: a layer's results are the same bits with every epilogue.
struct PairChoice {
  TapsPlan plan;
  double other_ns;
  bool taken;
};
PairChoice pair_choice(int n, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int kc, int nout, bool mn_major) {
  PairChoice r{taps_plan(n, h, w, kh, kw, sh, sw, ph, pw, kc, nout), 0.0, false};
  if (!r.plan.ok) return r;  // hence 3x3, stride 1, padding 1
  const long long rows = (long long)n * h * w;
  const int num_kb = 9 * (kc / 32), row_bn = pick_bn_for(nout, rows);
  const RowConvPlan plan = row_conv_plan(n, h, w, kh, kw, sh, sw, ph, pw, kc, nout, row_bn);
  const long long positions = (long long)n * plan.Hv * plan.Wp;
  const GemmPlan gp = plan_gemm(nout, rows, num_kb, mn_major);
  r.other_ns = row_conv_pays(plan, row_bn, positions, nout, num_kb, gp.ns) ? row_conv_ns(plan, row_bn, positions, nout, num_kb) : gp.ns;
  r.taken = r.plan.ns <= r.other_ns;
  return r;
}
}  // namespace

// stats / stats_rows (both may be NULL): when given and the shape allows, the kernel also writes partial
// rows [rows][3][cout] of per-channel (count, mean, M2) of y and *stats_rows receives their number;
// *stats_rows == 0 means this launch did not produce statistics.
int mtb_tc_conv2d_forward_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                              const float* wt, const float* bias, float* y, int relu, void* workspace, long long workspace_bytes, void* stream,
                              float* stats, int* stats_rows, const MtbBnEval* bn_eval, const float* residual) {
  if (stats_rows) *stats_rows = 0;
  const PairChoice pairs = pair_choice(n, h, w, kh, kw, sh, sw, ph, pw, cin, cout, false);
  if (pairs.taken) {
    const bool with_stats = stats && stats_rows && !relu && cout % 32 == 0 && !getenv("MTB_DISABLE_CONV_STATS");
    if (with_stats) *stats_rows = taps_stats_rows(pairs.plan);
    return run_taps<B_KMAJOR>(pairs.plan, n, h, w, cin, cout, x, wt, bias, residual, relu, y, (cudaStream_t)stream, with_stats ? stats : nullptr, bn_eval);
  }
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  const long long M = (long long)n * oh * ow, K = (long long)kh * kw * cin;
  const int row_bn = pick_bn_for(cout, M);
  const RowConvPlan plan = row_conv_plan(n, h, w, kh, kw, sh, sw, ph, pw, cin, cout, row_bn, bn_eval ? 12u * row_bn : 0u);
  const GemmPlan gp = plan_gemm(cout, M, (int)(K / 32), false);
  const bool staged = row_conv_pays(plan, row_bn, (long long)n * plan.Hv * plan.Wp, cout, (int)(K / 32), gp.ns);
  const int bn = staged ? row_bn : gp.bn;
  // the statistics and BatchNorm epilogues keep a CTA on one column tile: there must be a CTA for each
  const bool a_cta_per_column = (cout + bn - 1) / bn <= mtb_sm_count();
  if (bn_eval && !a_cta_per_column) {
    const int rc = mtb_tc_conv2d_forward_f32(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, x, wt, bias, y, 0, workspace, workspace_bytes, stream);
    return rc ? rc : mtb_bn_eval_apply(y, y, M, cout, *bn_eval, residual, relu, (cudaStream_t)stream);
  }
  const bool want_stats = stats && stats_rows && a_cta_per_column && !relu && cout % 32 == 0 && (!bias || al16(bias)) && !getenv("MTB_DISABLE_CONV_STATS");
  CUtensorMap mapA, mapB;
  int rc = tc::encode_tiled_2d(&mapB, wt, cout, K, K, 32, bn);
  if (rc) return rc;
  if (staged) {
    if (want_stats) *stats_rows = row_conv_stats_rows(plan, (long long)n * plan.Hv * plan.Wp, cout, bn);
    return run_row_conv<B_KMAJOR>(plan, bn, n, h, w, cin, kh, kw, ph, pw, cout, x, mapB, nullptr, bias, residual, relu, y, (cudaStream_t)stream,
                                  want_stats ? stats : nullptr, bn_eval);
  }
  rc = tc::encode_im2col_4d(&mapA, x, n, h, w, cin, -pw, -ph, pw - (kw - 1), ph - (kh - 1), sw, sh, 32, 128);
  if (rc) return rc;
  GemmParams p{};
  p.M = (int)M; p.N = cout; p.num_kb = (int)(K / 32);
  p.m_tiles = (int)((M + 127) / 128); p.n_tiles = (cout + bn - 1) / bn;
  p.out = y; p.ldo = cout; p.bias = bias; p.relu = relu;
  p.OW = ow; p.OH = oh; p.SW = sw; p.SH = sh; p.PW = pw; p.PH = ph; p.KW = kw; p.KH = kh; p.cchunks = cin / 32;
  p.splits = gp.splits; p.kb_per_split = gp.kb_per_split;
  // A short reduction (1x1) leaves the epilogue no main loop to hide the statistics behind, and takes less with them than
  // with BatchNorm's own pass all the same (both operators: 64 -> 128 channels, stride 2, to 16x16, 16 images 15.5 -> 12.3 us,
  // 128 images 22.9 -> 20.1, 192 images 30.0 -> 27.0, 512 images 57.0 -> 55.1; 256 -> 512 on 8 x 28x28 26.2 -> 19.0;
  // 64 -> 256 channels on 32 x 56x56 83.4 -> 78.0; ResNet-50 step 19.80 -> 19.23 ms).
  if (want_stats) {
    p.stats = stats;
    *stats_rows = gp.splits > 1 ? p.m_tiles * 4 : stats_rows_for(p.m_tiles * p.n_tiles, p.n_tiles);
    cudaStream_t st = (cudaStream_t)stream;
    return launch_tc_bn<A_IM2COL, B_KMAJOR, EPI_STATS>(bn, mapA, mapB, p, st);
  }
  if (bn_eval) {
    p.bn = *bn_eval;
    p.addend = residual;
    return launch_tc_bn<A_IM2COL, B_KMAJOR, EPI_BN>(bn, mapA, mapB, p, (cudaStream_t)stream);
  }
  return launch_tc_bn<A_IM2COL, B_KMAJOR>(bn, mapA, mapB, p, (cudaStream_t)stream);
}

bool mtb_tc_conv2d_dgrad_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                   const float* wt, const float* dx) {
  if (getenv("MTB_DISABLE_TC")) return false;
  if (!mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw)) return false;  // the other kernels say so
  if (!al16(dy) || !al16(wt) || !al16(dx)) return false;
  if (cout % 32 || cin % 4) return false;
  if (kh * kw > 64 || sh > 8 || sw > 8 || ph > 64 || pw > 64) return false;
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  if ((long long)n * oh * ow * cout * 4 < kMinIm2colBytes) return false;
  return true;
}

namespace {
// One axis of residue class a: its taps, its pixels (start + s * i, i < count) and the corners of the window its outputs see.
struct ClassAxis { int taps, start, count, lower, upper; };
ClassAxis class_axis(int a, int size, int osize, int k, int s, int pad) {
  ClassAxis r{};
  r.taps = a < k ? (k - a + s - 1) / s : 0;
  r.start = (((a - pad) % s) + s) % s;
  r.count = r.start < size ? (size - r.start + s - 1) / s : 0;
  const int c0 = (r.start + pad - a) / s;
  r.lower = c0 - (r.taps - 1);
  r.upper = r.count - osize + r.lower;
  return r;
}
}  // namespace

// Data gradient.  For stride 1 this is a convolution of dY with the filter rotated by 180
// degrees.  For stride s the input pixels fall into s*s residue classes; pixels of class (a, b)
// only see the taps kh = a (mod s), kw = b (mod s), and over the class's own (coarser) grid
// that is again a stride-1 convolution of dY with that sub-filter.  Each class is one launch of
// the implicit-GEMM kernel: dY plays the activation role (im2col-mode loads with zero fill
// beyond the edges), the weights are read in place as an MN-major operand (for one tap, rows
// are output channels = the reduction index, columns are input channels), and the epilogue
// scatters rows to the class's pixels.  Classes without taps (stride larger than the filter)
// receive zeros.  No atomics; every element of dX is written exactly once.
// addend (may be NULL): dx = dgrad + addend.  Fused into the epilogue on the row-staged path; the
// other paths write dgrad and add afterwards.
int mtb_tc_conv2d_dgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                            const float* wt, const float* addend, float* dx, void* workspace, long long workspace_bytes, void* stream) {
  if (addend != dx) {
    const PairChoice pairs = pair_choice(n, h, w, kh, kw, sh, sw, ph, pw, cout, cin, true);
    if (pairs.taken) return run_taps<B_MNMAJOR>(pairs.plan, n, h, w, cout, cin, dy, wt, nullptr, addend, 0, dx, (cudaStream_t)stream);
  }
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  // one tile width for all residue classes (the weight tensor map is shared): the one the cost model picks
  // for a class-sized problem
  const long long class_rows = (long long)n * h * w / (sh * sw);
  const int class_kb = ((kh + sh - 1) / sh) * ((kw + sw - 1) / sw) * (cout / 32);
  const int row_bn = pick_bn_for(cin, class_rows);
  const RowConvPlan plan = row_conv_plan(n, h, w, kh, kw, sh, sw, ph, pw, cout, cin, row_bn);
  const GemmPlan class_plan = plan_gemm(cin, class_rows, class_kb, true, 0, sh * sw);
  const bool staged = row_conv_pays(plan, row_bn, (long long)n * plan.Hv * plan.Wp, cin, class_kb, class_plan.ns);
  const int bn = staged ? row_bn : class_plan.bn;
  cudaStream_t st = (cudaStream_t)stream;
  CUtensorMap mapB;
  const long long wcols = (long long)kh * kw * cin;
  const bool b_blocks = cin % 32 == 0;  // a tap's columns then are whole blocks
  int rc = b_blocks ? tc::encode_blocks_3d(&mapB, wt, cout, wcols, wcols, 32, bn / 32) : tc::encode_tiled_2d(&mapB, wt, cout, wcols, wcols, 32, 32, true);
  if (rc) return rc;
  if (staged) {
    // stride 1: dX = dY convolved with the filter rotated by 180 degrees, same padding
    int tap_x[64];
    for (int jh = 0; jh < kh; ++jh)
      for (int jw = 0; jw < kw; ++jw) tap_x[jh * kw + jw] = ((kh - 1 - jh) * kw + (kw - 1 - jw)) * cin;
    return run_row_conv<B_MNMAJOR>(plan, bn, n, h, w, cout, kh, kw, ph, pw, cin, dy, mapB, tap_x, nullptr, addend, 0, dx, st, nullptr, nullptr, b_blocks);
  }
  bool need_zero = false;
  for (int a = 0; a < sh; ++a)
    for (int b = 0; b < sw; ++b) {
      const ClassAxis ah = class_axis(a, h, oh, kh, sh, ph), aw = class_axis(b, w, ow, kw, sw, pw);
      if (ah.count > 0 && aw.count > 0 && (ah.taps == 0 || aw.taps == 0)) need_zero = true;
    }
  // addend == dx: dx already holds the gradient to add to; every class adds its own pixels in its epilogue
  // and the pixels of classes without taps stay as they are.
  const bool in_place = addend != nullptr && addend == dx;
  // A 1x1 filter's data gradient is bound by writing dx, so its epilogue also reads the tensor to add and the separate
  // pass (read twice, write once) goes: 64 <- 256 channels on 128 x 56 x 56, see the measurements of the bottleneck step.
  // Filters with more taps are bound by the tensor pipe, which pays for every load in the epilogue (measured slower).
  const bool fused_add = addend != nullptr && !in_place && al16(addend) && kh * kw == 1 && sh * sw == 1;
  if (need_zero && !in_place) MTB_CUDA(cudaMemsetAsync(dx, 0, (size_t)n * h * w * cin * 4, st));
  // The classes write disjoint pixels.  When one class fills only part of the GPU they run side by side on
  // separate lanes.
  int live = 0;
  for (int a = 0; a < sh; ++a)
    for (int b = 0; b < sw; ++b) {
      const ClassAxis ah = class_axis(a, h, oh, kh, sh, ph), aw = class_axis(b, w, ow, kw, sw, pw);
      if (ah.count > 0 && aw.count > 0 && ah.taps > 0 && aw.taps > 0) ++live;
    }
  const long long class_units = ((class_rows + 127) / 128) * ((cin + bn - 1) / bn);
  const bool side_by_side = live > 1 && class_units < mtb_sm_count() && !getenv("MTB_DGRAD_SERIAL");
  const int lanes = side_by_side ? (live < kMaxLanes ? live : kMaxLanes) : 1;
  cudaStream_t lane_stream[kMaxLanes];
  rc = mtb_fork_lanes(st, lanes, lane_stream);
  if (rc) return rc;
  int launched = 0;
  for (int a = 0; a < sh; ++a) {
    for (int b = 0; b < sw; ++b) {
      const ClassAxis ah = class_axis(a, h, oh, kh, sh, ph), aw = class_axis(b, w, ow, kw, sw, pw);
      if (ah.count == 0 || aw.count == 0 || ah.taps == 0 || aw.taps == 0) continue;
      cudaStream_t cst = lane_stream[launched++ % lanes];
      CUtensorMap mapA;
      rc = tc::encode_im2col_4d(&mapA, dy, n, oh, ow, cout, aw.lower, ah.lower, aw.upper, ah.upper, 1, 1, 32, 128);
      if (rc) return rc;
      GemmParams p{};
      const long long M = (long long)n * ah.count * aw.count;
      p.M = (int)M; p.N = cin; p.num_kb = ah.taps * aw.taps * (cout / 32);
      const GemmPlan gp = plan_gemm(cin, M, p.num_kb, true, bn, lanes);
      p.splits = gp.splits; p.kb_per_split = gp.kb_per_split;
      p.m_tiles = (int)((M + 127) / 128); p.n_tiles = (cin + bn - 1) / bn;
      p.out = dx; p.ldo = cin; p.bias = nullptr; p.relu = 0;
      p.addend = in_place || fused_add ? addend : nullptr;
      p.OW = aw.count; p.OH = ah.count; p.SW = 1; p.SH = 1; p.PW = -aw.lower; p.PH = -ah.lower; p.KW = aw.taps; p.KH = ah.taps;
      p.cchunks = cout / 32;
      p.b_per_tap = 1;
      p.b_blocks = b_blocks;
      for (int jh = 0; jh < ah.taps; ++jh)
        for (int jw = 0; jw < aw.taps; ++jw) {
          const int fkh = a + sh * (ah.taps - 1 - jh), fkw = b + sw * (aw.taps - 1 - jw);  // dY offset j <-> filter tap
          p.b_tap_x[jh * aw.taps + jw] = (fkh * kw + fkw) * cin;
        }
      p.o_strided = sh * sw > 1; p.o_Hc = ah.count; p.o_Wc = aw.count; p.o_H = h; p.o_W = w; p.o_h0 = ah.start; p.o_w0 = aw.start; p.o_sh = sh; p.o_sw = sw;
      rc = p.addend ? launch_tc_bn<A_IM2COL, B_MNMAJOR, EPI_ADD>(bn, mapA, mapB, p, cst) : launch_tc_bn<A_IM2COL, B_MNMAJOR>(bn, mapA, mapB, p, cst);
      if (rc) return rc;
    }
  }
  rc = mtb_join_lanes(st, lanes);
  if (rc) return rc;
  if (addend && !in_place && !fused_add) return mtb_add_f32(dx, addend, dx, (long long)n * h * w * cin, 1.0f, st);
  return MTB_OK;
}

// True when mtb_tc_conv2d_dgrad_f32 with addend == dx (accumulate in place) is available AND is the cheaper
// form: strided convolutions some of whose residue classes have no taps (1x1 with stride 2), where the
// out-of-place form costs a memset, a scattered write and a pass that adds the two tensors.
bool mtb_tc_conv2d_dgrad_in_place(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* dy,
                                  const float* wt, const float* dx) {
  if (!mtb_tc_conv2d_dgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, dy, wt, dx)) return false;
  if (sh * sw == 1 || getenv("MTB_DGRAD_OUT_OF_PLACE")) return false;
  return kh < sh || kw < sw;  // a residue class a >= kh (b >= kw) sees no tap
}

// ------------------------------------------------------------------------------ weight gradient
//
// dW^T[(tap, ci), co] = sum over output pixels m of patch(X)[m, (tap, ci)] * dY[m, co].
// Both operands are "MN-major" in memory (for a fixed pixel, channels are contiguous), so they
// are staged exactly as they lie: the A tile is 4 im2col-mode loads of 32 pixels x 32 channels
// (one per (tap, channel-block)), the B tile BN/32 boxes of 32 pixels x 32 output channels.
// The reduction runs over pixels, which is long (up to N*OH*OW) while the output is small, so
// the pixel range is split across CTAs; each writes an fp32 partial to scratch and a second
// kernel adds the partials in a fixed order and transposes into dW[co][tap][ci].
namespace {

// PB pixels (reduction elements) per stage; one A chunk = PB pixels x 32 channels.
template <int BN, int PB>
struct WCfg {
  static constexpr uint32_t kChunk = PB * 128;
  static constexpr uint32_t kABytes = 4 * kChunk;
  static constexpr uint32_t kBBytes = (BN / 32) * kChunk;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr int kStagesFit = (227 * 1024 - 2048) / kStageBytes;
  static constexpr int kStages = kStagesFit > 6 ? 6 : kStagesFit;
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + 1024;
  static constexpr uint32_t kTmemCols = 2 * BN;
};

struct WgradParams {
  int Kw;            // KH*KW*Cin: rows of the transposed gradient
  int Cout;
  int chunks;        // Kw / 32
  int cchunks;       // Cin / 32
  int m_tiles, n_tiles, splits;
  int kb_total;      // ceil(pixels / PB)
  int kb_per_split;
  int OW, OH, SW, SH, PW, PH, KW;
  int dy_blocks;     // dY through one copy per stage (Cout % 32 == 0)
  float* partial;    // [splits][Kw][Cout]
};

template <int BN, int PB>
__global__ void __launch_bounds__(kGemmThreads, 1)
tc_wgrad_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapDY, const WgradParams p) {
  using C = WCfg<BN, PB>;
  constexpr int STAGES = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[8], bar_empty[8], bar_tfull[2], bar_tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_tfull[b]), 1);
      mbar_init(smem_u32(&bar_tempty[b]), kEpilogueWarps);  // one arrival per epilogue warp
    }
    abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  mtb_wait_prior();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const int units = p.m_tiles * p.n_tiles * p.splits;
  volatile int* abort_ptr = &abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&mapX);
      prefetch_tensormap(&mapDY);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
        const int split = unit % p.splits, tile = unit / p.splits;
        const int m_tile = tile / p.n_tiles, n0 = (tile % p.n_tiles) * BN;
        const int kb0 = split * p.kb_per_split;
        const int kb1 = kb0 + p.kb_per_split < p.kb_total ? kb0 + p.kb_per_split : p.kb_total;
        int valid = p.chunks - m_tile * 4;
        if (valid > 4) valid = 4;
        const uint32_t bytes = (uint32_t)valid * C::kChunk + C::kBBytes;
        int q_c[4], q_kw[4], q_kh[4];
        for (int q = 0; q < 4; ++q) {
          const int chunk = m_tile * 4 + (q < valid ? q : 0);
          const int tap = chunk / p.cchunks;
          q_c[q] = (chunk - tap * p.cchunks) * 32;
          q_kh[q] = tap / p.KW;
          q_kw[q] = tap - q_kh[q] * p.KW;
        }
        // first pixel of the range, then advanced by PB pixels per block without divisions
        int m = kb0 * PB;
        int ow = m % p.OW, tq = m / p.OW;
        int oh = tq % p.OH, pn_ = tq / p.OH;
        for (int kb = kb0; kb < kb1; ++kb, m += PB) {
          if (!mbar_wait(smem_u32(&bar_empty[stage]), phase ^ 1u, abort_ptr, 11)) { ok = false; break; }
          const uint32_t full = smem_u32(&bar_full[stage]);
          mbar_expect_tx(full, bytes);
          const uint32_t a_dst = smem_base + stage * C::kStageBytes, b_dst = a_dst + C::kABytes;
          const int pw_ = ow * p.SW - p.PW, ph_ = oh * p.SH - p.PH;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q < valid) tma_load_im2col_4d(a_dst + q * C::kChunk, &mapX, full, q_c[q], pw_, ph_, pn_, (uint16_t)q_kw[q], (uint16_t)q_kh[q]);
          if (p.dy_blocks) {
            tma_load_3d(b_dst, &mapDY, full, 0, m, n0 / 32);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 32; ++j) tma_load_2d(b_dst + j * C::kChunk, &mapDY, full, n0 + 32 * j, m);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          ow += PB;
          while (ow >= p.OW) {
            ow -= p.OW;
            if (++oh == p.OH) { oh = 0; ++pn_; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // converged warp, elected issue (see tc_gemm_kernel)
    constexpr uint32_t idesc = idesc_tf32(128, BN, 1, 1);
    constexpr uint32_t hi = desc_hi_mnmajor();
    constexpr uint32_t step = 1024u >> 4;
    const uint32_t a_lo0 = desc_lo_mnmajor(smem_base, C::kChunk), b_lo0 = desc_lo_mnmajor(smem_base + C::kABytes, C::kChunk);
    int stage = 0;
    uint32_t phase = 0;
    int t = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++t) {
      const int split = unit % p.splits;
      const int kb0 = split * p.kb_per_split;
      const int kb1 = kb0 + p.kb_per_split < p.kb_total ? kb0 + p.kb_per_split : p.kb_total;
      const int buf = t & 1;
      const uint32_t use = (uint32_t)(t >> 1);
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_tempty[buf]), (use & 1u) ^ 1u, abort_ptr, 12));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      uint32_t acc = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[stage]), phase, abort_ptr, 13));
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_lo = a_lo0 + stage * (C::kStageBytes >> 4), b_lo = b_lo0 + stage * (C::kStageBytes >> 4);
        if (elect_one()) {
          mma_tf32_words(d_tmem, a_lo, hi, b_lo, hi, idesc, acc);
#pragma unroll
          for (int kk = 1; kk < PB / 8; ++kk) mma_tf32_words(d_tmem, a_lo + kk * step, hi, b_lo + kk * step, hi, idesc, 1u);
          mma_commit(smem_u32(&bar_empty[stage]));
        }
        __syncwarp();
        acc = 1u;
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (ok && elect_one()) mma_commit(smem_u32(&bar_tfull[buf]));
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3, c_first = warp < 6 ? 0 : BN / 2;
    int t = 0;
    const bool wide_ok = (p.Cout % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.partial) & 31u) == 0);  // 32-byte stores
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++t) {
      const int split = unit % p.splits, tile = unit / p.splits;
      const int m_tile = tile / p.n_tiles, n0 = (tile % p.n_tiles) * BN;
      const int kb0 = split * p.kb_per_split;
      const bool empty_unit = kb0 >= p.kb_total;  // cannot happen with the host's split choice; kept for safety
      const int buf = t & 1;
      const uint32_t use = (uint32_t)(t >> 1);
      // one lane polls (128 threads spinning on the barrier slow the other roles' barrier traffic down)
      bool ok = lane != 0 || mbar_wait(smem_u32(&bar_tfull[buf]), use & 1u, abort_ptr, 14);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int row = m_tile * 128 + quarter * 32 + lane;
      float* orow = p.partial + ((long long)split * p.Kw + row) * p.Cout;
#pragma unroll 1
      for (int c0 = c_first; c0 < c_first + BN / 2; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c0), r);
        tmem_ld_wait();
        const int col0 = n0 + c0;
        if (row < p.Kw && col0 < p.Cout) {
          if (col0 + 32 <= p.Cout) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float4 v = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
              float4 u = make_float4(__uint_as_float(r[j + 4]), __uint_as_float(r[j + 5]), __uint_as_float(r[j + 6]), __uint_as_float(r[j + 7]));
              if (empty_unit) v = u = make_float4(0.f, 0.f, 0.f, 0.f);
              st_row8(orow + col0 + j, v, u, wide_ok);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.Cout) orow[col0 + j] = empty_unit ? 0.f : __uint_as_float(r[j]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[buf]));
    }
  }

  tc_fence_before();
  __syncthreads();
  // Behind the barrier: the first thread's call counts for the CTA, and that of a producer that has nothing left to copy let the CTAs of
  // the planes' addition take registers beside the main stream's kernels while this one still had its accumulators to store (ResNet-18
  // step at 512 images 5.67 -> 5.47 ms, at 128 1925 -> 1903 us, ResNet-50 18.24 -> 18.16 ms).
  mtb_launch_dependents();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// dw[co][r] = sum_s partial[s][r][co]: a CTA takes 8 rows x 128 output channels, reads float4 along co (even and odd
// splits in one sum each, in index order), transposes through shared memory and writes 32-byte runs along r.
// Bound by latency where there is little to read: a 1x1 layer or a stem has one split per SM and a few thousand outputs,
// and blocks of 32 rows with two loads in flight took 25 us over 148 planes; with 8 rows and sixteen loads in flight
// four times as many CTAs take a quarter of the round trips each.
constexpr int kReduceRows = 8;
__global__ void __launch_bounds__(32 * kReduceRows) wgrad_reduce_transpose_kernel(const float* __restrict__ partial, float* __restrict__ dw, int Kw,
                                                                                   int Cout, int splits) {
  mtb_wait_prior();
  __shared__ float tile[128][kReduceRows + 1];
  const int r0 = blockIdx.x * kReduceRows, c0 = blockIdx.y * 128;
  const long long plane = (long long)Kw * Cout;
  {
    const int r = r0 + threadIdx.y, c = c0 + 4 * threadIdx.x;
    float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
    if (r < Kw && c < Cout) {  // Cout % 4 == 0 on this path, so the four channels are in range together
      const float* q = partial + (long long)r * Cout + c;
      auto add = [](float4& s, const float4& a) { s.x += a.x; s.y += a.y; s.z += a.z; s.w += a.w; };
      constexpr int AHEAD = 16;
      int z = 0;
      for (; z + AHEAD <= splits; z += AHEAD) {
        float4 v[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) v[u] = *reinterpret_cast<const float4*>(q + (z + u) * plane);
#pragma unroll
        for (int u = 0; u < AHEAD; u += 2) { add(s0, v[u]); add(s1, v[u + 1]); }
      }
      for (; z + 1 < splits; z += 2) {
        const float4 a = *reinterpret_cast<const float4*>(q + z * plane), b = *reinterpret_cast<const float4*>(q + (z + 1) * plane);
        add(s0, a);
        add(s1, b);
      }
      if (z < splits) add(s0, *reinterpret_cast<const float4*>(q + z * plane));
    }
    tile[4 * threadIdx.x + 0][threadIdx.y] = s0.x + s1.x;
    tile[4 * threadIdx.x + 1][threadIdx.y] = s0.y + s1.y;
    tile[4 * threadIdx.x + 2][threadIdx.y] = s0.z + s1.z;
    tile[4 * threadIdx.x + 3][threadIdx.y] = s0.w + s1.w;
  }
  __syncthreads();
  const int t = threadIdx.y * 32 + threadIdx.x, r = r0 + t % kReduceRows;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int cc = t / kReduceRows + 32 * k, c = c0 + cc;
    if (r < Kw && c < Cout) dw[(long long)c * Kw + r] = tile[cc][t % kReduceRows];
  }
}

struct WgradPlan {
  int bn, pb, m_tiles, n_tiles, splits, kb_total, kb_per_split;
  long long Kw, pixels;
};

WgradPlan wgrad_plan(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  WgradPlan q;
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  q.pixels = (long long)n * oh * ow;
  q.Kw = (long long)kh * kw * cin;
  q.bn = pick_bn(cout);
  q.m_tiles = (int)((q.Kw + 127) / 128);
  q.n_tiles = (cout + q.bn - 1) / q.bn;
  // An im2col-mode load costs roughly the same whatever its size (measured: 4 loads of 32 pixels per
  // stage ran at 100 TFLOP/s, 4 loads of 64 pixels at 169), so stages hold 64 pixels even where only
  // two stages then fit (BN = 256: 239 -> 290 TFLOP/s).
  q.pb = 64;
  q.kb_total = (int)((q.pixels + q.pb - 1) / q.pb);
  const int tiles = q.m_tiles * q.n_tiles;
  // as many splits as still fit the GPU in ONE wave (rounding up instead left a second, nearly empty wave:
  // 18 tiles x 9 splits = 162 units on 148 SMs ran 117 us, 8 splits run one wave)
  int splits = mtb_sm_count() / tiles;
  const int max_splits = (q.kb_total + 3) / 4;  // at least 4 reduction blocks per CTA
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  q.kb_per_split = (q.kb_total + splits - 1) / splits;
  q.splits = (q.kb_total + q.kb_per_split - 1) / q.kb_per_split;  // no empty split
  return q;
}

}  // namespace

// Which kernel family each of forward / data gradient / weight gradient can take for a shape: row-staged wherever
// its layout fits (the launch then takes that or im2col, whichever is priced lower: row_conv_pays, wgrad_rows_pay)
// (pointers assumed 16-byte aligned), and, for the row-staged kernels, how their shared and tensor
// memory is laid out against the furthest byte their copies write and their descriptors read.
// Host code only: callable without a device (the SM count then defaults to 148).
//   out[0..2]   path of forward, dgrad, wgrad: 0 FP32 (CUDA cores, or two-term products where scratch is passed and they pay), 1 im2col tcgen05,
//               2 row-staged tcgen05
//   out[3..9]   forward, row-staged: dynamic smem bytes, activation stage bytes, last byte written by
//               the row copies, last byte read through a descriptor, TMEM columns, tiles per item,
//               1 if the filter is resident
//   out[10..16] the same for dgrad
//   out[17..24] wgrad, row-staged: dynamic smem bytes, X panel bytes, last byte written, last byte
//               read, dY panel bytes, last byte written, last byte read, TMEM columns
MTB_API int mtb_conv2d_plan_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int* out) {
  MTB_REQUIRE(out && n > 0 && cin > 0 && cout > 0 && h > 0 && w > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0, "conv2d_plan: bad arguments");
  for (int i = 0; i < 25; ++i) out[i] = 0;
  const float* al = reinterpret_cast<const float*>(uintptr_t(256));
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  if (oh <= 0 || ow <= 0) return MTB_OK;
  auto describe = [&](int slot, int kc, int nout, long long rows) {
    const int bn = pick_bn_for(nout, rows);
    const RowConvPlan q = row_conv_plan(n, h, w, kh, kw, sh, sw, ph, pw, kc, nout, bn);
    if (!q.ok) return false;
    const long long span = 128LL * q.mt;
    out[slot + 0] = (int)q.smem_bytes;
    out[slot + 1] = (int)q.a_stage_bytes;
    out[slot + 2] = (int)(kRowLead + (long long)q.nr_max * q.Wp * 128);
    out[slot + 3] = (int)(kRowLead + ((q.Wp - 1) + (span - 1) + (long long)(kh - 1) * q.Wp + (kw - 1) - pw + 1) * 128);
    out[slot + 4] = 2 * q.mt * bn;
    out[slot + 5] = q.mt;
    out[slot + 6] = q.resident;
    return true;
  };
  if (mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al))
    out[0] = describe(3, cin, cout, (long long)n * oh * ow) ? 2 : 1;
  if (mtb_tc_conv2d_dgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al))
    out[1] = describe(10, cout, cin, (long long)n * h * w / (sh * sw)) ? 2 : 1;
  if (mtb_tc_conv2d_wgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al)) {
    const WgradRowsPlan q = wgrad_rows_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
    out[2] = q.ok ? 2 : 1;
    if (q.ok) {
      const int nr_y = (q.Wp - 1 + kWgRowsPB - 1) / q.Wp + 1, nr_x = nr_y + 2 * ph;
      out[17] = (int)q.smem_bytes;
      out[18] = (int)q.x_panel_bytes;
      out[19] = (int)(kRowLead + (long long)nr_x * q.Wp * 128);
      out[20] = (int)(kRowLead + ((q.Wp - 1) - pw + (long long)(kh - 1) * q.Wp + 4 * q.n_kwg - 1 + (kWgRowsPB - 1) + 1) * 128);
      out[21] = (int)q.y_panel_bytes;
      out[22] = (int)((long long)nr_y * q.Wp * 128);
      out[23] = (int)(((q.Wp - 1) + (kWgRowsPB - 1) + 1) * 128);
      out[24] = kh * q.n_kwg * q.ncc_g * q.bn;
    }
  }
  return MTB_OK;
}

// How the kernel that works in pairs of SMs (tc_conv_taps.cuh) lays out a shape, wherever its layout fits (whether it is taken: mtb_conv2d_pair_choice_f32).
// Host code only.  out[0..8] forward, out[9..17] data gradient: form (1 or 2; 0: does not fit), dynamic smem bytes, stage bytes, first and
// (one past the) last byte written by the row copies, first and last byte read through a descriptor, image rows a stage, TMEM columns.
MTB_API int mtb_conv2d_pair_plan_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int* out) {
  MTB_REQUIRE(out && n > 0 && cin > 0 && cout > 0 && h > 0 && w > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0, "conv2d_pair_plan: bad arguments");
  for (int dir = 0; dir < 2; ++dir, out += 9) {
    for (int i = 0; i < 9; ++i) out[i] = 0;
    const int kc = dir ? cout : cin;
    const TapsPlan q = taps_plan(n, h, w, kh, kw, sh, sw, ph, pw, kc, dir ? cin : cout);
    if (!q.ok) continue;
    out[0] = q.beside;
    out[1] = (int)q.smem_bytes;
    out[2] = (int)q.a_stage_bytes;
    for (int col = 0; col < (q.rows ? 1 : q.Wp); ++col) {  // column of a tile's first position: whole rows start at 0
      const int rows = q.rows ? q.rows + 2 : (col + 128) / q.Wp + 3, first = (q.origin - q.Wp - col) * 128, end = first + rows * q.Wp * 128;
      if (col == 0 || first < out[3]) out[3] = first;
      if (end > out[4]) out[4] = end;
      if (rows > out[7]) out[7] = rows;
    }
    out[5] = (q.origin - q.Wp - (q.beside == 1 ? 1 : 0)) * 128;
    out[6] = (q.origin + q.Wp + 127 + 1 + 1) * 128;
    out[8] = kTapsBufs * q.beside * 64;
  }
  return MTB_OK;
}

// Whether forward, data gradient (pointers assumed aligned, the gradient not in place) and weight gradient of a shape run by pairs of SMs.  Host code only.
// out[0..2] forward, out[3..5] data gradient: taken, and the prices that decide, in ns: this kernel's, and of the one that is taken otherwise.  out[6]: weight gradient taken.
MTB_API int mtb_conv2d_pair_choice_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int* out) {
  MTB_REQUIRE(out && n > 0 && cin > 0 && cout > 0 && h > 0 && w > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0, "conv2d_pair_choice: bad arguments");
  const float* al = reinterpret_cast<const float*>(uintptr_t(256));
  for (int dir = 0; dir < 2; ++dir, out += 3) {
    const PairChoice r = pair_choice(n, h, w, kh, kw, sh, sw, ph, pw, dir ? cout : cin, dir ? cin : cout, dir != 0);
    const bool supported = dir ? mtb_tc_conv2d_dgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al)
                               : mtb_tc_conv2d_forward_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al);
    out[0] = r.taken && supported;
    out[1] = (int)r.plan.ns;
    out[2] = (int)r.other_ns;
  }
  out[0] = mtb_tc_conv2d_wgrad_supported(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout, al, al, al) &&
           wgrad_pairs_pay(wgrad_pair_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout));
  return MTB_OK;
}

// Host code only: see kPairMinSmem for what it has to be.
MTB_API long long mtb_conv2d_pair_smem_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, int direction) {
  if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || w <= 0 || kh <= 0 || kw <= 0 || sh <= 0 || sw <= 0) return 0;
  if (direction == 2) {
    const WgradPairPlan q = wgrad_pair_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
    return q.ok ? q.smem_bytes : 0;
  }
  const TapsPlan q = taps_plan(n, h, w, kh, kw, sh, sw, ph, pw, direction ? cout : cin, direction ? cin : cout);
  return q.ok ? q.smem_bytes : 0;
}

long long mtb_tc_conv2d_workspace_bytes(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout) {
  if (cin % 32) return 0;
  WgradPlan q = wgrad_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  long long bytes = (long long)q.splits * q.Kw * cout * 4 + 256;
  const WgradRowsPlan rq = wgrad_rows_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (rq.ok) {
    const long long b2 = (long long)rq.splits * q.Kw * cout * 4 + 256;
    if (b2 > bytes) bytes = b2;
  }
  const WgradPairPlan pq = wgrad_pair_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (wgrad_pairs_pay(pq)) {
    const long long b2 = (long long)pq.splits * q.Kw * cout * 4 + 256;
    if (b2 > bytes) bytes = b2;
  }
  return bytes;
}

bool mtb_tc_conv2d_wgrad_supported(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                                   const float* dy, const float* dw) {
  if (getenv("MTB_DISABLE_TC")) return false;
  if (!mtb_window_fits(h, ph, kh) || !mtb_window_fits(w, pw, kw)) return false;  // the other kernels say so
  if (!al16(x) || !al16(dy) || !al16(dw)) return false;
  if (cin % 32 || cout % 4) return false;
  if (sh > 8 || sw > 8 || ph > 100 || pw > 100 || kh > 32 || kw > 32) return false;
  if ((long long)n * h * w * cin * 4 < kMinIm2colBytes) return false;
  return true;
}

int mtb_tc_conv2d_wgrad_f32(int n, int cin, int h, int w, int kh, int kw, int sh, int sw, int ph, int pw, int cout, const float* x,
                            const float* dy, float* dw, void* workspace, long long workspace_bytes, void* stream) {
  const int oh = (h + 2 * ph - kh) / sh + 1, ow = (w + 2 * pw - kw) / sw + 1;
  const WgradPairPlan pq = wgrad_pair_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (wgrad_pairs_pay(pq)) {
    MTB_REQUIRE(workspace && workspace_bytes >= (long long)pq.splits * kh * kw * cin * cout * 4, "conv2d_wgrad: workspace too small");
    return run_wgrad_pairs(pq, n, h, w, cout, x, dy, dw, (float*)workspace, (cudaStream_t)stream);
  }
  const WgradRowsPlan rq = wgrad_rows_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  if (wgrad_rows_pay(rq, cin, cout)) {
    MTB_REQUIRE(workspace && workspace_bytes >= (long long)rq.splits * kh * kw * cin * cout * 4, "conv2d_wgrad: workspace too small");
    return run_wgrad_rows(rq, n, cin, h, w, kh, kw, ph, pw, cout, x, dy, dw, (float*)workspace, (cudaStream_t)stream);
  }
  WgradPlan q = wgrad_plan(n, cin, h, w, kh, kw, sh, sw, ph, pw, cout);
  MTB_REQUIRE(workspace && workspace_bytes >= (long long)q.splits * q.Kw * cout * 4, "conv2d_wgrad: workspace too small");
  CUtensorMap mapX, mapDY;
  int rc = tc::encode_im2col_4d(&mapX, x, n, h, w, cin, -pw, -ph, pw - (kw - 1), ph - (kh - 1), sw, sh, 32, q.pb, true);
  if (rc) return rc;
  WgradParams p{};
  p.dy_blocks = cout % 32 == 0;
  rc = p.dy_blocks ? tc::encode_blocks_3d(&mapDY, dy, q.pixels, cout, cout, q.pb, q.bn / 32) : tc::encode_tiled_2d(&mapDY, dy, q.pixels, cout, cout, 32, q.pb, true);
  if (rc) return rc;
  p.Kw = (int)q.Kw; p.Cout = cout; p.chunks = (int)(q.Kw / 32); p.cchunks = cin / 32;
  p.m_tiles = q.m_tiles; p.n_tiles = q.n_tiles; p.splits = q.splits; p.kb_total = q.kb_total; p.kb_per_split = q.kb_per_split;
  p.OW = ow; p.OH = oh; p.SW = sw; p.SH = sh; p.PW = pw; p.PH = ph; p.KW = kw;
  p.partial = (float*)workspace;
  cudaStream_t st = (cudaStream_t)stream;
  const int units = q.m_tiles * q.n_tiles * q.splits;
  const int grid = units < mtb_sm_count() ? units : mtb_sm_count();
#define MTB_LAUNCH_WGRAD(BN_, PB_)                                                                                      \
  do {                                                                                                                  \
    static unsigned long long configured = 0;                                                                           \
    if (int rc_ = mtb_opt_in_smem((const void*)tc_wgrad_kernel<BN_, PB_>, (int)WCfg<BN_, PB_>::kSmemBytes, &configured)) \
      return rc_;                                                                                                       \
    MTB_LAUNCH(tc_wgrad_kernel<BN_, PB_>, dim3(grid), dim3(kGemmThreads), WCfg<BN_, PB_>::kSmemBytes, st, mapX, mapDY, p);                           \
  } while (0)
  if (q.bn == 64) MTB_LAUNCH_WGRAD(64, 64);
  else if (q.bn == 128) MTB_LAUNCH_WGRAD(128, 64);
  else MTB_LAUNCH_WGRAD(256, 64);
#undef MTB_LAUNCH_WGRAD
  MTB_LAUNCH_CHECK("tc_wgrad_kernel");
  dim3 rgrid((unsigned)((q.Kw + kReduceRows - 1) / kReduceRows), (unsigned)((cout + 127) / 128));
  MTB_LAUNCH(wgrad_reduce_transpose_kernel, rgrid, dim3(32, kReduceRows), 0, st, (const float*)workspace, dw, (int)q.Kw, cout, q.splits);
  MTB_LAUNCH_CHECK("wgrad_reduce_transpose_kernel");
  return MTB_OK;
}

#include "tc_split.cuh"
