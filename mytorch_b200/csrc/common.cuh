// Shared helpers for the sm_100a kernel library: error reporting, launch checks, grid sizing.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#define MTB_API extern "C" __attribute__((visibility("default")))

enum MtbStatus {
  MTB_OK = 0,
  MTB_ERR_INVALID = 1,      // bad argument (null pointer, negative size, unsupported shape)
  MTB_ERR_CUDA = 2,         // a CUDA runtime / driver call failed
  MTB_ERR_UNSUPPORTED = 3,  // shape not covered by the requested kernel family
  MTB_ERR_WORKSPACE = 4,    // caller's scratch buffer is too small
  MTB_ERR_DEVICE = 5,       // a kernel reported a device-side problem (bounded wait ran out)
};

// BatchNorm with running statistics, applied where a convolution stores its output (inference): (v - mean) * scale + beta
// with scale = gamma / sqrt(var + eps); mean == NULL: none.  gamma / beta may be NULL.
struct MtbBnEval {
  const float *mean, *var, *gamma, *beta;
  float eps;
};

int mtb_fail(int code, const char* fmt, ...);
int mtb_sm_count();
// Opt a kernel in to `bytes` of dynamic shared memory on the CURRENT device.  The attribute is kept
// per device, so `done_mask` (one per kernel, zero-initialised) remembers the ordinals already set.
int mtb_opt_in_smem(const void* kernel, int bytes, unsigned long long* done_mask);

// Lanes: up to three auxiliary streams per device for an entry point that enqueues several launches which
// do not depend on one another (and each fill only part of the GPU).  mtb_fork_lanes makes lanes 1..n-1 wait
// for everything enqueued on `main` so far and returns their streams (lane 0 is `main` itself);
// mtb_join_lanes makes `main` wait for them.  Inside a stream capture both become graph dependencies.
constexpr int kMaxLanes = 4;
int mtb_fork_lanes(cudaStream_t main, int lanes, cudaStream_t* out);
int mtb_join_lanes(cudaStream_t main, int lanes);

// Held by every entry point that leaves something in the caller's scratch in one launch and reads it in a later one: two host
// threads that share a device, its stream and its scratch (as two threads of the Python layer do) would otherwise mix their launches,
// and one would read what the other has written in between.  One lock for all devices: asking for the current one costs more than it.
class MtbScratchTurn {
 public:
  MtbScratchTurn();
  ~MtbScratchTurn();
  MtbScratchTurn(const MtbScratchTurn&) = delete;
  MtbScratchTurn& operator=(const MtbScratchTurn&) = delete;
};

#define MTB_REQUIRE(cond, ...) \
  do { if (!(cond)) return mtb_fail(MTB_ERR_INVALID, __VA_ARGS__); } while (0)

#define MTB_CUDA(call) \
  do { cudaError_t e__ = (call); \
       if (e__ != cudaSuccess) return mtb_fail(MTB_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e__)); } while (0)

#define MTB_LAUNCH_CHECK(name) \
  do { cudaError_t e__ = cudaGetLastError(); \
       if (e__ != cudaSuccess) return mtb_fail(MTB_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e__)); } while (0)

// Programmatic dependent launch: the next kernel's CTAs are launched while this one runs, so the launch latency between the
// two (about 1.5 us in a stream or graph) and the prologues (barriers, TMEM, tensor maps) are hidden.  Every kernel calls
// mtb_wait_prior() before it touches global memory: that returns when everything before it in the stream has completed and
// is visible, so the order of the results is the stream's.  mtb_launch_dependents() says nothing about results; where it is
// called decides how early the next kernel's CTAs take their places.  Most kernels call it first.  The tensor-core kernels call
// it when they are done: a CTA of theirs has its SM's shared memory and tensor memory to itself for most of the launch, and a
// dependent that allocates tensor memory beside it would wait inside the allocation.  The last steps of reductions
// (colsum_final, ce_mean, wgrad_reduce_*) leave it to their exit.
// Launches without the attribute are unaffected by either call.  Measured on every kernel against on none: an 18-layer residual
// network's step at batch 128 2400 -> 2123 us, its captured step at batch 64 1586 -> 1478 us, its inference at batch 100
// 577 -> 540 us, a captured three-convolution step 219 -> 204 us.
__device__ __forceinline__ void mtb_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void mtb_wait_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `early` false: an ordinary launch.
template <class... P, class... A>
static inline cudaError_t mtb_launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

#define MTB_LAUNCH(kernel, ...) MTB_CUDA(mtb_launch_after(true, kernel, __VA_ARGS__))

// Whether a window of `window` elements lies in `extent` of them with `pad` more on either side: where it does not, an output
// extent computed as (extent + 2 * pad - window) / stride + 1 may still be 1, as C divides towards zero.
static inline bool mtb_window_fits(int extent, int pad, int window) { return (long long)extent + 2LL * pad >= window; }

static inline int mtb_div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

// Grid for a grid-stride bandwidth kernel: enough CTAs to fill the machine a few times over,
// as a multiple of the SM count, but never more than the work needs.
static inline int mtb_stream_grid(long long work_items, int threads, int ctas_per_sm = 8) {
  long long need = (work_items + threads - 1) / threads;
  long long cap = (long long)mtb_sm_count() * ctas_per_sm;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

static inline bool mtb_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
