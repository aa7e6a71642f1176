// fmgpu_internal.cuh -- shared definitions of the libfmgpu kernels and host code.
//
// Arithmetic contract of the FP64 path (compiled with -fmad=false, so the only
// fused multiply-adds are the explicit fma() calls):
//   row sum     acc = 0; for slot s ascending: acc = fma(a_s, x_{i+off_s}, acc)
//   residual    r_i = b_i - rowsum_i
//   reductions  DR4096: one 256-thread block per 4096-element chunk; thread t
//               owns chunk positions 2t+512m+u (m = 0..7, u = 0..1) in (m,u)
//               order; a warp butterfly then a butterfly over the 8 warp sums;
//               the last block folds the chunk sums (thread t: chunks
//               t, t+256, ... with plain adds) through the same tree.
// This fixed order makes the GPU results independent of scheduling and equal
// to a sequential restatement that follows the same order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <vector>

#include "../../include/fmgpu.h"

namespace fmg {

constexpr int kBlock = 256;                 // threads per chunk block
constexpr int kChunk = 4096;                // elements per reduction chunk
constexpr int kPairsPerThread = kChunk / (kBlock * 2);
constexpr int kMaxLevels = 16;

// kernels launched by this library in this process (diagnostics)
extern std::atomic<long long> g_launches;

// device scalar slots of a grid (CG scalars, reduction results)
enum Scal {
  S_ALPHA = 0, S_BETA, S_LAM, S_NEGLAM, S_NEWALPHA, S_RATIO, S_RR, S_DOT, S_TMP,
  S_MFERR = 15,         // non-zero: a matrix-free operator kernel gave up waiting for a copy
  S_COUNT = 16
};

// epilogue of a chunked reduction, run by the last block on the folded value
enum Epi { EPI_STORE = 0, EPI_CG_LAMBDA = 1, EPI_CG_ALPHA = 2 };

struct Reduce {         // scratch of one chunked reduction
  double* part;         // >= number of chunks
  unsigned* counter;    // zero between reductions (reset by the last block)
  double* scal;         // grid scalar slots
  int epi;              // Epi
  int slot;             // destination slot for EPI_STORE
};

__device__ __forceinline__ long long clampi(long long j, long long N) {
  return j < 0 ? 0 : (j >= N ? N - 1 : j);
}

// Warp butterfly then butterfly over the 8 warp sums; the result is valid in
// thread 0.  smem must hold 8 doubles.  Blocks of 256 threads, 1D or (32, 8).
__device__ __forceinline__ double dr_fold256(double v, double* smem) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, o);
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;  // blocks of 256 threads, 1D or 2D
  const int warp = tid >> 5, lane = tid & 31;
  __syncthreads();  // smem may still be read by a previous fold
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  double w = 0.0;
  if (warp == 0) {
    w = lane < 8 ? smem[lane] : 0.0;
    w = w + __shfl_xor_sync(0xffffffffu, w, 4);
    w = w + __shfl_xor_sync(0xffffffffu, w, 2);
    w = w + __shfl_xor_sync(0xffffffffu, w, 1);
  }
  return w;
}

// Chunk partial -> global; the last block to finish folds all partials and
// applies the epilogue.  Must be called by all threads of a 256-thread block
// whose blockIdx.x is the chunk index and gridDim.x the chunk count.
__device__ __forceinline__ void dr_finish(double lane_sum, const Reduce& R, double* smem) {
  __shared__ bool is_last;
  double s = dr_fold256(lane_sum, smem);
  if (threadIdx.x == 0) {
    R.part[blockIdx.x] = s;
    __threadfence();
    unsigned done = atomicAdd(R.counter, 1u);
    is_last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  double acc = 0.0;
  for (unsigned k = threadIdx.x; k < gridDim.x; k += kBlock) acc = acc + __ldcg(R.part + k);
  double tot = dr_fold256(acc, smem);
  if (threadIdx.x == 0) {
    double* sc = R.scal;
    switch (R.epi) {
      case EPI_CG_LAMBDA: {            // beta = (a,p); lam = alpha/beta
        double lam = sc[S_ALPHA] / tot;
        sc[S_BETA] = tot; sc[S_LAM] = lam; sc[S_NEGLAM] = -lam;
        break;
      }
      case EPI_CG_ALPHA: {             // new alpha = (q,r); ratio = new/alpha
        sc[S_NEWALPHA] = tot;
        sc[S_RATIO] = tot / sc[S_ALPHA];
        sc[S_ALPHA] = tot;
        break;
      }
      default: sc[R.slot] = tot;
    }
    *R.counter = 0u;
  }
}

// Programmatic dependent launch: a kernel launched with launch_early or
// launch_pdl (on a small grid) may start while its predecessor in the stream
// still runs.  pdl_next lets the successor start; pdl_wait waits until the
// predecessor has finished and its writes are visible.  Every kernel launched
// so calls pdl_next (or pdl_next_light) and pdl_wait, pdl_wait before its first access to anything that a kernel
// of the same sequence writes; before it, only what was in place when the
// sequence began (matrices, damping, factors, indices) is read.  __ldg and
// `const T* __restrict__` (which lets the compiler use it) are for those alone:
// the read-only path is defined for data nobody writes while the kernel lives,
// and a kernel started early lives while its predecessor still writes vectors
// and scalars.  They are read by plain loads from unrestricted pointers, which
// neither the compiler nor the caches serve from before the wait.  At least one
// thread of every launch passes pdl_wait, so a launch never ends before its
// predecessor and waiting for one kernel is waiting for all before it.
constexpr unsigned kPdlBlocks = 148;  // a small grid: at most a block per SM
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Letting the successor start takes a block's turn at issuing: on a large grid
// of blocks that do a few accesses a thread it is 40 % of their time (FP64 to
// FP32 of 2^27 elements 383 us, 541 so; 2^22 12.4 and 19.4), and such blocks end
// as soon as they could tell.  On small grids their successors gain by it (a
// 64^2-cell solve 787 us, 795 without).
__device__ __forceinline__ void pdl_next_light() {
  if (gridDim.x * gridDim.y * gridDim.z <= kPdlBlocks) pdl_next();
}

// The stream this thread's last such launch went to.  A sequence begins with a
// launch that waits for everything before it (the first one on a stream, and
// the first after launched(), which follows whatever writes a matrix, damping
// or factors); the launches after it overlap their starts (2-4 us a launch on
// small levels instead of 4-6).
extern thread_local cudaStream_t t_pdl_stream;
inline void pdl_break() { t_pdl_stream = nullptr; }

// Which launches overlap was measured kernel by kernel: kernels that fetch
// before they wait and light streaming ones gain at every size (launch_early);
// register- and cache-heavy ones that only wait gain on small grids and lose
// on large ones (launch_pdl: Q2 residual among the SOR sweeps of 129^3 nodes,
// 31.9 -> 34.9 ms a solve with all launches early; FCG update of 97^3 nodes,
// 3.83 -> 4.07 ms), and the elasticity rows lose always (launch_late).
template <typename... KA, typename... A>
inline void launch_after(bool early, void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                         A... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = early && t_pdl_stream == st ? 1 : 0;
  t_pdl_stream = st;
  cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...);
}
template <typename... KA, typename... A>
inline void launch_early(void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  launch_after(true, kern, grid, block, smem, st, args...);
}
template <typename... KA, typename... A>
inline void launch_pdl(void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  launch_after((long long)grid.x * grid.y * grid.z <= kPdlBlocks, kern, grid, block, smem, st, args...);
}
template <typename... KA, typename... A>
inline void launch_late(void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  launch_after(false, kern, grid, block, smem, st, args...);
}

inline unsigned nchunks(long long n) { return (unsigned)((n + kChunk - 1) / kChunk); }

}  // namespace fmg
