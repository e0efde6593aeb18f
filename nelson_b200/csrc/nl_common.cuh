// nl_common.cuh -- shared device helpers for the nelson_b200 CUDA library.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>

#include "../../include/nelson_b200.h"

namespace nl {

// Padded element strides of the per-block Hessian storage.  Blocks are
// row-major and padded to a multiple of 16 bytes so they move as 16-byte
// vectors.
template <typename T>
__host__ __device__ constexpr int pad16(int n) {
  return ((n * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T);
}
template <typename T, int BC>
struct Layout {
  static constexpr int W = pad16<T>(BC * 3);   // W / Y (= W V^-1) block, BC x 3
  static constexpr int U = pad16<T>(BC * BC);  // U block, BC x BC
  static constexpr int V = pad16<T>(9);        // V / V^-1 block, 3 x 3
};

// Host-side NVTX range over the enqueue of one phase (named like the phases
// of SolverCholeskySchurIterationTimeStat, nelson/SolverCholeskySchur.h:25-38),
// so a profiler timeline groups each phase's kernel launches.  Costs nothing
// when no tool is attached.
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// Device-side error / status word bits (nl_status in the C ABI).
enum : int {
  ST_VINV_FAIL = 1,      // a damped 3x3 point block was not positive definite
  ST_CHOL_FAIL = 2,      // a pivot of the reduced camera system was <= 0 or not finite
  ST_SPIN_TIMEOUT = 4,   // a bounded wait between blocks gave up
  ST_NONFINITE = 8,      // a non-finite cost or increment was produced
};

// Deterministic block reduction of one double: every thread passes its value,
// thread 0 gets the total (warp shuffles then a fixed-order sum over warps).
template <int NT>
__device__ inline double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NT / 32; i++) s += sh[i];
  }
  __syncthreads();
  return s;
}

// Programmatic dependent launch: a kernel lets the next one in its stream launch at
// its start, and waits for its predecessor's completion (and memory flush) before
// touching what that predecessor wrote.  Both are no-ops for a kernel launched
// without the attribute.  A kernel launched with it (launch_next) waits in every
// thread before anything else, also where it then has nothing to do: its completion
// tells the next one that all before it have completed.
__device__ inline void chain_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ inline void chain_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Start of a kernel of launch_next.  The release follows the wait: one kernel at most
// waits on the chip (with more, the shared memory they hold comes out of the running
// kernel's L1: the cost pass took 20 instead of 11 us).
// The pointers given are those through which the kernel only reads what preceding
// kernels wrote: their values count from here on, so that the compiler, which may take
// the data of a restricted read-only pointer as constant over the whole kernel, reads
// nothing of it before the wait.
template <typename... P>
__device__ __forceinline__ void chain_start(P&... p) {
  chain_wait();
  chain_release();
  (..., [](P& q) {
    unsigned long long v = (unsigned long long)q;
    asm volatile("" : "+l"(v)::"memory");
    q = (P)v;
  }(p));
}

// Launches `kern`, which begins with chain_start(); with pdl as a programmatic
// dependent of the stream's preceding kernel (0.6 us from one small kernel's end to
// the next one's start, 1.8 us without), in clusters of `cluster` CTAs.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_cluster(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t st, bool pdl,
                                  int cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (pdl) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = cluster;
    at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
    n++;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_next(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t st, bool pdl,
                               Args... args) {
  return launch_cluster(kern, grid, block, smem, st, pdl, 1, args...);
}

// True for all threads of the block of a launch that finishes last (`count`
// starts at zero and is left at zero): that block can read what the others
// wrote before the call.  Replaces a second launch for the final reduction.
__device__ inline bool last_block(int* count) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(count, 1) == (int)gridDim.x - 1;
    if (last) *count = 0;
  }
  __syncthreads();
  __threadfence();
  return last != 0;
}

// The N sums (shared memory) of CTA blockIdx.y of the gridDim.y that share item c:
// true for the CTA that finishes last, with the totals (added in CTA order) in
// `sum`.  `part`: gridDim.y x N per item; `count`: zero per item, left at zero.
template <int N, typename T>
__device__ inline bool item_total(T* sum, T* __restrict__ part, int* __restrict__ count, int c) {
  __shared__ int last;
  const int n = gridDim.y;
  if (n == 1) return true;
  part += (size_t)c * n * N;
  for (int i = threadIdx.x; i < N; i += blockDim.x) part[(size_t)blockIdx.y * N + i] = sum[i];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(count + c, 1) == n - 1;
    if (last) count[c] = 0;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    T s = (T)0;
    for (int y = 0; y < n; y++) s += __ldcg(part + (size_t)y * N + i);
    sum[i] = s;
  }
  __syncthreads();
  return true;
}

// Item of a thread where groups of `lanes` threads share one, `nt` threads per CTA
// (lanes divides nt).  Formed from the CTA's first item: the thread's number in the
// grid is lanes times as large and passes 2^31 where the items are far from it.
__host__ __device__ inline int group_item(unsigned block, int nt, int thread, int lanes) {
  return (int)(block * (unsigned)(nt / lanes)) + thread / lanes;
}

// CTAs per camera for a pass over a camera's observations with nt threads: enough for
// four CTAs per SM in all (three of the camera pass are resident, FP64 two; the
// rest start as those end), two rounds of work at least for each.
inline int ctas_per_camera(int nc, long long observations, int nt) {
  const long long avg = observations / (nc > 0 ? nc : 1), want = (4 * 148 + nc - 1) / (nc > 0 ? nc : 1);
  const long long n = want < avg / (2 * nt) ? want : avg / (2 * nt);
  return (int)(n < 1 ? 1 : n > 8 ? 8 : n);
}

__device__ inline double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ inline float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Left SO(3) increment exp(w) by Rodrigues' formula (FP64).
__device__ inline void so3_exp(const double* w, double* R) {
  const double th2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
  double A, B;
  if (th2 < 1e-8) {
    A = 1.0 - th2 / 6.0 + th2 * th2 / 120.0;
    B = 0.5 - th2 / 24.0 + th2 * th2 / 720.0;
  } else {
    const double th = sqrt(th2);
    double s, c;
    sincos(th, &s, &c);
    A = s / th;
    B = (1.0 - c) / th2;
  }
  const double K[9] = {0, -w[2], w[1], w[2], 0, -w[0], -w[1], w[0], 0};
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double k2 = K[i * 3 + 0] * K[0 * 3 + j] + K[i * 3 + 1] * K[1 * 3 + j] + K[i * 3 + 2] * K[2 * 3 + j];
      R[i * 3 + j] = A * K[i * 3 + j] + B * k2 + (i == j ? 1.0 : 0.0);
    }
}

}  // namespace nl
