// Host-side helpers shared by the entry points: status codes, last-error text,
// and construction of TMA tensor maps through the driver entry point (the
// library links only against the CUDA runtime).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/kfold_b200.h"

namespace kfb {

void set_error(const char* fmt, ...);
const char* get_error();

#define KFB_CHECK_ARG(cond, ...)        \
  do {                                  \
    if (!(cond)) {                      \
      ::kfb::set_error(__VA_ARGS__);    \
      return KFB_ERR_INVALID_ARGUMENT;  \
    }                                   \
  } while (0)

#define KFB_CUDA(expr)                                                                   \
  do {                                                                                   \
    cudaError_t e_ = (expr);                                                             \
    if (e_ != cudaSuccess) {                                                             \
      ::kfb::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
      return KFB_ERR_CUDA;                                                               \
    }                                                                                    \
  } while (0)

#define KFB_TRY(expr)            \
  do {                           \
    int s_ = (expr);             \
    if (s_ != KFB_OK) return s_; \
  } while (0)

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// Launch accounting.  Every kernel launch goes through a LaunchScope: it bumps the global launch
// counter and, while profiling is enabled, brackets the launch with CUDA events on its stream.
struct LaunchScope {
  LaunchScope(cudaStream_t stream, const char* tag);
  ~LaunchScope();
  cudaStream_t stream_;
  int slot_;
};

long long launch_count();
void profile_enable(bool on);
int profile_report(char* buf, size_t cap);

int sm_count();  // multiprocessors of the current device (cached per device)

// Launches `kernel`; a grid of at most one block per SM (or four, where blocks are light or fill an SM each) with programmatic
// stream serialisation: it may be scheduled while the kernel before it on the stream drains, so its start-up (block scheduling,
// barrier and tensor-memory set-up) runs under that kernel's tail.  Other grids are launched plainly: their first blocks would
// be packed onto the SMs that drain first and stay there (measured: the float32 channel-major LayerNorm, 200 blocks of 64 KB,
// 310 -> 454 us; the bf16 LayerNorm of a 768-token pair tensor 152 -> 187 us).
// Every kernel launched this way executes griddepcontrol.wait before it touches memory that the stream's earlier work wrote or
// reads, and griddepcontrol.launch_dependents only after that wait: what lies two or more kernels back is then always complete.
// Such a kernel has no __restrict__ pointer and reads nothing through __ldg or ld.global.nc: both promise that nobody else writes the
// data while the kernel lives, which the launch before it does until the wait, and the compiler may then move the loads ahead of the
// wait (it did: the rows of adaln_vec_kernel).  What the promise gave, loads that overtake earlier stores, is written out where it
// matters: a row's loads stand before its first store.
// cluster: CTAs per thread-block cluster (along x).
template <typename... KArgs, typename... Args>
inline int launch_kernel_clustered(cudaStream_t stream, void (*kernel)(KArgs...), unsigned cluster, dim3 grid, dim3 block, size_t smem,
                                   Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  const unsigned long long blocks = static_cast<unsigned long long>(grid.x) * grid.y * grid.z, sms = sm_count();
  if (blocks <= sms || (blocks <= 4 * sms && (smem <= 4096 || smem > 114 * 1024))) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  KFB_CUDA(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...));
  return KFB_OK;
}
template <typename... KArgs, typename... Args>
inline int launch_kernel(cudaStream_t stream, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args&&... args) {
  return launch_kernel_clustered(stream, kernel, 1, grid, block, smem, static_cast<Args&&>(args)...);
}

// Clusters of `cluster` CTAs of a kernel that the current device holds at once, after it has been allowed its shared memory; 0 where the device,
// or the part of one that this process may use, holds none or does not say.  (Only a failure of the question itself is cleared: an error that
// the caller has pending is the caller's.)  A call of some us: whoever asks keeps the answer for each device.
template <typename... KArgs>
inline int clusters_held(void (*kernel)(KArgs...), unsigned cluster, int threads, size_t smem) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = sm_count() / static_cast<int>(cluster) * static_cast<int>(cluster);
  cfg.blockDim = threads;
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int held = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&held, kernel, &cfg) == cudaSuccess)
    return held;
  cudaGetLastError();
  return 0;
}

#ifdef __CUDACC__
// (see launch_kernel)
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The start of every kernel that has nothing to do before its inputs: wait, then let the next kernel's blocks in -- at once when
// the grid is small (its time is latency, which the overlap hides), otherwise as this grid's blocks exit.  The line is two blocks
// for each of a B200's 148 multiprocessors, a constant where the host's rules ask sm_count(): reading %nsmid here cost 0.1 us a
// launch (64-token pair block 178.8 -> 182.6 us), and where a part has fewer only the time of grids near the line moves.
static constexpr unsigned kEarlyGrid = 2 * 148;
__device__ __forceinline__ void grid_dependency_enter() {
  grid_dependency_wait();
  if (gridDim.x * gridDim.y * gridDim.z <= kEarlyGrid) grid_dependency_launch();
}
#endif

// Encode a tiled tensor map.  dims/strides are given innermost first; strides[i] is the
// byte stride of dimension i+1 (dimension 0 is contiguous).  elem_bytes is 2 (bf16) or 4 (fp32).
// swizzle_bytes in {0, 32, 64, 128}: the inner box extent in bytes must equal it when non-zero.
int make_tmap(CUtensorMap* out, const void* base, int elem_bytes, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, int swizzle_bytes);

}  // namespace kfb
