// Launch-side helpers shared by every kernel file: return codes that keep the CUDA error they came from, and
// one-time kernel attribute set-up that is remembered per device.
//
// A launcher returns 0, a negative b2::StatusCode for a request it refuses before launching (kBadArgument,
// kTooLarge), or -(kCudaErrorBase + cudaError_t) when the CUDA runtime refused something: a launch under a stream
// capture that does not allow it, an attribute the device does not support, a sticky error left by earlier work.
// Folding all of these into kBadArgument would hide which one it was.
#pragma once
#include <atomic>
#include <cstdlib>
#include <utility>
#include <cuda_runtime.h>
#include "b2/config.h"
#include "b2/status.h"

namespace b2 {

constexpr int kCudaErrorBase = 1000;

inline int cuda_rc(cudaError_t e) { return e == cudaSuccess ? 0 : -(kCudaErrorBase + static_cast<int>(e)); }
// After a `<<<>>>` launch: 0, or the code of the error the launch left behind (which this call also clears).
inline int last_launch_rc() { return cuda_rc(cudaGetLastError()); }
// True when `rc` carries a cudaError_t; `cuda_error_of(rc)` recovers it.
inline bool is_cuda_rc(int rc) { return rc <= -kCudaErrorBase; }
inline cudaError_t cuda_error_of(int rc) { return static_cast<cudaError_t>(-rc - kCudaErrorBase); }

// Attributes set with cudaFuncSetAttribute belong to the (kernel, device) pair, so "done once" has to be kept per
// device: a process that drives two GPUs must set the attribute on each. `run(f)` calls f() (returning a
// cudaError_t) unless it already succeeded with the current device current; safe to call from several host threads
// (the worst case is that two of them both set the attribute).
class DeviceOnce {
 public:
  template <class F>
  int run(F&& f) {
    int dev = -1;
    const bool known = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices;
    if (known && done_[dev].load(std::memory_order_acquire)) return 0;
    const cudaError_t e = f();
    if (e != cudaSuccess) {
      cudaGetLastError();
      return cuda_rc(e);
    }
    if (known) done_[dev].store(1, std::memory_order_release);
    return 0;
  }
  // The usual case: opt one kernel into `bytes` of dynamic shared memory.
  template <class Kernel>
  int max_smem(Kernel kernel, int bytes) {
    return run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
  }

 private:
  static constexpr int kMaxDevices = 64;
  std::atomic<unsigned char> done_[kMaxDevices] = {};
};

// Programmatic dependent launch. A kernel launched through `launch_pdl` may be scheduled while the kernel before it in
// the stream is still running: its CTAs start, run whatever precedes their `ptx::grid_dep_wait()` (barrier and TMEM
// set-up in the GEMMs, nothing in the small kernels) and block there until the earlier kernel has completed and its
// writes are visible. That takes the launch latency, and for the tensor-core kernels the prologue, off the critical
// path of a step made of hundreds of short dependent kernels; stream capture records the same edges in a CUDA graph.
// Rules every kernel launched this way follows: (1) every thread executes grid_dep_wait() before its first global
// memory access and before any return; (2) `ptx::grid_dep_launch()` right after it lets the next kernel be scheduled.
// (`launch_beside`, below, is for the one exception.) A kernel without the wait must not be launched through any of the functions below: its predecessor has usually allowed it to
// start long before its own results are in memory. `<<< >>>` keeps stream order for such a kernel.
//
// Where it is used: launches of one wave (`launch_small`: at most four thread blocks per SM), the kernels of decode-sized steps, whose
// launch gap is a good part of their time. 13 steps of a one-request chat through eight layers of width 2048: 6.33 -> 5.68 ms; an
// expert layer of 5 rows: 100 -> 89 us. Not for larger launches (8B serving steps at one and two GPUs: 10.75 / 10.88 ms with it,
// 10.85 / 10.83 without) nor for the scans of recurrent layers, a few long thread blocks each: started early they gather on the SMs
// that fall free first (decode rows beside a prompt through gated linear attention: 119 -> 168 us). B2_PDL=1 / 0: every / no launch.
inline int pdl_mode() {
  static const int mode = [] {
    const char* e = std::getenv("B2_PDL");
    return e == nullptr ? -1 : e[0] == '1' ? 1 : 0;
  }();
  return mode;
}
inline bool pdl_enabled() { return pdl_mode() == 1; }
inline bool pdl_for_small(dim3 grid) {
  return pdl_mode() == 1 || (pdl_mode() != 0 && static_cast<long>(grid.x) * grid.y * grid.z <= 4 * kNumSMs);
}

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// `launch_pdl` for launches of one wave whatever B2_PDL says (0 excepted); larger ones are launched in order.
template <class... KArgs, class... Args>
inline cudaError_t launch_small(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for_small(grid) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// For a kernel that neither reads what the kernel before it writes nor writes what that one touches: it may run beside it, so it is
// launched programmatically whatever its size. It must not touch memory that a kernel further ahead still works on, so the one before it has to be launched in order
// or wait itself before it lets others start (grid_dep_sync does). The kernel does not wait at its beginning, but one of its blocks
// calls grid_dep_wait at its end: what comes after it, and waits for it alone, then also comes after the one before.
template <class... KArgs, class... Args>
inline cudaError_t launch_beside(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_mode() != 0 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// `launch_small` with `cluster` thread blocks (a divisor of the grid, at most 8) scheduled together on one GPC.
template <class... KArgs, class... Args>
inline cudaError_t launch_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_for_small(grid) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace b2
