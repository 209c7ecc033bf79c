// Kernel launch with programmatic dependent launch (PDL) for the training step.
//
// A training update is ~5400 dependent kernels on one stream.  Launched normally, each waits for its
// predecessor to drain completely before its own CTAs are even scheduled, and then spends its first
// microseconds on set-up (barrier initialisation, TMEM allocation, descriptor prefetch).  With the
// programmatic-stream-serialization attribute a kernel's CTAs may be scheduled as soon as every CTA of
// the predecessor has executed `griddepcontrol.launch_dependents` (the kernels here do so right after
// their set-up) and an SM has room; the kernel runs its own set-up and then blocks in
// `griddepcontrol.wait`, which returns when the predecessor has completed and its writes are visible.
// Rule every kernel launched through this helper keeps: no global memory access before `pdl_wait()`, by the compiler's hand
// either (see `pdl_wait` on `__restrict__`).  The decode kernels have a launch helper and rules of their own (decode.cu):
// they request data that no launch in front of them writes before they wait.  So do products marked WsGemm::b_ahead.
// WS_TRAIN_PDL=0 launches normally.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>

namespace ws {

// SMs of the chip that these kernels are built for.  Where a grid or a rule counts on this number and not on the device's, it decides how sums are
// divided (partial rows whose number callers compute), or a line was measured with it.
constexpr int CHIP_SMS = 148;

inline bool train_pdl_enabled() {
  static const bool enabled = [] {
    const char* e = std::getenv("WS_TRAIN_PDL");
    return e == nullptr || e[0] != '0';
  }();
  return enabled;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(bool dependent, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent && train_pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args... args) {
  return launch_kernel(true, kern, grid, block, smem, stream, args...);
}

// Allows KERNEL more shared memory than a launch has by default, once on each device of the process.
template <auto KERNEL>
inline bool allow_shared_memory(int bytes) {
  static std::atomic<unsigned long long> allowed{0};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device >= 64) return false;
  const unsigned long long bit = 1ull << device;
  if (allowed.load(std::memory_order_relaxed) & bit) return true;
  if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
  allowed.fetch_or(bit, std::memory_order_relaxed);
  return true;
}

}  // namespace ws
