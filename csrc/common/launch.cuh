// Kernel launch helper with programmatic dependent launch.
//
// Every kernel of the training step starts with pdl_launch_dependents() and runs pdl_wait() before
// its first access to global memory. Launched through launch_kernel(..., /*pdl=*/true), the next
// kernel in the stream may then be scheduled onto SMs as the CTAs of the current one retire, run
// its prologue (barrier initialisation, tensor-memory allocation, descriptor prefetch) and park in
// pdl_wait() until the current kernel has completed and its memory is visible. Inside a captured
// CUDA graph the launches become programmatic dependency edges. What is gained is the launch
// latency and the prologue of every kernel at each of the ~310 boundaries of a micro-step.
// Measured inside CUDA graphs (two runs each way on one box, the runs of one side 0.3 % apart): a training
// step of the 2-layer, 128-wide model 503 -> 488 us, of the 124M model 35.1 -> 34.7 ms, of the 350M model
// 50.0 -> 49.3 ms. Evaluations, replays of both graphs in turn: 16 x 512 tokens 3.04 -> 2.91 ms (124M), 8 x 1024
// 3.13 -> 3.02, 4 x 1024 1.77 -> 1.67, 16 x 1024 5.70 -> 5.68; of 512 to 2,048 tokens between 4.9 % slower and 10 %
// faster. (An earlier state of the kernels was 0.8 % slower with it.) So the engine asks for it, through the
// launching thread's pdl_scope, for training steps and for evaluations of 4096 tokens and more
// (PDL_EVAL_TOKENS); elsewhere it is off.
// Z2H_PDL=1 or 0 in the environment decides for all launches.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdlib>

namespace z2h {

// cudaFuncAttributeMaxDynamicSharedMemorySize (and the SM count) belong to a (kernel, device)
// pair, not to the process: a host program that drives several GPUs from one process must set
// them once per device. `seen` is a per-call-site bit mask of devices already configured; the
// function returns true exactly once per device (devices 64 and up are configured every time).
inline bool first_use_on_current_device(std::atomic<unsigned long long>& seen, int* device = nullptr) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (device != nullptr) *device = dev;
  if (dev < 0 || dev >= 64) return true;
  const unsigned long long bit = 1ull << dev;
  return (seen.fetch_or(bit) & bit) == 0;
}

// Number of SMs of the current device (cached per device).
inline int sm_count_current_device() {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  const bool cached = dev >= 0 && dev < 64;
  int n = cached ? cache[dev].load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (cached) cache[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// What the current thread asked for (z2h_pdl_scope); other threads' launches are not affected.
inline thread_local int pdl_scope = 0;

inline bool pdl_enabled() {
  static const int env = [] {
    const char* e = std::getenv("Z2H_PDL");
    return e == nullptr || e[0] == 0 ? -1 : (e[0] == '1' ? 1 : 0);
  }();
  return env >= 0 ? env == 1 : pdl_scope != 0;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t stream, bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  int n = 0;
  if (pdl && pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace z2h
