// Host helpers of the launch wrappers.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace umcp {

inline int grid_for(int n, int per_block) {
  int g = (n + per_block - 1) / per_block;
  return g < 1 ? 1 : g;
}

// A value fixed per device and computed once on it (thread-safe: meshes may
// be made on several threads). cudaFuncSetAttribute applies to the current
// device only, and the persistent grids follow each device's SM count, so
// neither may be shared between the devices of one process.
constexpr int kMaxDevices = 64;
// Launch with programmatic stream serialization: the kernel may be scheduled
// while the kernel before it on the stream drains, and waits for it in
// grid_dependency_wait (which it calls before reading that kernel's results).
template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

struct PerDevice {
  std::once_flag once[kMaxDevices];
  int value[kMaxDevices] = {};
};
template <class F>
inline int per_device(PerDevice &pd, F make) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDevices) return make();
  std::call_once(pd.once[dev], [&] { pd.value[dev] = make(); });
  return pd.value[dev];
}
inline int sm_count() {
  static PerDevice pd;
  return per_device(pd, [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  });
}


}  // namespace umcp
