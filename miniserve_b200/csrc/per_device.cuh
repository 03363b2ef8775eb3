// What a process learns of, or asks of, each of its devices once. Host code alone, so that it can be tested without a GPU.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

namespace ms {

constexpr int KNOWN_DEVICES = 64;  // (of a device beyond these everything is asked each time)

// Multiprocessors of the calling thread's device (0 if it cannot be had: only the choice of a form hangs on it).
inline int sm_count() {
  static std::atomic<int> known[KNOWN_DEVICES] = {};
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 0;
  if (dev < KNOWN_DEVICES && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (dev < KNOWN_DEVICES) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Lets `kernel` have `bytes` of dynamic shared memory on the calling thread's device: the attribute belongs to a device. `allowed`: a bit for
// each device that said yes, the caller's, one per kernel; a refusal is asked again the next time.
inline cudaError_t allow_shared_memory(const void* kernel, int bytes, std::atomic<unsigned long long>& allowed) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  const bool known = dev >= 0 && dev < KNOWN_DEVICES;
  if (known && ((allowed.load(std::memory_order_relaxed) >> dev) & 1ull)) return cudaSuccess;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess && known) allowed.fetch_or(1ull << dev, std::memory_order_relaxed);
  return err;
}

}  // namespace ms
