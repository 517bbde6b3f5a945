// Numbers of the current device that launch rules depend on, asked for once
// per device and kept in atomics, so that several threads may ask at once.
#ifndef JB_DEVICE_H
#define JB_DEVICE_H
#include <atomic>

#include <cuda_runtime.h>

namespace jb {

struct PerDevice {
  std::atomic<int> v[64];  // value + 1, 0: not asked yet

  // The current device's number; ask(device) is called at its first use.
  template <class Ask>
  int get(Ask ask) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    if (dev < 0 || dev >= 64) return ask(dev);
    int n = v[dev].load(std::memory_order_relaxed);
    if (!n) {
      n = ask(dev) + 1;
      v[dev].store(n, std::memory_order_relaxed);
    }
    return n - 1;
  }
};

static inline int sm_count() {
  static PerDevice known;
  return known.get([](int dev) {
    int n = 0;
    return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 1;
  });
}

}  // namespace jb

#endif  // JB_DEVICE_H
