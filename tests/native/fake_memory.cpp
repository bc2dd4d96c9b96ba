// cudaMalloc and cudaFree of a library linked with --wrap=cudaMalloc and
// --wrap=cudaFree: a budget on the bytes it holds on the device, above which
// an allocation fails as it does when the device is full.
#include <cstddef>
#include <map>
#include <mutex>

#include <cuda_runtime.h>

extern "C" {
cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __real_cudaFree(void* p);

static std::mutex mtx;
static std::map<void*, size_t> held;
static size_t total = 0, peak = 0, budget = ~static_cast<size_t>(0);

cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> lock(mtx);
  if (n > budget - total) return cudaErrorMemoryAllocation;
  const cudaError_t e = __real_cudaMalloc(p, n);
  if (e == cudaSuccess) {
    held[*p] = n;
    total += n;
    if (total > peak) peak = total;
  }
  return e;
}

cudaError_t __wrap_cudaFree(void* p) {
  std::lock_guard<std::mutex> lock(mtx);
  const auto it = held.find(p);
  if (it != held.end()) {
    total -= it->second;
    held.erase(it);
  }
  return __real_cudaFree(p);
}

size_t fake_memory_held() { return total; }
size_t fake_memory_peak() {  // the most held since the last call
  const size_t most = peak;
  peak = total;
  return most;
}
void fake_memory_more(size_t n) { budget = total + n; }  // what may still be allocated
}
