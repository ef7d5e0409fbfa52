// A smaller GPU, as far as stream-ordered allocations go: loaded before the CUDA
// runtime it counts what is allocated and answers cudaErrorMemoryAllocation
// beyond a limit.  Nothing reaches the device that would not have otherwise.
#include <dlfcn.h>

#include <map>
#include <mutex>

namespace {
std::mutex mu;
std::map<void*, size_t> blocks;
size_t live = 0, peak = 0, limit = ~size_t(0);
template <typename F>
F real(const char* name) {
  void* rt = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return reinterpret_cast<F>(dlsym(rt, name));
}
}  // namespace

extern "C" {
int cudaMallocAsync(void** p, size_t n, void* stream) {
  static auto call = real<int (*)(void**, size_t, void*)>("cudaMallocAsync");
  std::lock_guard<std::mutex> lock(mu);
  if (live + n > limit) return 2;  // cudaErrorMemoryAllocation
  const int e = call(p, n, stream);
  if (e == 0) {
    blocks[*p] = n;
    live += n;
    if (live > peak) peak = live;
  }
  return e;
}
int cudaFreeAsync(void* p, void* stream) {
  static auto call = real<int (*)(void*, void*)>("cudaFreeAsync");
  std::lock_guard<std::mutex> lock(mu);
  auto it = blocks.find(p);
  if (it != blocks.end()) {
    live -= it->second;
    blocks.erase(it);
  }
  return call(p, stream);
}
void low_memory_limit(size_t n) { limit = n; }
size_t low_memory_live() { return live; }
size_t low_memory_peak(int reset) {
  const size_t v = peak;
  if (reset) peak = live;
  return v;
}
}
