// per_context.h -- what the launchers find out or set once per CUDA context.
//
// A kernel's shared-memory limit and its occupancy belong to the device that was
// current when they were set or asked: on a second device of the process a
// launch above 48 KB is refused until the limit is raised there too.  Contexts
// stand for devices here, so that a reset device counts as another one.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace dmg {

// Identity of the current CUDA context, unique for the life of the process
// (cuCtxGetId); 0 where it cannot be asked.
inline unsigned long long context_id() {
  using Fn = int (*)(void* ctx, unsigned long long* id);
  static const Fn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<Fn>(p);
  }();
  unsigned long long id = 0;
  return fn && fn(nullptr, &id) == 0 ? id : 0;
}

// One value per context, found by `find(&value)` when the context is not the
// one that it was last found in.  A failure is returned and not kept.
class PerContext {
 public:
  template <typename F>
  cudaError_t get(F&& find, int* value = nullptr) {
    const unsigned long long id = context_id();
    std::lock_guard<std::mutex> lock(mu_);
    if (id == 0 || id != id_) {
      int v = 0;
      const cudaError_t e = find(&v);
      if (e != cudaSuccess) return e;
      id_ = id;
      value_ = v;
    }
    if (value) *value = value_;
    return cudaSuccess;
  }

 private:
  std::mutex mu_;
  unsigned long long id_ = 0;
  int value_ = 0;
};

}  // namespace dmg
