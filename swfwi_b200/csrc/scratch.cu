// Scratch of calls that return synchronised (common.hpp).
//
// cudaMalloc and cudaFree take about 0.35 and 0.3 ms here whatever the size,
// a third of an ensemble analysis of 64 members.  So one buffer per CUDA
// context, of at most kKeepBytes, is kept between such calls; a second
// concurrent call allocates its own, and an allocation of this library that
// finds the device full frees the kept ones before it gives up.
#include <cuda.h>
#include <mutex>
#include <vector>
#include "common.hpp"

namespace swfwi {
namespace {

constexpr size_t kKeepBytes = 32u << 20;

struct Kept {
  int dev;
  unsigned long long ctx;
  void *p;
  size_t bytes;
};
std::mutex g_mu;
std::vector<Kept> g_kept;   // at most one a context

// The current context's id, unique in the process (a context made after
// cudaDeviceReset has another); 0: none could be had, nothing is kept.
unsigned long long context_id() {
  using Fn = CUresult (*)(CUcontext, unsigned long long *);
  static const Fn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool ok = cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
                    q == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<Fn>(p) : nullptr;
  }();
  unsigned long long id = 0;
  return fn && fn(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

}  // namespace

Scratch::Scratch(size_t bytes) {
  SWFWI_CUDA(cudaGetDevice(&dev_));
  ctx_ = context_id();
  if (ctx_) {
    std::lock_guard<std::mutex> g(g_mu);
    for (size_t i = 0; i < g_kept.size(); i++)
      if (g_kept[i].ctx == ctx_ && g_kept[i].bytes >= bytes) {
        p_ = g_kept[i].p;
        bytes_ = g_kept[i].bytes;
        g_kept.erase(g_kept.begin() + i);
        return;
      }
  }
  p_ = device_alloc(bytes);
  bytes_ = bytes;
}

Scratch::~Scratch() {
  void *drop = p_;
  if (idle_ && ctx_ && bytes_ <= kKeepBytes) {
    std::lock_guard<std::mutex> g(g_mu);
    Kept *mine = nullptr;
    for (Kept &k : g_kept)
      if (k.ctx == ctx_) mine = &k;
    try {
      if (!mine) {
        // contexts this device had before are gone, and their memory with them
        for (size_t i = g_kept.size(); i-- > 0;)
          if (g_kept[i].dev == dev_) g_kept.erase(g_kept.begin() + i);
        g_kept.push_back({dev_, ctx_, p_, bytes_});
        drop = nullptr;
      } else if (mine->bytes < bytes_) {
        drop = mine->p;
        mine->p = p_;
        mine->bytes = bytes_;
      }
    } catch (...) {
    }
  }
  if (drop) cudaFree(drop);
}

void *device_alloc(size_t bytes) {
  void *p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaErrorMemoryAllocation && release_kept_scratch()) {
    cudaGetLastError();
    e = cudaMalloc(&p, bytes);
  }
  SWFWI_CUDA(e);
  return p;
}

bool release_kept_scratch() {
  const unsigned long long ctx = context_id();
  void *p = nullptr;
  {
    std::lock_guard<std::mutex> g(g_mu);
    for (size_t i = 0; i < g_kept.size(); i++)
      if (ctx && g_kept[i].ctx == ctx) {
        p = g_kept[i].p;
        g_kept.erase(g_kept.begin() + i);
        break;
      }
  }
  if (p) cudaFree(p);
  return p != nullptr;
}

}  // namespace swfwi
