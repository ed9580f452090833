// Scratch of calls that return synchronised (common.hpp).
//
// cudaMalloc and cudaFree take about 0.35 and 0.3 ms here whatever the size,
// a third of an ensemble analysis of 64 members.  So one buffer per CUDA
// context, of at most kKeepBytes, is kept between such calls; a second
// concurrent call allocates its own, and an allocation of this library that
// finds the device full frees the kept ones before it gives up.  Below it, the
// page of host words of a context.
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

namespace {

constexpr int kPageWords = 1024;   // 4 KB
struct Page {
  int dev;
  unsigned long long ctx;   // 0: a page of its own, freed with its word
  int *base;
  std::vector<int> free;    // word numbers not held
};
std::vector<Page> g_pages;

int *pinned(size_t words) {
  void *p = nullptr;
  SWFWI_CUDA(cudaHostAlloc(&p, words * sizeof(int), cudaHostAllocMapped));
  return static_cast<int *>(p);
}

}  // namespace

HostWord::HostWord() {
  int dev = 0;
  SWFWI_CUDA(cudaGetDevice(&dev));
  const unsigned long long ctx = ctx_ = context_id();
  std::lock_guard<std::mutex> g(g_mu);
  Page *page = nullptr;
  for (Page &q : g_pages)
    if (ctx && q.ctx == ctx && !q.free.empty()) page = &q;
  if (!page) {
    // pages of contexts this device had before are gone with those; a word
    // held beyond them finds no page any more
    for (size_t i = g_pages.size(); ctx && i-- > 0;)
      if (g_pages[i].dev == dev && g_pages[i].ctx && g_pages[i].ctx != ctx) g_pages.erase(g_pages.begin() + i);
    Page q{dev, ctx, pinned(ctx ? kPageWords : 1), {}};
    for (int i = (ctx ? kPageWords : 1) - 1; i >= 0; i--) q.free.push_back(i);
    g_pages.push_back(std::move(q));
    page = &g_pages.back();
  }
  p_ = page->base + page->free.back();
  page->free.pop_back();
  *p_ = 0;
}

HostWord::~HostWord() {
  std::lock_guard<std::mutex> g(g_mu);
  for (size_t i = 0; i < g_pages.size(); i++) {
    Page &q = g_pages[i];
    if (q.ctx != ctx_ || p_ < q.base || p_ >= q.base + (q.ctx ? kPageWords : 1)) continue;
    if (!q.ctx) {
      cudaFreeHost(q.base);
      g_pages.erase(g_pages.begin() + i);
      return;
    }
    q.free.push_back((int)(p_ - q.base));   // room for it was there before
    // one page a context stays; others go when their last word does
    if ((int)q.free.size() == kPageWords)
      for (size_t j = 0; j < g_pages.size(); j++)
        if (j != i && g_pages[j].ctx == q.ctx) {
          cudaFreeHost(q.base);
          g_pages.erase(g_pages.begin() + i);
          break;
        }
    return;
  }
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
