// Status codes, errors and a small device buffer type for the host layer.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>
#include "swfwi_gpu.h"

namespace swfwi {

struct Error : std::runtime_error {
  int status;
  Error(int s, const std::string &m) : std::runtime_error(m), status(s) {}
};

void set_last_error(const std::string &m);
std::string last_error();

inline void cuda_check(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    int st = (e == cudaErrorMemoryAllocation) ? SWFWI_ERR_OOM : SWFWI_ERR_CUDA;
    throw Error(st, std::string(what) + ": " + cudaGetErrorString(e));
  }
}

#define SWFWI_CUDA(call) ::swfwi::cuda_check((call), #call)
#define SWFWI_REQUIRE(cond, msg)                                  \
  do {                                                            \
    if (!(cond)) throw ::swfwi::Error(SWFWI_ERR_BAD_ARG, (msg));  \
  } while (0)

// Runs f, converting exceptions into a status code and a last-error text.
template <typename F>
int guarded(F &&f) {
  try {
    f();
    return SWFWI_OK;
  } catch (const Error &e) {
    set_last_error(e.what());
    return e.status;
  } catch (const std::bad_alloc &) {
    set_last_error("host allocation failed");
    return SWFWI_ERR_OOM;
  } catch (const std::exception &e) {
    set_last_error(e.what());
    return SWFWI_ERR_CUDA;
  }
}

// Lets a kernel's launches have `bytes` of dynamic shared memory.  The limit is
// the current device's (and its context's) own, so launches that need it ask
// each time; it takes a fraction of a microsecond.
template <typename K>
void allow_smem(K *kernel, size_t bytes) {
  SWFWI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

// cudaMalloc; if the device is full, once more without this context's kept
// scratch.
void *device_alloc(size_t bytes);
// Frees the scratch kept for the current context; false: there was none.
bool release_kept_scratch();

// Device scratch of a call that returns synchronised: taken from the buffer
// kept for the context if it is large enough and free, else allocated.  Once
// the work that uses it has ended the call says so by idle(), and the buffer
// may be kept; without that (an exception) it is freed, which waits.
class Scratch {
 public:
  explicit Scratch(size_t bytes);
  ~Scratch();
  Scratch(const Scratch &) = delete;
  Scratch &operator=(const Scratch &) = delete;
  void *get() const { return p_; }
  void idle() { idle_ = true; }

 private:
  int dev_ = 0;
  unsigned long long ctx_ = 0;
  void *p_ = nullptr;
  size_t bytes_ = 0;
  bool idle_ = false;
};

// A word of host memory that kernels can write, zero at first.  The words of a
// context share one page, which pinning costs a millisecond or two once.
// Whoever holds a word ends its work before giving it back.
class HostWord {
 public:
  HostWord();
  ~HostWord();
  HostWord(const HostWord &) = delete;
  HostWord &operator=(const HostWord &) = delete;
  int *get() const { return p_; }
  int value() const { return *static_cast<volatile int *>(p_); }
  void clear() { *static_cast<volatile int *>(p_) = 0; }

 private:
  int *p_ = nullptr;
  unsigned long long ctx_ = 0;   // context of its page
};

// Owning device allocation (cudaMalloc / cudaFree).
template <typename T>
class DevBuf {
 public:
  DevBuf() = default;
  explicit DevBuf(size_t n) { resize(n); }
  ~DevBuf() { release(); }
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  DevBuf(DevBuf &&o) noexcept : p_(o.p_), n_(o.n_), cap_(o.cap_) {
    o.p_ = nullptr;
    o.n_ = o.cap_ = 0;
  }
  DevBuf &operator=(DevBuf &&o) noexcept {
    if (this != &o) {
      release();
      p_ = o.p_; n_ = o.n_; cap_ = o.cap_;
      o.p_ = nullptr;
      o.n_ = o.cap_ = 0;
    }
    return *this;
  }
  // Grows the allocation when needed; shrinking keeps the capacity.
  void resize(size_t n) {
    if (n > cap_) {
      release();
      p_ = static_cast<T *>(device_alloc(n * sizeof(T)));
      cap_ = n;
    }
    n_ = n;
  }
  void release() {
    if (p_) cudaFree(p_);
    p_ = nullptr;
    n_ = cap_ = 0;
  }
  size_t capacity() const { return cap_; }
  T *get() const { return p_; }
  size_t size() const { return n_; }
  void upload(const T *h, size_t n, cudaStream_t st) {
    resize(n);
    if (n) SWFWI_CUDA(cudaMemcpyAsync(p_, h, n * sizeof(T), cudaMemcpyHostToDevice, st));
  }
  void upload(const std::vector<T> &h, cudaStream_t st) { upload(h.data(), h.size(), st); }
  void zero(cudaStream_t st) {
    if (n_) SWFWI_CUDA(cudaMemsetAsync(p_, 0, n_ * sizeof(T), st));
  }

 private:
  T *p_ = nullptr;
  size_t n_ = 0;
  size_t cap_ = 0;
};

}  // namespace swfwi
