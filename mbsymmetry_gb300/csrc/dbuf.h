// Device buffer helper and the host-side bounds check of the work lists.
#pragma once

#include <atomic>
#include <string>
#include <vector>

#include "common.h"

namespace gwgb {

// Device bytes held by the buffers of every live handle in this process.
extern std::atomic<int64_t> g_device_bytes;
// Test hook (gwgb_test_fail_alloc): this thread's device allocations first, first + 1, ... fail, `count` of them.
struct FailAlloc {
  int32_t first = 0, count = 0;
};
extern thread_local FailAlloc g_fail_alloc;

template <typename T>
struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  void alloc(size_t count) {
    free();
    if (!count) return;
    if (FailAlloc &f = g_fail_alloc; f.count > 0 && --f.first <= 0) {
      --f.count;
      throw Error(GWGB_E_NOMEM, "device allocation failed (test hook)");
    }
    const cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();  // or the next kernel launch would report it
    }
    GWGB_CUDA(e);
    n = count;
    g_device_bytes += (int64_t)(n * sizeof(T));
  }
  void upload(const std::vector<T> &v, cudaStream_t st) {
    alloc(v.size());
    if (n) GWGB_CUDA(cudaMemcpyAsync(p, v.data(), n * sizeof(T), cudaMemcpyHostToDevice, st));
  }
  void free() {
    if (p) cudaFree(p);
    g_device_bytes -= (int64_t)(n * sizeof(T));
    p = nullptr;
    n = 0;
  }
};

// Host-side bounds check of one work item: [begin, begin + len) must lie in a
// buffer of `size` elements.  Every task list is checked when it is built, so
// no kernel launch can read or write outside its buffers whatever the layout.
inline void check_range(int64_t begin, int64_t len, int64_t size, const char *what) {
  if (begin < 0 || len < 0 || begin + len > size)
    throw Error(GWGB_E_INVALID, std::string("internal work list out of bounds: ") + what);
}

}  // namespace gwgb
