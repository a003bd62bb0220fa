// A plan's device arrays: one allocation for all of them.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace hphi {

class PlanUpload {
 public:
  template <typename V>
  void add(const std::vector<V> &h, const V **d) {
    part_.push_back(Part{h.data(), sizeof(V) * h.size(), at_, (const void **)d});
    at_ += (std::max<size_t>(16, sizeof(V) * h.size()) + 255) / 256 * 256;
  }
  // The arrays' pointers are set; the allocation goes to *allocs.  -1: no device memory, or the copy failed.
  int run(std::vector<void *> *allocs) {
    void *q = nullptr;
    if (cudaMalloc(&q, std::max<size_t>(256, at_)) != cudaSuccess) return -1;
    allocs->push_back(q);
    std::vector<char> all;  // small plans go over in one copy
    if (at_ <= ((size_t)1 << 18)) all.resize(at_);
    for (const Part &p : part_) {
      *p.d = (char *)q + p.at;
      if (!all.empty() && p.bytes) std::memcpy(all.data() + p.at, p.h, p.bytes);
      if (all.empty() && p.bytes && cudaMemcpy((char *)q + p.at, p.h, p.bytes, cudaMemcpyHostToDevice) != cudaSuccess) return -1;
    }
    return all.empty() || cudaMemcpy(q, all.data(), all.size(), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
  }

 private:
  struct Part {
    const void *h;
    size_t bytes, at;
    const void **d;
  };
  std::vector<Part> part_;
  size_t at_ = 0;
};

}  // namespace hphi
