// Batches of mid-size matrices on all SMs (zq_forest.cu).
#pragma once

#include <vector>

#include "zq_common.cuh"
#include "zq_kernels.h"

namespace zq {

constexpr int SMALL_MAX = 32;  // largest order a warp solves (zq_small.cu)
// Which matrices of a batch the forest takes: orders 33 to 256 always (above, the
// per-matrix path runs). Orders up to 32 have a warp each (zq_small.cu); where a batch
// has so few of them that a warp's serial chain shows, the forest is sooner from order
// 16 up: 60 matrices take 0.57 ms here and 1.0 ms there at n = 19, 0.92 and 2.6 ms at
// n = 32, but 0.28 and 0.26 ms at n = 8, and 2000 of n = 19 take 9.9 and 2.1 ms.
constexpr int FOREST_FEW = 128;
inline bool forest_takes(int n, int small_count) {
  return n > SMALL_MAX || (small_count <= FOREST_FEW && n >= 16);
}
// small_count: the matrices of order 1 to SMALL_MAX
inline int forest_small_count(int count, const int* n2s) {
  int k = 0;
  for (int b = 0; b < count; ++b) k += n2s[b] > 0 && n2s[b] / 2 <= SMALL_MAX;
  return k;
}

struct ForestItem {
  int n, ld;
  long long off, eoff;  // complex offset of the matrix, offset of its eigenvalues
  bool operator==(const ForestItem& o) const { return n == o.n && ld == o.ld && off == o.off && eoff == o.eoff; }
};

// One batch layout and its device memory. Items are kept in the order given
// (largest first). Not thread-safe; run() must not overlap an earlier run()
// of the same object on another stream.
class BatchForest {
 public:
  // pooled: the device memory comes from the device's stream-ordered pool, in the order
  // of the stream given to build(), instead of cudaMalloc
  explicit BatchForest(bool pooled = false) : pooled_(pooled) {}
  ~BatchForest();
  BatchForest(const BatchForest&) = delete;
  BatchForest& operator=(const BatchForest&) = delete;
  int build(const std::vector<ForestItem>& items, cudaStream_t st);
  bool matches(const std::vector<ForestItem>& items) const { return items == items_; }
  // build()'s code where the batch cannot run jointly (no room for its scratch, no cluster
  // for its largest order) but one matrix per CTA still can (zq_batched.cu)
  static bool declined(int rc) { return rc == ZQ_ERR_NOMEM || rc == ZQ_ERR_LIMIT; }
  bool empty() const { return items_.empty(); }
  int run(double2* D, double* eig, cudaStream_t st);
  // device, an int per item in the order given: the last run's count of its eigenvalues that are
  // not finite (its QL would not have converged)
  const int* info() const { return info_; }
  int count() const { return (int)items_.size(); }
  size_t bytes() const { return bytes_; }
  void release();

 private:
  int reserve(size_t bytes, cudaStream_t st);
  void drop();
  struct Chunk;                    // a part of the batch; the parts run one after another on the same scratch
  std::vector<ForestItem> items_;
  std::vector<Chunk*> chunks_;
  const bool pooled_;
  cudaStream_t st_ = nullptr;  // pooled: the memory's stream
  void* dev_ = nullptr;
  size_t bytes_ = 0;
  int* info_ = nullptr;
};

}  // namespace zq
