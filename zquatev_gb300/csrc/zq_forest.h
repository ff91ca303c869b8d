// Batches of mid-size matrices (order above FOREST_MIN) on all SMs (zq_forest.cu).
#pragma once

#include <vector>

#include "zq_kernels.h"

namespace zq {

// Orders the forest takes: the persistent kernel's one-warp range (zq_batched.cu)
// stays with it, and above 256 the per-matrix path runs.
constexpr int FOREST_MIN = 33, FOREST_MAX = 256;

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
  ~BatchForest();
  int build(const std::vector<ForestItem>& items, cudaStream_t st);
  bool matches(const std::vector<ForestItem>& items) const { return items == items_; }
  bool empty() const { return items_.empty(); }
  int run(double2* D, double* eig, cudaStream_t st);
  const int* error_flag() const { return err_; }  // device: a bounded wait ran out
  size_t bytes() const { return bytes_; }
  void release();

 private:
  struct Chunk;                    // a part of the batch whose scratch fits at once
  std::vector<ForestItem> items_;
  std::vector<Chunk*> chunks_;
  void* dev_ = nullptr;
  size_t bytes_ = 0;
  int* err_ = nullptr;
};

}  // namespace zq
