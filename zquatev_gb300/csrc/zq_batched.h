// Batches of small matrices: the task table shared by the CTA-per-matrix kernel
// (zq_batched.cu) and the warp-per-matrix kernel (zq_small.cu).
#pragma once

#include <cuda_runtime.h>

#include "zq_context.h"

namespace zq {

struct BatchTask {
  long long off;    // complex offset of D (from the launch's D) when Dp is null
  long long eoff;   // offset of eig (from the launch's eig) when Ep is null
  double2* Dp;      // or the matrix itself (requests in separate allocations)
  double* Ep;
  int n, ld;
  int out_slot;     // index into the info array
  int pad;
};

// tasks[0..count), each of order at most nmax (<= SMALL_MAX); `ctas` as in
// batched_launch sets how many CTAs share an SM
int small_launch(const BatchTask* tasks, int count, int nmax, int* dev_counter, double2* D, double* eig, int ctas,
                 int* dev_info, cudaStream_t st);

// one matrix of order 1 to 24 (48 KB of shared memory need no opt-in), on the stream
int small_solve(double2* D, int64_t ld, int n, double* eig, cudaStream_t st);

}  // namespace zq
