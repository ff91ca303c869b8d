// Direct application of the stored reflectors to the eigenvectors (zq_applyq.cu).
#pragma once

#include "zq_kernels.h"

namespace zq {

constexpr int APPLYQ_MAX = 800;

struct ApplyQTask {
  double2* D;         // (null: at off from the call's base) left half: w_j below the diagonal; receives the eigenvectors
  const double* phi;  // 4 n: the phases
  const double* Z;    // n x n eigenvectors of the real tridiagonal
  int64_t ld, ldz;
  int n;
  int col0;           // first grid column of this matrix (batches)
  long long off;
};

// D <- eigenvectors (U -V*; V U*) of one matrix (tasks null), or of a batch
// whose columns [first, first + cols) belong to tasks[task_of[column]]
int apply_q(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int first, int cols, int nmax,
            cudaStream_t st);

// The same for batches with enough columns to fill the GPU (orders up to 256):
// one warp per column, four columns (task, first column) per block; leaves the
// columns in the right halves for apply_q_finish.
constexpr int APPLYQ_WARP_COLUMNS = 4;
int apply_q_warp(const ApplyQTask* tasks, const int2* blocks, int count, double2* base, int nmax, cudaStream_t st);
int apply_q_finish(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int first, int cols, int nmax,
                   cudaStream_t st);

}  // namespace zq
