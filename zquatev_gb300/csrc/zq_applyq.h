// Direct application of the stored reflectors to the eigenvectors (zq_applyq.cu).
#pragma once

#include "zq_kernels.h"

namespace zq {

constexpr int APPLYQ_MAX = 800;

struct ApplyQTask {
  double2* D;         // left half: w_j below the diagonal; receives the eigenvectors
  const double* phi;  // 4 n: the phases
  const double* Z;    // n x n eigenvectors of the real tridiagonal
  int64_t ld, ldz;
  int n;
  int col0;           // first grid column of this matrix (batches)
};

// D <- eigenvectors (U -V*; V U*) of one matrix (tasks null), or of a batch
// whose column i of `cols` belongs to tasks[task_of[i]]
int apply_q(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int cols, int nmax, cudaStream_t st);

}  // namespace zq
