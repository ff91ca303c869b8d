// FP64-accurate products by residue arithmetic on the bf16 tensor cores (zq_crt.cu).
#pragma once

#include "zq_kernels.h"

namespace zq {

// One operand of a complex product: element (idx, k) of op(A), or (k, idx) of
// op(B), over the K terms of one or two segments (the second scaled by s2).
struct CrtSide {
  const double2* X1; int64_t ld1; int op1; int K1;
  const double2* X2; int64_t ld2; int op2; int K2;
  double s2;
};

// moduli needed for operands of `bits` bits and sums of `terms` products (0: out of range)
int crt_moduli(int bits, double terms);

// sizes of one product's operand residues, output residues (bytes)
struct CrtShape {
  int mp, np, Kp, moduli, prods;  // prods: 3 complex (re, im, re + im), 1 real
  size_t a_bytes, b_bytes, r_bytes;
};
CrtShape crt_shape(int m, int n, int K, int moduli, bool cplx);

// residues of an operand whose rows (A) or columns (B) carry the exponents exps
int crt_split(const CrtSide& s, bool is_a, int count, int count_pad, int Kp, const int* exps, int bits, int moduli,
              void* out, cudaStream_t st);
// C (m x n) from the operands' residues; err is raised when a pipeline wait runs out
int crt_multiply(const CrtShape& sh, const void* a, const void* b, void* r, bool lower, int* err, cudaStream_t st);
int crt_join(const CrtShape& sh, const void* r, int m, int n, int bits, const int* ea, const int* eb, bool lower,
             double2* C, int64_t ldc, cudaStream_t st);

// real C (m x n, ldc) = A (m x k, lda) B (k x n, ldb), column-major doubles, FP64-accurate
size_t crt_dgemm_workspace(int m, int n, int k);
int crt_dgemm(int m, int n, int k, const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
              void* ws, int* err, cudaStream_t st);

}  // namespace zq
