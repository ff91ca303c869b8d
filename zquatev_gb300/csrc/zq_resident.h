// Tridiagonalisation with the matrix resident in shared memory (zq_resident.cu).
#pragma once

#include "zq_kernels.h"
#include "zq_quat.cuh"

namespace zq {

constexpr int RESIDENT_MMAX = 2048;  // bound of the search for the largest order that fits

// one matrix: columns k0.. of an order-n reduction whose trailing block is up to date
template <typename R>
struct TriTask {
  cplx<R>* M;  // [A; B], 2n x n, column-major (in a queue: null, at off from the queue's base, or a pointer)
  int n, k0;
  int64_t ld;
  double *d, *e, *tau;
  long long off;
};

// exchange area of one group of CTAs (device memory)
template <typename R>
struct TriGroup {
  unsigned* counter;  // barrier arrivals
  unsigned* abort;    // a wait ran out
  int* slot;          // the task taken from the queue (two, in turn)
  double *cpart, *npart;  // per CTA: partials of c and of |x|^2
  double* q2;             // |x_1|^2 of the column
  Q4<R>*x, *y, *col, *part;
};

inline __host__ __device__ size_t tri_group_bytes(int G, int m, int T, size_t real_bytes) {
  const size_t nt = (size_t)((m + T - 1) / T);
  return 256 + sizeof(double) * 2 * (size_t)G + 4 * real_bytes * (3 * (size_t)m + nt * (size_t)m) + 256;
}

template <typename R>
__device__ __forceinline__ TriGroup<R> tri_group(unsigned char* base, int G, int m, int T) {
  TriGroup<R> g;
  g.counter = reinterpret_cast<unsigned*>(base);
  g.abort = g.counter + 1;
  g.slot = reinterpret_cast<int*>(g.counter + 2);
  g.cpart = reinterpret_cast<double*>(base + 256);
  g.npart = g.cpart + G;
  g.q2 = reinterpret_cast<double*>(base + 128);
  g.x = reinterpret_cast<Q4<R>*>(base + ((256 + sizeof(double) * 2 * (size_t)G + 31) & ~(size_t)31));
  g.y = g.x + m;
  g.col = g.y + m;
  g.part = g.col + m;
  return g;
}

template <typename R>
struct TriArgs {
  TriTask<R> one;              // tasks == null: this matrix
  const TriTask<R>* tasks;     // or a queue of them, matrices at base + off
  cplx<R>* base;
  int ntasks;
  int* queue;                  // zeroed before the launch
  int G, m_max;                // CTAs per group; largest trailing order
  unsigned char* ws;           // per group, ws_stride bytes apart; the first 64 bytes of each zeroed
  size_t ws_stride;
  int* err;                    // raised when a wait ran out (may be null: NaN in d only)
  long long limit;
};

// A queue of FP64 matrices (device arrays; orders at most m_max), each reduced by
// a cluster of G CTAs; ws as tri_queue_bytes(G, m_max), queue one int.
int tri_queue(const TriTask<double>* tasks, int ntasks, double2* base, int m_max, int G, void* ws, int* queue,
              cudaStream_t st);
size_t tri_queue_bytes(int G, int m_max, int ntasks);
// cluster size that finishes a queue of these orders (largest first) soonest, and
// the estimated time in clock cycles; 0: no cluster holds the largest
int tri_queue_cluster(const int* orders, int count, double* cycles);

// CTAs of a cooperative launch with one CTA per SM (0: not available)
int sm_count();
// CTAs for the reduction of an order-n matrix (alone: no other solve runs beside it)
int resident_ctas(int n, bool alone);
// whether an order-m block fits the shared memory of `ctas` CTAs, and the largest that does
template <typename R> bool resident_fits(int m, int ctas);
template <typename R> int resident_max(int ctas);
// columns k0..n-1 of v's reduction
template <typename R> int tri_resident(const TridiagView<R>& v, int k0, int ctas, cudaStream_t st);
size_t resident_workspace_bytes(int n, size_t real_bytes);

}  // namespace zq
