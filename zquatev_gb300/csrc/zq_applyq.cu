// Back-transformation of the FP64 path for orders up to APPLYQ_MAX: every
// eigenvector column x = Phi z takes the stored reflectors directly,
//   x <- (I - W_j W_j^H) x for j = n-3 .. 0,
// instead of forming Q Phi and multiplying (zq_backtransform.cu; reference
// zquatev.cc:86-90 and blocked.cc:477-544).
//
// Why: the columns are independent, so no two CTAs ever wait for each other and
// the FP64 work (32 n^3 flops) spreads over all SMs at any order, where the
// blocked form ran chains of small products (n = 384: 24 ms, n = 127: 6.9 ms;
// both now bound by the FP64 pipe and one reduction per reflector).
//
// One CTA of NW warps per column. Thread (row lane rl, component k) holds
// component k of rows rl + 8 NW i in registers. Per row and reflector the
// thread multiplies its component with the four components of w (from shared
// memory): 4 FMAs for the quaternion dot product c = (w^H x, [w, x]), 4 for the
// update, and the lanes' products meet once per reflector. The next reflectors
// are prefetched through registers into a three-buffer ring, which leaves one
// block barrier per reflector.
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_applyq.h"

#include <atomic>

namespace zq {
namespace {

struct alignas(16) W4 { double v[4]; };

// signs of C_k = sum_q s w[q] x[k^q] and of U_k = sum_q s w[q] C[k^q], bit q set: minus
//   C_1: + - + -   C_2: + - - +   C_3: + + - -
//   U_0: + - - -   U_1: + + - +   U_2: + + + -   U_3: + - + +
__device__ __forceinline__ unsigned c_signs(int k) { return (0xC6A0u >> (4 * k)) & 15u; }
__device__ __forceinline__ unsigned u_signs(int k) { return (0x284Eu >> (4 * k)) & 15u; }
__device__ __forceinline__ double signed_by(double v, unsigned neg) {
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)neg << 63));
}

// One thread's state of a column.
template <int NW, int NR>
struct ColState {
  double x[NR], wn[NR];     // component of the column; of the prefetched reflector
  const double* A;          // this component of w: A[2 (r + j ld)]
  double* ring;             // three reflectors of 8 NW NR rows, four components each
  int n, ld, rl, k, buf;
  unsigned cs, us;
};
template <int NW, int NR, int FROM>
__device__ __forceinline__ void aq_fetch(ColState<NW, NR>& s, int j) {
  const double* a = s.A + 2 * (int64_t)(j >= 0 ? j : 0) * s.ld;
#pragma unroll
  for (int i = FROM; i < NR; ++i) {
    const int r = s.rl + 8 * NW * i;
    s.wn[i] = (j >= 0 && r > j && r < s.n) ? __ldg(a + 2 * r) : 0.0;
  }
}
template <int NW, int NR, int FROM>
__device__ __forceinline__ void aq_stage(ColState<NW, NR>& s, int buf) {
  double* w = s.ring + (size_t)buf * (32 * NW * NR) + 4 * s.rl + s.k;
#pragma unroll
  for (int i = FROM; i < NR; ++i) w[32 * NW * i] = s.wn[i];
}
// Reflectors j whose first row lies in pass I0, then those of pass I0 - 1, ...:
// the passes a reflector does not reach are left out at compile time (a
// predicated-off FP64 instruction still holds the pipe: with run-time tests
// around each pass the kernel issued 2.2 times the FP64 work it needed).
template <int NW, int NR, int I0>
__device__ __forceinline__ void aq_segment(ColState<NW, NR>& s, int j, double (*red)[NW][4]) {
  constexpr int RP = 8 * NW, LOW = I0 > 0 ? I0 - 1 : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (; j >= 0 && j >= RP * I0 - 1; --j) {
    const W4* w = reinterpret_cast<const W4*>(s.ring + (size_t)s.buf * (32 * NW * NR)) + s.rl;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = I0; i < NR; ++i) {
      const W4 wv = w[RP * i];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(wv.v[q], s.x[i], acc[q]);
    }
    // component k of c: the products w[q] x[k ^ q] lie with the lane of component k ^ q
    double c = signed_by(acc[0], s.cs & 1u);
#pragma unroll
    for (int q = 1; q < 4; ++q) c += signed_by(__shfl_xor_sync(0xffffffffu, acc[q], q), (s.cs >> q) & 1u);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    const int nb = s.buf == 2 ? 0 : s.buf + 1;
    aq_stage<NW, NR, LOW>(s, nb);
    if (NW > 1) {
      if (lane < 4) red[j & 1][warp][lane] = c;
      __syncthreads();
      c = red[j & 1][0][s.k];
#pragma unroll
      for (int u = 1; u < NW; ++u) c += red[j & 1][u][s.k];
    } else {
      __syncwarp();
    }
    aq_fetch<NW, NR, LOW>(s, j - 2);
    double u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = signed_by(__shfl_xor_sync(0xffffffffu, c, q), ((s.us >> q) & 1u) ^ 1u);
#pragma unroll
    for (int i = I0; i < NR; ++i) {
      const W4 wv = w[RP * i];
#pragma unroll
      for (int q = 0; q < 4; ++q) s.x[i] = fma(wv.v[q], u[q], s.x[i]);
    }
    s.buf = nb;
  }
  if constexpr (I0 > 0) aq_segment<NW, NR, I0 - 1>(s, j, red);
}

template <int NW, int NR>
__global__ void __launch_bounds__(32 * NW) k_apply_q(const ApplyQTask* tasks, const int* task_of, ApplyQTask one, int first) {
  pdl_wait();
  constexpr int RP = 8 * NW;  // rows per pass
  extern __shared__ __align__(16) unsigned char aq_smem[];
  __shared__ double s_red[2][NW][4];
  const int tid = threadIdx.x;
  ApplyQTask t = one;
  int col = first + blockIdx.x;
  if (tasks) {
    t = tasks[task_of[col]];
    if (!t.D) t.D = one.D + t.off;
    col -= t.col0;
  }
  const int n = t.n;
  ColState<NW, NR> s;
  s.n = n; s.ld = (int)t.ld; s.k = tid & 3; s.rl = tid >> 2; s.buf = 0;
  s.cs = c_signs(s.k); s.us = u_signs(s.k);
  s.ring = reinterpret_cast<double*>(aq_smem);
  s.A = reinterpret_cast<const double*>(t.D + (s.k < 2 ? 0 : n)) + (s.k & 1);
  // x = Phi z
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int r = s.rl + RP * i;
    s.x[i] = r < n ? t.phi[4 * r + s.k] * t.Z[r + (int64_t)col * t.ldz] : 0.0;
  }
  aq_fetch<NW, NR, 0>(s, n - 3);
  aq_stage<NW, NR, 0>(s, 0);
  aq_fetch<NW, NR, 0>(s, n - 4);
  if (NW > 1) __syncthreads(); else __syncwarp();
  aq_segment<NW, NR, NR - 1>(s, n - 3, s_red);
  // the column, in the right half of D (the reflectors are still being read)
  double* X = reinterpret_cast<double*>(t.D + (s.k < 2 ? 0 : n) + (int64_t)(n + col) * t.ld) + (s.k & 1);
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int r = s.rl + RP * i;
    if (r < n) X[2 * r] = s.x[i];
  }
}

// ------------------------------------------------------- one warp per column
// With enough columns to fill the GPU a warp takes a whole column, eight rows a
// pass: the products meet inside the warp (6 FP64 instructions per reflector
// instead of 9, against 8 per pass), four columns share each reflector in
// shared memory. NP passes; segments of U passes.
template <int NP>
struct WarpState {
  double x[NP];
  const double* wsrc;  // this thread's component of w: wsrc[2 (r + j ld)]
  double* ring;
  int n, rl, k, buf;
  int64_t ld;
  unsigned cs, us;
};
constexpr int AW = 4;  // warps (columns) per CTA
template <int NP>
__device__ __forceinline__ void aw_fetch(const WarpState<NP>& s, int j, double (&wn)[(NP + AW - 1) / AW]) {
  const int r0 = threadIdx.x >> 2;
  const double* a = s.wsrc + 2 * (int64_t)(j >= 0 ? j : 0) * s.ld;
#pragma unroll
  for (int i = 0; i < (NP + AW - 1) / AW; ++i) {
    const int r = r0 + 8 * AW * i;
    wn[i] = (j >= 0 && r > j && r < s.n) ? __ldg(a + 2 * r) : 0.0;
  }
}
template <int NP>
__device__ __forceinline__ void aw_stage(const WarpState<NP>& s, int buf, const double (&wn)[(NP + AW - 1) / AW]) {
  double* w = s.ring + (size_t)buf * (32 * NP) + threadIdx.x;
#pragma unroll
  for (int i = 0; i < (NP + AW - 1) / AW; ++i)
    if ((threadIdx.x >> 2) + 8 * AW * i < 8 * NP) w[32 * AW * i] = wn[i];
}
template <int NP, int U, int S>
__device__ __forceinline__ void aw_segment(WarpState<NP>& s, int j, double (&wn)[(NP + AW - 1) / AW]) {
  constexpr int I0 = S * U;  // first pass of this segment's reflectors
  for (; j >= 0 && j >= 8 * I0 - 1; --j) {
    const W4* w = reinterpret_cast<const W4*>(s.ring + (size_t)s.buf * (32 * NP)) + s.rl;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = I0; i < NP; ++i) {
      const W4 wv = w[8 * i];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(wv.v[q], s.x[i], acc[q]);
    }
    double c = signed_by(acc[0], s.cs & 1u);
#pragma unroll
    for (int q = 1; q < 4; ++q) c += signed_by(__shfl_xor_sync(0xffffffffu, acc[q], q), (s.cs >> q) & 1u);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    const int nb = s.buf == 2 ? 0 : s.buf + 1;
    aw_stage<NP>(s, nb, wn);
    aw_fetch<NP>(s, j - 2, wn);
    double u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = signed_by(__shfl_xor_sync(0xffffffffu, c, q), ((s.us >> q) & 1u) ^ 1u);
#pragma unroll
    for (int i = I0; i < NP; ++i) {
      const W4 wv = w[8 * i];
#pragma unroll
      for (int q = 0; q < 4; ++q) s.x[i] = fma(wv.v[q], u[q], s.x[i]);
    }
    __syncthreads();  // the next reflector is staged; buffer nb + 1 is free in every warp
    s.buf = nb;
  }
  if constexpr (S > 0) aw_segment<NP, U, S - 1>(s, j, wn);
}

// CTA: four consecutive columns of one matrix (the last CTA of a matrix may
// have idle warps, which still take part in the staging)
template <int NP, int U>
__global__ void __launch_bounds__(32 * AW) k_apply_q_warp(const ApplyQTask* tasks, const int2* blocks, double2* base) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char aq_smem[];
  const int2 bl = blocks[blockIdx.x];  // (task, first column)
  ApplyQTask t = tasks[bl.x];
  if (!t.D) t.D = base + t.off;
  const int n = t.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = bl.y + warp;
  const bool live = col < n;
  WarpState<NP> s;
  s.n = n; s.ld = t.ld; s.k = lane & 3; s.rl = lane >> 2; s.buf = 0;
  s.cs = c_signs(s.k); s.us = u_signs(s.k);
  s.ring = reinterpret_cast<double*>(aq_smem);
  s.wsrc = reinterpret_cast<const double*>(t.D + (s.k < 2 ? 0 : n)) + (s.k & 1);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int r = s.rl + 8 * i;
    s.x[i] = live && r < n ? t.phi[4 * r + s.k] * t.Z[r + (int64_t)col * t.ldz] : 0.0;
  }
  double wn[(NP + AW - 1) / AW];
  aw_fetch<NP>(s, n - 3, wn);
  aw_stage<NP>(s, 0, wn);
  aw_fetch<NP>(s, n - 4, wn);
  __syncthreads();
  aw_segment<NP, U, (NP - 1) / U>(s, n - 3, wn);
  if (!live) return;
  double* X = reinterpret_cast<double*>(t.D + (s.k < 2 ? 0 : n) + (int64_t)(n + col) * t.ld) + (s.k & 1);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const int r = s.rl + 8 * i;
    if (r < n) X[2 * r] = s.x[i];
  }
}

template <int NP, int U>
int launch_warp(const ApplyQTask* tasks, const int2* blocks, double2* base, int count, cudaStream_t st) {
  constexpr int smem = 3 * (int)sizeof(W4) * 8 * NP;
  static_assert(smem <= 47 * 1024, "shared memory");
  ZQ_CUDA(launch_pdl_smem(k_apply_q_warp<NP, U>, dim3(count), dim3(32 * AW), smem, st, tasks, blocks, base));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

// (U; V) from the right half into the left half, (-conj V; conj U) in its place
__global__ void k_apply_q_finish(const ApplyQTask* tasks, const int* task_of, ApplyQTask one, int first) {
  pdl_wait();
  ApplyQTask t = one;
  int col = first + blockIdx.x;
  if (tasks) {
    t = tasks[task_of[col]];
    if (!t.D) t.D = one.D + t.off;
    col -= t.col0;
  }
  double2* L = t.D + (int64_t)col * t.ld;
  double2* X = t.D + (int64_t)(t.n + col) * t.ld;
  for (int r = threadIdx.x; r < t.n; r += blockDim.x) {
    const double2 u = X[r], v = X[t.n + r];
    L[r] = u;
    L[t.n + r] = v;
    X[r] = make_double2(-v.x, v.y);
    X[t.n + r] = make_double2(u.x, -u.y);
  }
}

template <int NW, int NR>
int launch(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int first, int cols,
           cudaStream_t st) {
  constexpr int smem = 3 * (int)sizeof(W4) * 8 * NW * NR;
  if (smem > 47 * 1024) {
    static std::atomic<unsigned long long> set{0};
    int dev = 0;
    ZQ_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(set.load() & bit)) {
      ZQ_CUDA(cudaFuncSetAttribute(k_apply_q<NW, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      set.fetch_or(bit);
    }
  }
  ZQ_CUDA(launch_pdl_smem(k_apply_q<NW, NR>, dim3(cols), dim3(32 * NW), smem, st, tasks, task_of, one, first));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace

int apply_q(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int first, int cols, int nmax,
            cudaStream_t st) {
  if (cols <= 0 || nmax <= 0) return ZQ_OK;
  int rc;
  // rows in registers: the smallest count that holds the largest order. One
  // warp per column up to 32 rows (no block barrier), four above
  if (nmax <= 16) rc = launch<1, 2>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 32) rc = launch<1, 4>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 64) rc = launch<4, 2>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 96) rc = launch<4, 3>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 128) rc = launch<4, 4>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 192) rc = launch<4, 6>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 256) rc = launch<4, 8>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 320) rc = launch<4, 10>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 384) rc = launch<4, 12>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 448) rc = launch<4, 14>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 512) rc = launch<4, 16>(tasks, task_of, one, first, cols, st);
  else if (nmax <= 640) rc = launch<4, 20>(tasks, task_of, one, first, cols, st);
  else if (nmax <= APPLYQ_MAX) rc = launch<4, 25>(tasks, task_of, one, first, cols, st);
  else return ZQ_ERR_ARG;
  if (rc) return rc;
  return apply_q_finish(tasks, task_of, one, first, cols, nmax, st);
}

int apply_q_warp(const ApplyQTask* tasks, const int2* blocks, int count, double2* base, int nmax, cudaStream_t st) {
  if (count <= 0) return ZQ_OK;
  if (nmax <= 64) return launch_warp<8, 1>(tasks, blocks, base, count, st);
  if (nmax <= 96) return launch_warp<12, 1>(tasks, blocks, base, count, st);
  if (nmax <= 128) return launch_warp<16, 1>(tasks, blocks, base, count, st);
  if (nmax <= 160) return launch_warp<20, 2>(tasks, blocks, base, count, st);
  if (nmax <= 192) return launch_warp<24, 2>(tasks, blocks, base, count, st);
  if (nmax <= 224) return launch_warp<28, 2>(tasks, blocks, base, count, st);
  if (nmax <= 256) return launch_warp<32, 2>(tasks, blocks, base, count, st);
  return ZQ_ERR_ARG;
}

int apply_q_finish(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int first, int cols, int nmax,
                   cudaStream_t st) {
  ZQ_CUDA(launch_pdl_smem(k_apply_q_finish, dim3(cols), dim3(nmax <= 64 ? 64 : 128), 0, st, tasks, task_of, one, first));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace zq
