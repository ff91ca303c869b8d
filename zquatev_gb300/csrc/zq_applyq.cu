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
__global__ void __launch_bounds__(32 * NW) k_apply_q(const ApplyQTask* tasks, const int* task_of, ApplyQTask one) {
  constexpr int RP = 8 * NW;  // rows per pass
  extern __shared__ __align__(16) unsigned char aq_smem[];
  __shared__ double s_red[2][NW][4];
  const int tid = threadIdx.x;
  ApplyQTask t = one;
  int col = blockIdx.x;
  if (tasks) {
    t = tasks[task_of[blockIdx.x]];
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

// (U; V) from the right half into the left half, (-conj V; conj U) in its place
__global__ void k_apply_q_finish(const ApplyQTask* tasks, const int* task_of, ApplyQTask one) {
  ApplyQTask t = one;
  int col = blockIdx.x;
  if (tasks) {
    t = tasks[task_of[blockIdx.x]];
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
int launch(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int cols, cudaStream_t st) {
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
  k_apply_q<NW, NR><<<cols, 32 * NW, smem, st>>>(tasks, task_of, one);
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace

int apply_q(const ApplyQTask* tasks, const int* task_of, const ApplyQTask& one, int cols, int nmax, cudaStream_t st) {
  if (cols <= 0 || nmax <= 0) return ZQ_OK;
  int rc;
  // rows in registers: the smallest count that holds the largest order. One
  // warp per column up to 64 rows (no block barrier), four above
  if (nmax <= 16) rc = launch<1, 2>(tasks, task_of, one, cols, st);
  else if (nmax <= 32) rc = launch<1, 4>(tasks, task_of, one, cols, st);
  else if (nmax <= 64) rc = launch<4, 2>(tasks, task_of, one, cols, st);
  else if (nmax <= 96) rc = launch<4, 3>(tasks, task_of, one, cols, st);
  else if (nmax <= 128) rc = launch<4, 4>(tasks, task_of, one, cols, st);
  else if (nmax <= 192) rc = launch<4, 6>(tasks, task_of, one, cols, st);
  else if (nmax <= 256) rc = launch<4, 8>(tasks, task_of, one, cols, st);
  else if (nmax <= 320) rc = launch<4, 10>(tasks, task_of, one, cols, st);
  else if (nmax <= 384) rc = launch<4, 12>(tasks, task_of, one, cols, st);
  else if (nmax <= 448) rc = launch<4, 14>(tasks, task_of, one, cols, st);
  else if (nmax <= 512) rc = launch<4, 16>(tasks, task_of, one, cols, st);
  else if (nmax <= 640) rc = launch<4, 20>(tasks, task_of, one, cols, st);
  else if (nmax <= APPLYQ_MAX) rc = launch<4, 25>(tasks, task_of, one, cols, st);
  else return ZQ_ERR_ARG;
  if (rc) return rc;
  k_apply_q_finish<<<cols, nmax <= 64 ? 64 : 128, 0, st>>>(tasks, task_of, one);
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace zq
