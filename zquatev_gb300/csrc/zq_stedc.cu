// Stage (c): GPU divide-and-conquer eigensolver for a real symmetric
// tridiagonal matrix (all FP64).
//
// Replaces LAPACK zhbev("V","L",n,kd=1) at zquatev.cc:74-84. The reference's
// tridiagonal is complex Hermitian; the quaternion reduction here produces a
// quaternion tridiagonal whose off-diagonal phases are removed exactly by a
// diagonal quaternion similarity (zq_backtransform.cu), leaving this real
// symmetric problem T = Z diag(lambda) Z^T.
//
// Method (Cuppen's divide and conquer with Gu-Eisenstat eigenvectors, written
// from the published algorithm):
//   * scale T to max |entry| = 1;
//   * tear every off-diagonal e_i: T = blockdiag(T1, T2) + e_i u u^T, so the
//     recursion bottoms out at 1x1 leaves (d_i - e_{i-1} - e_i);
//   * merge bottom-up, one batched launch sequence per tree depth:
//       prepare  - z from the children's eigenvectors, merge-sort the poles,
//                  deflate small z and close poles (Givens), sort the deflated;
//       secular  - one thread per root of 1 + rho sum z_k^2/(d_k - x), solved in
//                  coordinates shifted to the nearer pole with a safeguarded
//                  two-pole rational model (bisection fallback);
//       zhat     - recompute z from the roots (Gu-Eisenstat) for orthogonality;
//       vectors  - eigenvectors of the rank-one problem, scattered into the
//                  merge matrix M in final (ascending) order;
//       rotate   - fold the deflation rotations into M's rows;
//       gemm     - Z_node = blockdiag(Z1, Z2) * M  (grouped DGEMM).
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_recip.cuh"
#include "zq_crt.h"
#include "zq_tc32.h"

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

namespace zq {

constexpr double DEPS = 1.1102230246251565e-16;  // 2^-53

__device__ __forceinline__ int dc_find_node(const DcNode* nodes, int cnt, int pos) {
  // nodes sorted by a; returns index of node with a <= pos < b, or -1
  int lo = 0, hi = cnt - 1, r = -1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    if (nodes[mid].a <= pos) { r = mid; lo = mid + 1; } else hi = mid - 1;
  }
  if (r >= 0 && pos < nodes[r].b) return r;
  return -1;
}

template <typename ZT>
__global__ void k_dc_leaf(const DcNode* nodes, int cnt, const double* dmod, ZT* Zout, double* lamout) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const int a = nodes[i].a;
  Zout[nodes[i].zoff + a + (int64_t)a * nodes[i].ld] = (ZT)1;
  lamout[a] = dmod[a];
}

// What the secular equation reads of the kept poles: rho z^2, and float copies for
// its first iterations (pole as a pair hi + lo, rho z^2), in areas whose staged
// contents are no longer needed.
__device__ __forceinline__ float2* dc_pole_pairs(const DcWork& w) { return reinterpret_cast<float2*>(w.sd); }
__device__ __forceinline__ float* dc_pole_weights(const DcWork& w) { return reinterpret_cast<float*>(w.perm); }
__device__ __forceinline__ void dc_publish_poles(const DcWork& w, int a, int K, double rho2) {
  for (int q = threadIdx.x; q < K; q += blockDim.x) {
    const double d = w.nd_val[a + q], z = w.nd_z[a + q], rz = rho2 * z * z;
    const float hi = (float)d;
    w.sz[a + q] = rz;
    dc_pole_pairs(w)[a + q] = make_float2(hi, (float)(d - (double)hi));
    dc_pole_weights(w)[a + q] = (float)rz;
  }
}

// one CTA per internal node. The merged poles (value, z, source column) are
// staged in shared memory when the node fits (m <= scap). Deflation runs in
// parallel unless two kept poles are close enough to need a rotation (see the
// fast path); then the sequential scan runs (each rotation changes the next
// comparison) in one thread, with its operands a shared-memory load away, and
// the deflated list is ranked from shared memory.
constexpr int DC_SCAP = 8192;  // largest node staged in shared memory (20 bytes per pole)
template <typename ZT>
__global__ void __launch_bounds__(256) k_dc_prepare(DcNode* nodes, DcWork w, const ZT* Zin, const double* lamin,
                                                    int scap) {
  pdl_wait();
  extern __shared__ double dc_sm[];
  DcNode& nd = nodes[blockIdx.x];
  const int a = nd.a, c = nd.c, b = nd.b;
  const int m = b - a, n1 = c - a, n2 = b - c;
  const int64_t n = nd.ld;
  Zin += nd.zoff;
  const int tid = threadIdx.x;
  const double rho2 = 2.0 * nd.rho;
  const double rs2 = 0.70710678118654752440;
  const bool staged = m <= scap;
  double* D = staged ? dc_sm : w.sd + a;
  double* Zs = staged ? dc_sm + scap : w.sz + a;
  int* P = staged ? reinterpret_cast<int*>(dc_sm + 2 * scap) : w.perm + a;
  __shared__ double s_red[8];
  __shared__ int s_cnt[3];
  // Values that are not numbers have no place in a sorted order: several may take
  // one position. Every position starts as a valid entry, so that no index below is
  // ever out of range.
  for (int i = tid; i < m; i += blockDim.x) { D[i] = 0.0; Zs[i] = 0.0; P[i] = i; }
  __syncthreads();
  // merge the two sorted eigenvalue lists; z in sorted order
  double dm = 0.0, zm = 0.0;
  for (int i = tid; i < m; i += blockDim.x) {
    double val, z;
    int pos;
    if (i < n1) {
      val = lamin[a + i];
      z = (double)Zin[(c - 1) + (int64_t)(a + i) * n] * rs2;
      // count of right values strictly less than val
      int lo = 0, hi = n2;
      while (lo < hi) { const int mid = (lo + hi) >> 1; if (lamin[c + mid] < val) lo = mid + 1; else hi = mid; }
      pos = i + lo;
    } else {
      const int i2 = i - n1;
      val = lamin[c + i2];
      z = (double)Zin[c + (int64_t)(a + i) * n] * rs2;
      int lo = 0, hi = n1;
      while (lo < hi) { const int mid = (lo + hi) >> 1; if (lamin[a + mid] <= val) lo = mid + 1; else hi = mid; }
      pos = i2 + lo;
    }
    D[pos] = val;
    Zs[pos] = z;
    P[pos] = i;
    dm = fmax(dm, fabs(val));
    zm = fmax(zm, fabs(z));
  }
  const double dmax = block_max(dm, s_red);  // (its barriers also publish D, Zs, P)
  const double zmax = block_max(zm, s_red);
  const double tol = 8.0 * DEPS * fmax(dmax, zmax);
  // Fast path (all threads): z-deflation flags, compaction by a block scan,
  // then the close-pole test on every consecutive pair of the kept poles with
  // their original values. The sequential scan below changes a pole only
  // after a test passes, and every test before the first pass sees original
  // values: so if no pair passes here, the scan would rotate nothing and its
  // lists are exactly these (the deflated ones already in ascending order).
  // Any passing pair sends the node to the sequential scan.
  {
    const int per = (m + (int)blockDim.x - 1) / (int)blockDim.x;  // contiguous entries per thread
    const int i0 = tid * per, i1 = (i0 + per < m) ? i0 + per : m;
    int keep = 0;
    for (int i = i0; i < i1; ++i) keep += !(rho2 * fabs(Zs[i]) <= tol);
    // exclusive scan of the per-thread counts (warp shuffles, then the warps)
    const int lane = tid & 31, wid = tid >> 5;
    int incl = keep;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __shared__ int s_wsum[8], s_flag;
    if (lane == 31) s_wsum[wid] = incl;
    if (tid == 0) s_flag = 0;
    __syncthreads();
    int wbase = 0;
    for (int q = 0; q < wid; ++q) wbase += s_wsum[q];
    int Ktot = 0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) Ktot += s_wsum[q];
    int kpos = wbase + incl - keep;   // kept poles before this thread's chunk
    int dpos = i0 - kpos;             // deflated ones before it
    for (int i = i0; i < i1; ++i) {
      if (!(rho2 * fabs(Zs[i]) <= tol)) {
        w.nd_val[a + kpos] = D[i]; w.nd_z[a + kpos] = Zs[i]; w.nd_col[a + kpos] = P[i]; ++kpos;
      } else {
        w.df_val[a + dpos] = D[i]; w.df_col[a + dpos] = P[i];
        w.df_sval[a + dpos] = D[i]; w.df_scol[a + dpos] = P[i]; ++dpos;
      }
    }
    __syncthreads();
    // pair test on the kept poles (k - 1, k), as the sequential scan forms it
    for (int q = tid + 1; q < Ktot; q += blockDim.x) {
      double sv = w.nd_z[a + q - 1], cc = w.nd_z[a + q];
      const double tau = hypot(cc, sv);
      cc /= tau; sv = -sv / tau;
      const double t = w.nd_val[a + q] - w.nd_val[a + q - 1];
      if (fabs(t * cc * sv) <= tol) s_flag = 1;
    }
    __syncthreads();
    if (!s_flag) {
      __syncthreads();
      dc_publish_poles(w, a, Ktot, rho2);
      if (tid == 0) { nd.K = Ktot; nd.ndefl = m - Ktot; nd.nrot = 0; nd.rho2 = rho2; }
      return;
    }
  }
  if (tid == 0) {
    int K = 0, nd_ = 0, nr = 0;
    int pj = -1;
    for (int j = 0; j < m; ++j) {
      if (rho2 * fabs(Zs[j]) <= tol) {
        w.df_val[a + nd_] = D[j]; w.df_col[a + nd_] = P[j]; ++nd_;
        continue;
      }
      if (pj < 0) { pj = j; continue; }
      double s = Zs[pj], cc = Zs[j];
      const double tau = hypot(cc, s);
      cc /= tau; s = -s / tau;
      const double t = D[j] - D[pj];
      if (fabs(t * cc * s) <= tol) {
        Zs[j] = tau; Zs[pj] = 0.0;
        w.rot_p[a + nr] = P[pj]; w.rot_j[a + nr] = P[j];
        w.rot_c[a + nr] = cc; w.rot_s[a + nr] = s; ++nr;
        const double tt = D[pj] * cc * cc + D[j] * s * s;
        D[j] = D[pj] * s * s + D[j] * cc * cc;
        D[pj] = tt;
        w.df_val[a + nd_] = D[pj]; w.df_col[a + nd_] = P[pj]; ++nd_;
        pj = j;
      } else {
        w.nd_val[a + K] = D[pj]; w.nd_z[a + K] = Zs[pj]; w.nd_col[a + K] = P[pj]; ++K;
        pj = j;
      }
    }
    if (pj >= 0) { w.nd_val[a + K] = D[pj]; w.nd_z[a + K] = Zs[pj]; w.nd_col[a + K] = P[pj]; ++K; }
    nd.K = K; nd.ndefl = nd_; nd.nrot = nr; nd.rho2 = rho2;
    s_cnt[0] = nd_;
    s_cnt[1] = K;
  }
  __syncthreads();
  dc_publish_poles(w, a, s_cnt[1], rho2);
  // sort the deflated list (values, columns) by rank; ties by index
  const int nd_ = s_cnt[0];
  const double* fv = w.df_val + a;
  for (int i = tid; i < nd_; i += blockDim.x) { w.df_sval[a + i] = fv[i]; w.df_scol[a + i] = w.df_col[a + i]; }
  __syncthreads();  // (valid entries whatever the ranks of values that are not numbers)
  if (staged) {  // the staged poles are dead now: their space holds the deflated values
    for (int i = tid; i < nd_; i += blockDim.x) dc_sm[i] = w.df_val[a + i];
    __syncthreads();
    fv = dc_sm;
  }
  for (int i = tid; i < nd_; i += blockDim.x) {
    const double v = fv[i];
    int rank = 0;
    for (int l = 0; l < nd_; ++l) {
      const double u = fv[l];
      rank += (u < v) || (u == v && l < i);
    }
    w.df_sval[a + rank] = v;
    w.df_scol[a + rank] = w.df_col[a + i];
  }
}

// secular equation: one warp per root; the lanes split the sums over the
// poles (butterfly reductions leave identical totals on every lane, so the
// iteration's control flow stays warp-uniform)
//
// FP64 instructions bound it (K^2 poles and roots, ~7 iterations), so each pole
// takes ten: the products rho z^2 are formed once (w.sz), the reciprocals of the
// distances are those of zq_recip.cuh (kept poles of a scaled node lie 1e-15 and
// more apart, their roots 1e-31 and more from them: in its range), and the two sides of the root share one
// accumulation loop each. The root is first approached in FP32 (dc_approach),
// whose instructions cost a sixteenth, so that two or three FP64 iterations remain.
// The step of the two-pole rational model around tau, for root i between the
// poles at distances di, dj (i = K - 1: one pole): f the function's value, dpsi,
// dphi the derivatives of its two sums. False: no step.
template <typename T>
__device__ __forceinline__ bool dc_model_step(bool inner, T di, T dj, T f, T dpsi, T dphi, T& eta) {
  if (inner) {
    const T B1 = di * di * dpsi, B2 = dj * dj * dphi;
    const T qa = f - B1 / di - B2 / dj;
    const T qb = qa * (di + dj) + B1 + B2;
    const T qc = qa * di * dj + B1 * dj + B2 * di;
    // roots of qa x^2 - qb x + qc = 0
    if (qa == T(0)) {
      if (qb == T(0)) return false;
      eta = qc / qb;
      return true;
    }
    const T disc = qb * qb - T(4) * qa * qc;
    if (!(disc >= T(0))) return false;
    const T sq = sqrt(disc);
    const T den = (qb >= T(0)) ? (qb + sq) : (qb - sq);
    const T r1 = den / (T(2) * qa);
    const T r2 = (den != T(0)) ? T(2) * qc / den : r1;
    if (r2 > di && r2 < dj) { eta = r2; return true; }
    if (r1 > di && r1 < dj) { eta = r1; return true; }
    return false;
  }
  const T B1 = di * di * dpsi;
  const T c = f - B1 / di;
  if (!(c > T(0))) return false;
  eta = di + B1 / c;
  return true;
}
// A first value for root i (origin o, tau in (lo, hi)): the same iteration in
// FP32, on pole distances taken from the pairs. A guess only: the FP64 iteration
// starts from it with its own bracket.
__device__ float dc_approach(const float2* D, const float* rz, int K, int i, int o, int lane, int above, float lo,
                             float hi) {
  const float2 Do = D[o];
  auto dist = [&](int k) { const float2 d = D[k]; return (d.x - Do.x) + (d.y - Do.y); };
  float tau = 0.5f * (lo + hi);
  for (int it = 0; it < 24; ++it) {
    float psi = 0.f, phi = 0.f, dpsi = 0.f, dphi = 0.f;
#pragma unroll 4
    for (int k = lane; k <= i; k += 32) {
      const float inv = __frcp_rn(dist(k) - tau), t = rz[k] * inv;
      psi += t;
      dpsi = fmaf(t, inv, dpsi);
    }
#pragma unroll 4
    for (int k = above; k < K; k += 32) {
      const float inv = __frcp_rn(dist(k) - tau), t = rz[k] * inv;
      phi += t;
      dphi = fmaf(t, inv, dphi);
    }
    psi = warp_sum(psi); phi = warp_sum(phi); dpsi = warp_sum(dpsi); dphi = warp_sum(dphi);
    const float f = 1.f + psi + phi;
    if (f < 0.f) lo = tau; else hi = tau;
    if (!(fabsf(f) > 1e-6f * (1.f + fabsf(psi) + fabsf(phi)))) break;  // (also when not a number)
    float eta, tn = 0.5f * (lo + hi);
    if (dc_model_step(i < K - 1, dist(i) - tau, i < K - 1 ? dist(i + 1) - tau : 0.f, f, dpsi, dphi, eta)) {
      const float t = tau + eta;
      if (t > lo && t < hi) tn = t;
    }
    const bool done = fabsf(tn - tau) <= 1e-6f * fabsf(tn);
    tau = tn;
    if (done) break;
  }
  return tau;
}
// Nodes with more poles than this start from the FP32 root (n = 3000: 5.2 ms; from the
// middle of the gap at every order 1.4 ms more). One or two poles start in the middle:
// there the FP64 iteration hits the roots of equal leaves, as of a Toeplitz matrix,
// exactly, and an error made there goes up the whole tree (root mean square of such
// eigenvalues' errors over the norm, n = 40 to 4000: 2.9e-16 with an FP32 start, 2.1e-16
// without; lines at 4, 8 and 64 poles 2.3e-16, 2.3e-16 and 2.2e-16 at up to 5% more time).
constexpr int DC_APPROACH_MIN = 2;
__global__ void __launch_bounds__(128) k_dc_secular(const DcNode* nodes, int cnt, DcWork w) {
  pdl_wait();
  const int pos = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  const int ni = dc_find_node(nodes, cnt, pos);
  if (ni < 0) return;
  const DcNode nd = nodes[ni];
  const int a = nd.a, K = nd.K;
  const int i = pos - a;
  if (i >= K) return;
  const double* D = w.nd_val + a;
  const double* rz = w.sz + a;  // rho z_k^2
  const double rho = nd.rho2;
  // the lane's poles up to the root's own, and the first one above
  const int above = lane + ((i + 32 - lane) & ~31);
  int o;
  double lo, hi;
  if (i < K - 1) {
    const double gap = D[i + 1] - D[i];
    const double mid = 0.5 * gap;
    double fs = 0.0;
    for (int k = lane; k < K; k += 32) fs = fma(rz[k], recip((D[k] - D[i]) - mid), fs);
    const double f = 1.0 + warp_sum(fs);
    if (f >= 0.0) { o = i; lo = 0.0; hi = mid; }
    else { o = i + 1; lo = -mid; hi = 0.0; }
  } else {
    o = K - 1; lo = 0.0; hi = rho;
  }
  const double Do = D[o];
  double tau = 0.5 * (lo + hi);
  if (K > DC_APPROACH_MIN) {
    const double t = (double)dc_approach(dc_pole_pairs(w) + a, dc_pole_weights(w) + a, K, i, o, lane, above, (float)lo, (float)hi);
    if (t > lo && t < hi) tau = t;
  }
  for (int it = 0; it < 200; ++it) {
    double psi = 0.0, phi = 0.0, dpsi = 0.0, dphi = 0.0;
#pragma unroll 4
    for (int k = lane; k <= i; k += 32) {
      const double inv = recip((D[k] - Do) - tau);
      const double t = rz[k] * inv;
      psi += t;
      dpsi = fma(t, inv, dpsi);
    }
#pragma unroll 4
    for (int k = above; k < K; k += 32) {
      const double inv = recip((D[k] - Do) - tau);
      const double t = rz[k] * inv;
      phi += t;
      dphi = fma(t, inv, dphi);
    }
    psi = warp_sum(psi); phi = warp_sum(phi); dpsi = warp_sum(dpsi); dphi = warp_sum(dphi);
    const double f = 1.0 + psi + phi;
    if (f == 0.0) break;
    if (f < 0.0) lo = tau; else hi = tau;
    const double errb = 8.0 * DEPS * (1.0 + fabs(psi) + fabs(phi)) + DEPS * fabs(tau) * (dpsi + dphi);
    // within the rounding error of f: one last step without another evaluation
    // (stopping on the spot left eigenvalues 1.7 times less accurate)
    const bool close = fabs(f) <= errb;
    if (!close && hi - lo <= 2.0 * DEPS * fmax(fabs(lo), fabs(hi))) break;
    // two-pole rational model around the current point
    double eta = 0.0;
    const bool ok = dc_model_step(i < K - 1, (D[i] - Do) - tau, i < K - 1 ? (D[i + 1] - Do) - tau : 0.0, f, dpsi, dphi, eta);
    double tn = ok ? tau + eta : 0.5 * (lo + hi);
    if (close) {
      if (ok && tn > lo && tn < hi) tau = tn;
      break;
    }
    if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
    if (tn == tau) break;
    tau = tn;
  }
  if (lane == 0) {
    w.r_orig[a + i] = o;
    w.r_tau[a + i] = tau;
    w.r_lam[a + i] = Do + tau;
  }
}

// Gu-Eisenstat: zhat_k from the computed roots; one warp per k, the product
// over the roots split over the lanes
__global__ void __launch_bounds__(128) k_dc_zhat(const DcNode* nodes, int cnt, DcWork w) {
  pdl_wait();
  const int pos = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  const int ni = dc_find_node(nodes, cnt, pos);
  if (ni < 0) return;
  const DcNode nd = nodes[ni];
  const int a = nd.a, K = nd.K;
  const int k = pos - a;
  if (k >= K) return;
  const double* D = w.nd_val + a;
  const double Dk = D[k];
  const int* O = w.r_orig + a;
  const double* T = w.r_tau + a;
  // (lambda_{K-1} - D_k) / rho
  double prod = (lane == 0) ? ((D[O[K - 1]] - Dk) + T[K - 1]) / nd.rho2 : 1.0;
#pragma unroll 4
  for (int j = lane; j < K - 1; j += 32) {
    const double num = (D[O[j]] - Dk) + T[j];  // lambda_j - D_k
    const double den = (j < k) ? (D[j] - Dk) : (D[j + 1] - Dk);
    prod *= num / den;  // (a rounding less than with a reciprocal, which the eigenvectors' orthogonality showed)
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) prod *= __shfl_xor_sync(0xffffffffu, prod, off);
  if (lane == 0) {
    const double zk = w.nd_z[a + k];
    const double zh = sqrt(fmax(prod, 0.0));
    w.zhat[a + k] = (zk >= 0.0) ? zh : -zh;
  }
}

// one CTA per column slot of every internal node: writes a full column of M
template <typename ZT>
__global__ void __launch_bounds__(128) k_dc_vectors(const DcNode* nodes, int cnt, DcWork w, ZT* Mb, double* lamout) {
  pdl_wait();
  const int pos = blockIdx.x;
  const int ni = dc_find_node(nodes, cnt, pos);
  if (ni < 0) return;
  const DcNode nd = nodes[ni];
  const int a = nd.a, m = nd.b - nd.a, K = nd.K, ndf = nd.ndefl;
  const int s = pos - a;
  const int tid = threadIdx.x;
  __shared__ double s_red[4];
  int outpos;
  double val;
  if (s < K) {
    val = w.r_lam[a + s];
    int lo = 0, hi = ndf;  // deflated values strictly below
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (w.df_sval[a + mid] < val) lo = mid + 1; else hi = mid; }
    outpos = s + lo;
  } else {
    const int i = s - K;
    val = w.df_sval[a + i];
    int lo = 0, hi = K;  // roots <= val
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (w.r_lam[a + mid] <= val) lo = mid + 1; else hi = mid; }
    outpos = i + lo;
  }
  ZT* col = Mb + nd.zoff + a + (int64_t)(a + outpos) * nd.ld;
  for (int r = tid; r < m; r += blockDim.x) col[r] = (ZT)0;
  __syncthreads();
  if (s < K) {
    const double* D = w.nd_val + a;
    const int o = w.r_orig[a + s];
    const double t = w.r_tau[a + s];
    const double Do = D[o];
    double ss = 0.0;
    for (int k = tid; k < K; k += blockDim.x) {
      const double del = (D[k] - Do) - t;
      const double vk = w.zhat[a + k] * recip(del);
      ss += vk * vk;
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) s_red[tid >> 5] = ss;
    __syncthreads();
    const double nrm = sqrt(s_red[0] + s_red[1] + s_red[2] + s_red[3]);
    const double inv = 1.0 / nrm;
    for (int k = tid; k < K; k += blockDim.x) {
      const double del = (D[k] - Do) - t;
      col[w.nd_col[a + k]] = (ZT)(w.zhat[a + k] * recip(del) * inv);
    }
  } else {
    if (tid == 0) col[w.df_scol[a + (s - K)]] = (ZT)1;
  }
  if (tid == 0) lamout[a + outpos] = val;
}

// apply the deflation rotations (in reverse order) to every column of M
template <typename ZT>
__global__ void k_dc_rotate(const DcNode* nodes, int cnt, DcWork w, ZT* Mb) {
  pdl_wait();
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  const int ni = dc_find_node(nodes, cnt, pos);
  if (ni < 0) return;
  const DcNode nd = nodes[ni];
  if (nd.nrot == 0) return;
  const int a = nd.a;
  ZT* col = Mb + nd.zoff + a + (int64_t)pos * nd.ld;
  for (int r = nd.nrot - 1; r >= 0; --r) {
    const int P = w.rot_p[a + r], J = w.rot_j[a + r];
    const double c = w.rot_c[a + r], s = w.rot_s[a + r];
    const double vp = col[P], vj = col[J];
    col[P] = (ZT)(c * vp - s * vj);
    col[J] = (ZT)(s * vp + c * vj);
  }
}

// Scale and tear, one block per matrix: the largest |entry| becomes 1, the
// off-diagonals leave the diagonal. An entry that is Inf or NaN makes the scale and
// so the whole matrix NaN: deflation compares and sorts, and would pass a part of it
// off as finite.
__global__ void k_dc_scale(const double* d, const double* e, const DcMat* mats, double* dmod, double* es, double* scal) {
  pdl_wait();
  __shared__ double sh[32];
  const DcMat mt = mats[blockIdx.x];
  const int n = mt.n;
  d += mt.p; e += mt.p; dmod += mt.p; es += mt.p;
  unsigned long long mb = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    mb = max(mb, abs_bits(d[i]));
    if (i < n - 1) mb = max(mb, abs_bits(e[i]));
  }
  constexpr unsigned long long INF = 0x7ffull << 52;  // (a NaN would get lost in the maximum)
  const double m = block_max(bits_to_double(min(mb, INF)), sh);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool finite = abs_bits(m) < INF;
  if (threadIdx.x == 0) scal[blockIdx.x] = !finite ? nan : (m > 0.0 ? fmax(m, 2.2250738585072014e-308) : m);
  const double inv = !finite ? nan : ((m > 0.0) ? 1.0 / fmax(m, 2.2250738585072014e-308) : 1.0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double el = (i > 0) ? e[i - 1] * inv : 0.0;
    const double er = (i < n - 1) ? e[i] * inv : 0.0;
    dmod[i] = d[i] * inv - el - er;
    if (i < n - 1) es[i] = er;
  }
}

// eigenvalues times the scale, into place (NaN when the scale is, or a merge product failed)
// `info` (may be null): counts, per matrix, the eigenvalues that are not finite
__global__ void k_dc_unscale(const double* lam, const DcMat* mats, const double* scal, double* eig, int* err,
                             int* info) {
  pdl_wait();
  const DcMat mt = mats[blockIdx.x];  // (x: a batch may have more matrices than the other dimensions take)
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= mt.n) return;
  const double s = scal[blockIdx.x];
  const double v = lam[mt.p + i];
  const bool failed = *err != 0;
  if (failed && i == 0) err[1] = 1;
  const double out = failed || s != s ? __longlong_as_double(0x7ff8000000000000ll) : (s > 0.0 ? v * s : v);
  eig[mt.eoff + i] = out;
  if (info && abs_bits(out) >= (0x7ffull << 52)) atomicAdd(info + blockIdx.x, 1);
}

// Z_node = blockdiag(Z1, Z2) M for small nodes: a thread per entry. The tiled
// products' 64 x 64 blocks would do mostly padding here.
template <typename ZT>
__global__ void __launch_bounds__(256) k_dc_merge(const DcNode* nodes, int cnt, const ZT* Zin, const ZT* Mb, ZT* Zout,
                                                  int mmax) {
  pdl_wait();
  const DcNode nd = nodes[blockIdx.x];
  const int m = nd.b - nd.a;
  const int64_t ld = nd.ld, o = nd.zoff + nd.a + (int64_t)nd.a * ld;
  const int n1 = nd.c - nd.a;
  for (int t = blockIdx.y * blockDim.x + threadIdx.x; t < m * m; t += gridDim.y * blockDim.x) {
    const int r = t % m, c = t / m;
    const int k0 = r < n1 ? 0 : n1, k1 = r < n1 ? n1 : m;
    const ZT* z = Zin + o + r;
    const ZT* mm = Mb + o + (int64_t)c * ld;
    ZT s0 = 0, s1 = 0;
    int k = k0;
#pragma unroll 4
    for (; k + 1 < k1; k += 2) {
      s0 = fma(z[(int64_t)k * ld], mm[k], s0);
      s1 = fma(z[(int64_t)(k + 1) * ld], mm[k + 1], s1);
    }
    if (k < k1) s0 = fma(z[(int64_t)k * ld], mm[k], s0);
    Zout[o + r + (int64_t)c * ld] = s0 + s1;
  }
}

// Couplings of either sign: with S the diagonal of the couplings' running signs, S T S
// has their moduli (the tear needs rho > 0) and the same eigenvalues. One block.
constexpr int DC_SIGN_T = 1024;
__global__ void __launch_bounds__(DC_SIGN_T) k_dc_signs(const double* __restrict__ e, int n, double* __restrict__ e_abs,
                                                        double* __restrict__ signs) {
  pdl_wait();
  __shared__ unsigned s_odd[DC_SIGN_T / 32];  // per warp: which threads' chunks hold an odd number of negative couplings
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + DC_SIGN_T - 1) / DC_SIGN_T, i0 = min(tid * per, n), i1 = min(i0 + per, n);
  bool odd = false;  // chunk: positions i0 .. i1, the coupling e[i - 1] leads to position i
  for (int i = i0; i < i1; ++i) odd ^= i > 0 && e[i - 1] < 0.0;
  const unsigned mask = __ballot_sync(0xffffffffu, odd);
  if (lane == 0) s_odd[warp] = mask;
  __syncthreads();
  int before = __popc(mask & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) before += __popc(s_odd[w]);
  bool neg = before & 1;
  for (int i = i0; i < i1; ++i) {
    neg ^= i > 0 && e[i - 1] < 0.0;
    signs[i] = neg ? -1.0 : 1.0;
    if (i > 0) e_abs[i - 1] = fabs(e[i - 1]);
  }
}
// Z_out = S Z
__global__ void __launch_bounds__(256) k_dc_signed_copy(const double* __restrict__ Z, int n, const double* __restrict__ signs,
                                                        double* __restrict__ Z_out, int64_t ldz) {
  pdl_wait();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const double s = signs[r];
  for (int c = blockIdx.y; c < n; c += gridDim.y) Z_out[r + (int64_t)c * ldz] = s * Z[r + (int64_t)c * n];
}

__global__ void k_dc_setrho(DcNode* nodes, int cnt, const double* es) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cnt && nodes[i].b - nodes[i].a > 1) nodes[i].rho = es[nodes[i].c - 1];
}

// ----------------------------------------------------------------------------
// host side: plan (tree, descriptors) and execution
// ----------------------------------------------------------------------------
// FP64 merges of nodes from this order up run on the tensor cores as residue
// products (zq_crt.cu; FP64-accurate): GB300's FP64 pipe gives 1.25 TFLOP/s, the
// residue product ~25 TFLOP/s of FP64-equivalent work at n = 3000. Below it
// the products are too small for their six launches (a depth of eight
// nodes of 375: 0.34 ms on the FP64 pipe, 0.8 ms as sixteen residue products).
constexpr int DC_CRT_MIN = 600;
// Depths whose nodes all have at most this order: one thread per entry of the
// merged vectors instead of the tiled products (n = 127: a tile's product took
// 40 us on one SM; an entry takes m / 2 multiply-adds).
constexpr int DC_MERGE_MAX = 128;
static size_t dc_crt_doubles(int n) {
  if (n < DC_CRT_MIN) return 0;
  const int h = (n + 1) / 2;
  return crt_dgemm_workspace(h, n, h) / sizeof(double) + 64;
}

size_t DcPlan::workspace_doubles(int n, bool lean) {
  // Z x2, M, lam x2, dmod, es, scal + the per-position DcWork arrays, the matrix table
  const size_t nn = (size_t)n * n;
  return 3 * nn + 2 * (size_t)n + 2 * (size_t)n + 8 + 16 * (size_t)n + 64 + (lean ? 0 : dc_crt_doubles(n));
}

size_t DcPlan::forest_doubles() const {
  return 3 * nn + 20 * (size_t)n + mats_host.size() + 72;
}

int DcPlan::build(int n_) { return build(std::vector<int>{n_}, std::vector<long long>{0}); }

int DcPlan::build(const std::vector<int>& ns, const std::vector<long long>& eoffs) {
  n = 0;
  nn = 0;
  mats_host.clear();
  zoff.clear();
  nodes_host.clear();
  depth_off.clear();
  depth_cnt.clear();
  leaf_off.clear();
  leaf_cnt.clear();
  // recursive halving, breadth first over all trees
  struct Tmp { int a, b, depth, mat; };
  std::vector<Tmp> all;
  std::vector<Tmp> cur;
  for (size_t q = 0; q < ns.size(); ++q) {
    if (ns[q] <= 0) continue;
    cur.push_back({n, n + ns[q], 0, (int)mats_host.size()});
    mats_host.push_back(DcMat{n, ns[q], eoffs[q]});
    zoff.push_back((long long)nn);
    n += ns[q];
    nn += (size_t)ns[q] * ns[q];
  }
  if (n <= 0) return ZQ_OK;
  int depth = 0;
  while (!cur.empty()) {
    std::vector<Tmp> nxt;
    for (auto& t : cur) {
      all.push_back(t);
      if (t.b - t.a > 1) {
        const int c = t.a + (t.b - t.a) / 2;
        nxt.push_back({t.a, c, depth + 1, t.mat});
        nxt.push_back({c, t.b, depth + 1, t.mat});
      }
    }
    cur.swap(nxt);
    ++depth;
  }
  max_depth = depth - 1;
  auto node = [&](const Tmp& x) {
    DcNode nd{};
    const DcMat& m = mats_host[x.mat];
    nd.a = x.a; nd.b = x.b;
    nd.c = x.b - x.a > 1 ? x.a + (x.b - x.a) / 2 : x.a;
    nd.ld = m.n;
    nd.zoff = zoff[x.mat] - m.p - (long long)m.p * m.n;  // positions count from the first matrix
    return nd;
  };
  // group by depth (the order of `all`): internal nodes and leaves separately, each sorted by a
  depth_mmax.clear();
  std::vector<size_t> first(max_depth + 2, all.size());
  for (size_t q = all.size(); q-- > 0;) first[all[q].depth] = q;
  for (int t = 0; t <= max_depth; ++t) {
    depth_off.push_back((int)nodes_host.size());
    int cnt = 0, mmax = 0;
    for (size_t q = first[t]; q < first[t + 1]; ++q)
      if (all[q].b - all[q].a > 1) {
        nodes_host.push_back(node(all[q]));
        ++cnt;
        mmax = std::max(mmax, all[q].b - all[q].a);
      }
    depth_cnt.push_back(cnt);
    depth_mmax.push_back(mmax);
  }
  for (int t = 0; t <= max_depth; ++t) {
    leaf_off.push_back((int)nodes_host.size());
    int cnt = 0;
    for (size_t q = first[t]; q < first[t + 1]; ++q)
      if (all[q].b - all[q].a == 1) {
        nodes_host.push_back(node(all[q]));
        ++cnt;
      }
    leaf_cnt.push_back(cnt);
  }
  // GEMM descriptors per depth (pointers bound at execution time by offsets)
  gemm_host.clear();
  gemm_off.clear();
  gemm_tiles.clear();
  for (int t = 0; t <= max_depth; ++t) {
    gemm_off.push_back((int)gemm_host.size());
    int tiles = 0;
    // depths of small nodes run on k_dc_merge, without descriptors
    for (int q = 0; q < depth_cnt[t] && depth_mmax[t] > DC_MERGE_MAX; ++q) {
      const DcNode& nd = nodes_host[depth_off[t] + q];
      const int m = nd.b - nd.a, n1 = nd.c - nd.a, n2 = nd.b - nd.c;
      const int64_t ld = nd.ld;
      DgemmDesc top{}, bot{};
      top.m = n1; top.n = m; top.k = n1; top.alpha = 1.0; top.beta = 0.0;
      // offsets stored as element indices; converted to pointers in run()
      top.off_a = top.off_b = top.off_c = nd.zoff + nd.a + nd.a * ld;
      bot.m = n2; bot.n = m; bot.k = n2; bot.alpha = 1.0; bot.beta = 0.0;
      bot.off_a = nd.zoff + nd.c + nd.c * ld; bot.off_b = nd.zoff + nd.c + nd.a * ld; bot.off_c = bot.off_b;
      top.lda = top.ldb = top.ldc = ld;
      bot.lda = bot.ldb = bot.ldc = ld;
      top.tile0 = tiles; tiles += ceil_div(top.m, 64) * ceil_div(top.n, 64);
      bot.tile0 = tiles; tiles += ceil_div(bot.m, 64) * ceil_div(bot.n, 64);
      gemm_host.push_back(top);
      gemm_host.push_back(bot);
    }
    gemm_tiles.push_back(tiles);
  }
  return ZQ_OK;
}

// Binds device pointers into the descriptor copies and uploads everything.
int DcPlan::upload(double* ws, DcNode* dnodes, DgemmDesc* ddescs, cudaStream_t st, DcMat* mats, bool lean) {
  base = ws;
  Z[0] = ws; Z[1] = ws + nn; Mb = ws + 2 * nn;
  double* p = ws + 3 * nn;
  lam[0] = p; p += n; lam[1] = p; p += n;
  dmod = p; p += n; es = p; p += n;
  err = reinterpret_cast<int*>(p); p += 8;
  scal = p; p += mats_host.size();
  mats_dev = mats;
  if (!mats) { mats_dev = reinterpret_cast<DcMat*>(p); p += sizeof(DcMat) / sizeof(double) * mats_host.size(); }
  w.sd = p; p += n; w.sz = p; p += n;
  w.nd_val = p; p += n; w.nd_z = p; p += n;
  w.df_val = p; p += n; w.df_sval = p; p += n;
  w.rot_c = p; p += n; w.rot_s = p; p += n;
  w.r_tau = p; p += n; w.r_lam = p; p += n; w.zhat = p; p += n;
  int* ip = reinterpret_cast<int*>(p);
  w.perm = ip; ip += n; w.nd_col = ip; ip += n; w.df_col = ip; ip += n; w.df_scol = ip; ip += n;
  w.rot_p = ip; ip += n; w.rot_j = ip; ip += n; w.r_orig = ip; ip += n;
  // a single matrix: after the position arrays, on a 256-byte boundary of the workspace
  crt_ws = !lean && mats_host.size() == 1 && n >= DC_CRT_MIN ? ws + ((3 * nn + 20 * (size_t)n + 24 + 31) & ~(size_t)31) : nullptr;
  nodes_dev = dnodes;
  descs_dev = ddescs;
  // bind pointers: at depth t, A (children) lives in Z[(t+1)&1], output in Z[t&1]
  std::vector<DgemmDesc> bound = gemm_host;
  for (int t = 0; t <= max_depth; ++t) {
    for (int q = 0; q < gemm_cnt(t); ++q) {
      DgemmDesc& d = bound[gemm_off[t] + q];
      d.A = Z[(t + 1) & 1] + d.off_a;
      d.B = Mb + d.off_b;
      d.C = Z[t & 1] + d.off_c;
    }
  }
  // single-precision views of the same buffers (Z, M as float) for run_single
  Zf[0] = reinterpret_cast<float*>(Z[0]);
  Zf[1] = reinterpret_cast<float*>(Z[1]);
  Mbf = reinterpret_cast<float*>(Mb);
  fdescs_dev = reinterpret_cast<DgemmDescT<float>*>(ddescs + gemm_host.size() + 2);
  std::vector<DgemmDescT<float>> fbound(gemm_host.size());
  for (size_t i = 0; i < gemm_host.size(); ++i) {
    const DgemmDesc& h = gemm_host[i];
    DgemmDescT<float>& f = fbound[i];
    f.lda = h.lda; f.ldb = h.ldb; f.ldc = h.ldc;
    f.off_a = h.off_a; f.off_b = h.off_b; f.off_c = h.off_c;
    f.m = h.m; f.n = h.n; f.k = h.k; f.ta = h.ta; f.tb = h.tb; f.tile0 = h.tile0;
    f.alpha = 1.f; f.beta = 0.f;
  }
  for (int t = 0; t <= max_depth; ++t) {
    for (int q = 0; q < gemm_cnt(t); ++q) {
      DgemmDescT<float>& d = fbound[gemm_off[t] + q];
      d.A = Zf[(t + 1) & 1] + d.off_a;
      d.B = Mbf + d.off_b;
      d.C = Zf[t & 1] + d.off_c;
    }
  }
  if (!mats_host.empty())
    ZQ_CUDA(cudaMemcpyAsync(mats_dev, mats_host.data(), sizeof(DcMat) * mats_host.size(), cudaMemcpyHostToDevice, st));
  if (!nodes_host.empty())
    ZQ_CUDA(cudaMemcpyAsync(dnodes, nodes_host.data(), sizeof(DcNode) * nodes_host.size(), cudaMemcpyHostToDevice, st));
  if (!bound.empty())
    ZQ_CUDA(cudaMemcpyAsync(ddescs, bound.data(), sizeof(DgemmDesc) * bound.size(), cudaMemcpyHostToDevice, st));
  if (!fbound.empty())
    ZQ_CUDA(cudaMemcpyAsync(fdescs_dev, fbound.data(), sizeof(DgemmDescT<float>) * fbound.size(), cudaMemcpyHostToDevice,
                            st));
  // the host copies must outlive the async copies: synchronise once at plan time
  ZQ_CUDA(cudaStreamSynchronize(st));
  return ZQ_OK;
}

template <typename ZT>
static int dc_run(DcPlan& P, const double* d, const double* e, double* lam_out, ZT* const Zb[2], ZT* Mb,
                  const DgemmDescT<ZT>* descs, cudaStream_t st, int* info = nullptr, int* flags = nullptr) {
  const int n = P.n, nmat = (int)P.mats_host.size();
  int nmax = 0;
  for (const DcMat& m : P.mats_host) nmax = std::max(nmax, m.n);
  int* const err = flags ? flags : P.err;
  if (!flags) ZQ_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
  ZQ_CUDA(launch_pdl_smem(k_dc_scale, dim3(nmat), dim3(nmax <= 256 ? 64 : 256), 0, st, d, e, P.mats_dev, P.dmod, P.es, P.scal));
  ZQ_LAUNCH_CHECK();
  if (!P.nodes_host.empty()) {
    ZQ_CUDA(launch_pdl_smem(k_dc_setrho, dim3(ceil_div((int)P.nodes_host.size(), 256)), dim3(256), 0, st, P.nodes_dev, (int)P.nodes_host.size(), P.es));
    ZQ_LAUNCH_CHECK();
  }
  // Z buffers need zeros outside the diagonal blocks only where they are read:
  // every read is inside a node's block, which is fully written first.
  for (int t = P.max_depth; t >= 0; --t) {
    ZT* Zo = Zb[t & 1];
    ZT* Zi = Zb[(t + 1) & 1];
    double* lo = P.lam[t & 1];
    const double* li = P.lam[(t + 1) & 1];
    if (P.leaf_cnt[t] > 0) {
      ZQ_CUDA(launch_pdl_smem(k_dc_leaf<ZT>, dim3(ceil_div(P.leaf_cnt[t], 128)), dim3(128), 0, st, P.nodes_dev + P.leaf_off[t], P.leaf_cnt[t], P.dmod, Zo,
                                                                    lo));
      ZQ_LAUNCH_CHECK();
    }
    const int cnt = P.depth_cnt[t];
    if (cnt == 0) continue;
    DcNode* nd = P.nodes_dev + P.depth_off[t];
    {
      // shared-memory staging of the merged poles for the depth's largest node
      const int scap = P.depth_mmax[t] <= DC_SCAP ? P.depth_mmax[t] : 0;
      const size_t smem = (size_t)scap * 20;
      if (smem > 48 * 1024) {
        static std::atomic<unsigned long long> attr_set{0};
        int dev = 0;
        ZQ_CUDA(cudaGetDevice(&dev));
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(attr_set.load() & bit)) {
          ZQ_CUDA(cudaFuncSetAttribute(k_dc_prepare<ZT>, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SCAP * 20));
          attr_set.fetch_or(bit);
        }
      }
      ZQ_CUDA(launch_pdl_smem(k_dc_prepare<ZT>, dim3(cnt), dim3(256), smem, st, nd, P.w, Zi, li, scap));
      ZQ_LAUNCH_CHECK();
    }
    ZQ_CUDA(launch_pdl_smem(k_dc_secular, dim3(ceil_div(n, 4)), dim3(128), 0, st, nd, cnt, P.w));
    ZQ_LAUNCH_CHECK();
    ZQ_CUDA(launch_pdl_smem(k_dc_zhat, dim3(ceil_div(n, 4)), dim3(128), 0, st, nd, cnt, P.w));
    ZQ_LAUNCH_CHECK();
    ZQ_CUDA(launch_pdl_smem(k_dc_vectors<ZT>, dim3(n), dim3(128), 0, st, nd, cnt, P.w, Mb, lo));
    ZQ_LAUNCH_CHECK();
    ZQ_CUDA(launch_pdl_smem(k_dc_rotate<ZT>, dim3(ceil_div(n, 128)), dim3(128), 0, st, nd, cnt, P.w, Mb));
    ZQ_LAUNCH_CHECK();
    if (P.depth_mmax[t] <= DC_MERGE_MAX) {
      const int mm = P.depth_mmax[t];
      const dim3 grid((unsigned)cnt, (unsigned)std::min(64, ceil_div(mm * mm, 256)));
      ZQ_CUDA(launch_pdl_smem(k_dc_merge<ZT>, grid, dim3(mm <= 8 ? 64 : 256), 0, st, nd, cnt, Zi, Mb, Zo, mm));
      ZQ_LAUNCH_CHECK();
    } else if (P.gemm_tiles[t] > 0) {
      bool done = false;
      if constexpr (std::is_same<ZT, float>::value) {
        // FP32 merges of large nodes on the tensor cores (TF32 x3), one product per child
        if (P.tc_err && P.depth_mmax[t] >= 512 && fp32_products_on_tensor_cores(TC_USE_DC)) {
          for (int q = 0; q < P.gemm_cnt(t); ++q) {
            const DgemmDesc& h = P.gemm_host[P.gemm_off[t] + q];
            Tc32Args g{};
            g.cplx = 0; g.m = h.m; g.n = h.n; g.nseg = 1;
            g.seg[0].a.p = Zi + h.off_a; g.seg[0].a.ld = h.lda; g.seg[0].a.kfast = 0; g.seg[0].a.sign = 1.f;
            g.seg[0].b.p = Mb + h.off_b; g.seg[0].b.ld = h.ldb; g.seg[0].b.kfast = 1; g.seg[0].b.sign = 1.f;
            g.seg[0].k = h.k;
            g.alpha = make_float2(1.f, 0.f); g.beta = make_float2(0.f, 0.f);
            g.C = Zo + h.off_c; g.ldc = h.ldc;
            g.splits = 1;
            g.err = P.tc_err;
            if (int rc = tc32_gemm(g, st)) return rc;
          }
          done = true;
        }
      }
      if constexpr (std::is_same<ZT, double>::value) {
        if (P.crt_ws && P.depth_mmax[t] >= DC_CRT_MIN) {
          for (int q = 0; q < P.gemm_cnt(t); ++q) {
            const DgemmDesc& h = P.gemm_host[P.gemm_off[t] + q];
            if (int rc = crt_dgemm(h.m, h.n, h.k, Zi + h.off_a, h.lda, Mb + h.off_b, h.ldb, Zo + h.off_c, h.ldc, P.crt_ws,
                                   err, st))
              return rc;
          }
          done = true;
        }
      }
      if (!done) {
        grouped_launch<ZT>(descs + P.gemm_off[t], P.gemm_cnt(t), P.gemm_tiles[t], st);
        ZQ_LAUNCH_CHECK();
      }
    }
  }
  ZQ_CUDA(launch_pdl_smem(k_dc_unscale, dim3((unsigned)nmat, (unsigned)ceil_div(nmax, 128)), dim3(128), 0, st, P.lam[0], P.mats_dev,
                          P.scal, lam_out, err, info));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int DcPlan::run_forest(const double* d, const double* e, double* eig, int* info, cudaStream_t st) {
  if (n <= 0) return ZQ_OK;
  return dc_run<double>(*this, d, e, eig, Z, Mb, descs_dev, st, info);
}

int DcPlan::run(const double* d, const double* e, double* lam_out, double*& z_out, cudaStream_t st, int* flags) {
  if (n <= 0) return ZQ_OK;
  if (int rc = dc_run<double>(*this, d, e, lam_out, Z, Mb, descs_dev, st, nullptr, flags)) return rc;
  z_out = Z[0];
  return ZQ_OK;
}

int DcPlan::run_signed(const double* d, const double* e, double* lam_out, double* Z_out, int64_t ldz, double* e_abs,
                       double* signs, cudaStream_t st) {
  if (n <= 0) return ZQ_OK;
  ZQ_CUDA(launch_pdl_smem(k_dc_signs, dim3(1), dim3(DC_SIGN_T), 0, st, e, n, e_abs, signs));
  ZQ_LAUNCH_CHECK();
  double* Zi = nullptr;
  if (int rc = run(d, e_abs, lam_out, Zi, st)) return rc;
  ZQ_CUDA(launch_pdl_smem(k_dc_signed_copy, dim3((unsigned)ceil_div(n, 256), (unsigned)std::min(n, 8192)), dim3(256), 0, st, Zi, n, signs,
                          Z_out, ldz));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int DcPlan::run_single(const double* d, const double* e, double* lam_out, float*& z_out, cudaStream_t st) {
  if (n <= 0) return ZQ_OK;
  if (int rc = dc_run<float>(*this, d, e, lam_out, Zf, Mbf, fdescs_dev, st)) return rc;
  z_out = Zf[0];
  return ZQ_OK;
}

}  // namespace zq
