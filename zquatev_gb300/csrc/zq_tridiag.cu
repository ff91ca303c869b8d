// Stage (a)+(b): blocked, structure-preserving tridiagonalisation of a
// quaternion-Hermitian matrix on the GPU.
//
// Reference: ts::impl::panel_update (blocked.cc:45-546) and
// ts::impl::unblocked_update (unblocked.cc:44-131), driven by the panel loop at
// zquatev.cc:68-72. The reference zeroes each column with a Householder on the
// B part (blocked.cc:167-178), a symplectic Givens (blocked.cc:234-337) and a
// Householder on the A part (blocked.cc:339-413), keeping a Kressner compact-WY
// form with 3x3-block T, R, S matrices.
//
// Here each column k is zeroed by ONE quaternion Householder reflector
//   P_k = I - W_k W_k^H,   W_k = [w, J conj(w)]  (2L x 2, W^H W = 2 I),
// with w = (wa, wb) built from the quaternion column x = (A[k+1:,k], B[k+1:,k]):
//   w = f * (x + s * x_1 e_1),  s = |x| / |x_1|,  f = 1 / sqrt(|x| (|x| + |x_1|)),
// which maps x to the quaternion -s * x_1 e_1 (the subdiagonal entry e_k; its
// quaternion phase is removed later by a diagonal quaternion similarity, see
// zq_backtransform.cu). This is the same family of symplectic unitary
// transforms as the reference (Householder + Givens + Householder is one
// quaternion reflector followed by a quaternion phase), with one reflector
// and one quaternion matrix-vector product per column instead of two.
//
// Blocking follows the LAPACK zlatrd/zhetrd scheme lifted to quaternions: for
// a panel of nb columns, keep W (in the reduced columns of M) and the aux
// vectors Y with  H_current = H_panelstart - sum_i (W_i Y_i^H + Y_i W_i^H),
//   y = g - (c/2) w,  g = H_current w,  c = w^H g (real),
// and after the panel apply the structured rank-4nb update (her2k-like) to the
// lower triangles of the trailing A (Hermitian) and B (antisymmetric):
//   A -= Wa Ya^H + conj(Wb) conj(Yb)^H + Ya Wa^H + conj(Yb) conj(Wb)^H
//   B -= Wb Ya^H - conj(Wa) conj(Yb)^H + Yb Wa^H - conj(Ya) conj(Wb)^H
//
// Per column the launch sequence is
//   colupd  (finish y_{k-1}; apply the panel's deferred updates to column k;
//            norm partials; the last CTA to finish combines them into the
//            reflector head f, f m and the subdiagonal entry e_j)
//   hemv    (quaternion Hermitian mat-vec of the panel-start trailing matrix
//            with w = f x formed on the fly, lower triangles of A and B only,
//            per-tile deterministic partials; extra CTAs form the dot-product
//            partials of w against the panel's previous W, Y)
//   hreduce (sum tile partials and the dot partials, subtract the
//            deferred-update corrections -> g; partials of c; w written in
//            place of x)
// The kernels are launched with programmatic dependent launch (each starts
// with pdl_wait), so a kernel's launch overlaps the tail of the previous one.
// All arithmetic is FP64 (template R = double) for the plain path; the same
// kernels instantiate with R = float for the mixed-precision path, where norms
// and reflector scalars are formed in double here and in pairs of floats (48
// bits) in the resident kernel.
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_resident.h"
#include "zq_tc32.h"

#include <cuda.h>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace zq {

constexpr int RB = 32;        // rows per CTA for the row-parallel kernels
constexpr int TB = 64;        // tile edge of the trailing update
constexpr int NT = 256;       // threads per CTA

// ----------------------------------------------------------------------------
// reflector head of column j (warp 0 of one CTA): combines the colupd norm
// partials into nu = |x| and, with x_1 = (scal[0..3]), forms
//   f = 1 / sqrt(nu (nu + |x_1|)),  head of w = f (1 + nu/|x_1|) x_1,
//   e_j = -(nu/|x_1|) x_1  (x_1 = 0: head f nu, e_j = -nu; x = 0: no reflector),
// written to scal[4] (f), scal[5..8] (f m), e[4j..4j+3] and tau[j]. The reads
// bypass L1: the partials come from other CTAs of the running grid.
// ----------------------------------------------------------------------------
// The head's arithmetic (warp 0; lane 0 returns true with the results)
template <typename R>
__device__ bool head_math(const TridiagView<R>& v, int j, int nnp, double& f, double (&m)[4], double (&ee)[4]) {
  const int lane = threadIdx.x;
  const int L = v.n - 1 - j;
  if (lane >= 32 || L < 1) return false;  // the last column has no subdiagonal entry
  const double qa0 = __ldcg(v.scal + 0), qa1 = __ldcg(v.scal + 1), qb0 = __ldcg(v.scal + 2), qb1 = __ldcg(v.scal + 3);
  // nu = scale * sqrt(sum of ssq_i (s_i / scale)^2), scale = max s_i: up to
  // 256 partials are loaded once into registers (one memory latency, one
  // division); more fall back to two passes over memory
  constexpr int PL = 8;
  double sc = 0.0, sq = 0.0;
  if (nnp <= 32 * PL) {
    double ps[PL], pq[PL];
#pragma unroll
    for (int u = 0; u < PL; ++u) {
      const int i = lane + 32 * u;
      ps[u] = (i < nnp) ? __ldcg(v.npart + 2 * i) : 0.0;
      pq[u] = (i < nnp) ? __ldcg(v.npart + 2 * i + 1) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < PL; ++u) sc = fmax(sc, ps[u]);
    sc = warp_max(sc);
    const double inv = sc > 0.0 ? 1.0 / sc : 0.0;
#pragma unroll
    for (int u = 0; u < PL; ++u) { const double q = ps[u] * inv; sq += pq[u] * q * q; }
  } else {
    for (int i = lane; i < nnp; i += 32) sc = fmax(sc, __ldcg(v.npart + 2 * i));
    sc = warp_max(sc);
    const double inv = sc > 0.0 ? 1.0 / sc : 0.0;
    for (int i = lane; i < nnp; i += 32) {
      const double q = __ldcg(v.npart + 2 * i) * inv;
      sq += __ldcg(v.npart + 2 * i + 1) * q * q;
    }
  }
  sq = warp_sum(sq);
  const double nu = sc * sqrt(sq);
  if (lane != 0) return false;
  // |x_1| in units of the largest entry: its squares stay in range at any scale of the matrix
  const double inv = sc > 0.0 ? 1.0 / sc : 0.0;
  const double a0 = qa0 * inv, a1 = qa1 * inv, b0 = qb0 * inv, b1 = qb1 * inv;
  const double q1 = sc * sqrt(a0 * a0 + a1 * a1 + b0 * b0 + b1 * b1);
  f = 0.0;
  m[0] = m[1] = m[2] = m[3] = 0.0;
  ee[0] = qa0; ee[1] = qa1; ee[2] = qb0; ee[3] = qb1;   // L == 1: the entry itself is e_j
  if (L >= 2) {
    if (nu > 0.0) {
      if (q1 > 0.0) {
        const double s = nu / q1;
        f = 1.0 / (sqrt(nu) * sqrt(nu + q1));
        m[0] = qa0 * (1.0 + s); m[1] = qa1 * (1.0 + s); m[2] = qb0 * (1.0 + s); m[3] = qb1 * (1.0 + s);
        ee[0] = -s * qa0; ee[1] = -s * qa1; ee[2] = -s * qb0; ee[3] = -s * qb1;
      } else {
        f = 1.0 / nu;
        m[0] = nu;
        ee[0] = -nu; ee[1] = 0.0; ee[2] = 0.0; ee[3] = 0.0;
      }
    } else {
      ee[0] = ee[1] = ee[2] = ee[3] = 0.0;  // x == 0: nothing to reduce
    }
  }
  return true;
}

template <typename R>
__device__ void head_write(const TridiagView<R>& v, int j, double f, const double (&m)[4], const double (&ee)[4]) {
  v.scal[4] = f;
  for (int q = 0; q < 4; ++q) v.scal[5 + q] = m[q] * f;
  for (int q = 0; q < 4; ++q) v.e[4 * j + q] = ee[q];
  v.tau[j] = (f > 0.0) ? 1.0 : 0.0;
}

template <typename R>
__device__ void reflector_head(const TridiagView<R>& v, int j, int nnp) {
  double f, m[4], ee[4];
  if (head_math(v, j, nnp, f, m, ee)) head_write(v, j, f, m, ee);
}

// FP32 columns: squares of floats neither overflow nor vanish in double, so the
// partials are plain sums of squares, and the scalars come from two reciprocal
// square roots (with ss = |x|^2, q2 = |x_1|^2: g = sqrt(ss q2) = |x||x_1|,
// s = |x|/|x_1| = ss / g, f = 1 / sqrt(ss + g)): ~25 dependent FP64 instructions
// instead of ~130, each ~75 cycles here. The four components of m and e are
// formed by four lanes.
template <>
__device__ void reflector_head<float>(const TridiagView<float>& v, int j, int nnp) {
  const int lane = threadIdx.x;
  const int L = v.n - 1 - j;
  if (lane >= 32 || L < 1) return;  // the last column has no subdiagonal entry
  const double x1 = __ldcg(v.scal + (lane & 3));
  double ss = 0.0;
  for (int i = lane; i < nnp; i += 128) {  // four loads in flight
    double p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p[u] = i + 32 * u < nnp ? __ldcg(v.npart + 2 * (i + 32 * u) + 1) : 0.0;
    ss += (p[0] + p[1]) + (p[2] + p[3]);
  }
  double q2 = x1 * x1;
  q2 += __shfl_xor_sync(0xffffffffu, q2, 1);
  q2 += __shfl_xor_sync(0xffffffffu, q2, 2);
  ss = warp_sum(ss);
  double f = 0.0, m = 0.0, ee = x1;   // L == 1: the entry itself is e_j
  if (L >= 2) {
    const double t = ss * q2;
    if (t > 0.0) {
      const double rg = rsqrt(t);
      const double s = ss * rg;
      f = rsqrt(fma(t, rg, ss));
      m = x1 * fma(f, s, f);
      ee = -s * x1;
    } else if (ss > 0.0) {           // x_1 = 0
      f = rsqrt(ss);
      m = (lane & 3) == 0 ? 1.0 : 0.0;
      ee = (lane & 3) == 0 ? -ss * f : 0.0;
    } else {
      ee = ss == 0.0 ? 0.0 : ss;     // nothing to reduce (or not a number: keep it visible)
    }
  }
  if (lane >= 4) return;
  float* hf = reinterpret_cast<float*>(v.scal + 12);
  hf[1 + lane] = (float)m;
  v.e[4 * j + lane] = ee;
  if (lane == 0) {
    hf[0] = (float)f;
    hf[5] = (f > 0.0) ? 1.f : 0.f;
    v.tau[j] = (f > 0.0) ? 1.0 : 0.0;
  }
}

// the reflector head in the kernel's precision: f, f m (4 reals), and whether
// a reflector exists (f > 0)
template <typename R>
struct WHead {
  R f, m[4];
  bool live;
};

__device__ __forceinline__ void load_head(const TridiagView<float>& v, WHead<float>& h) {
  const float* hf = reinterpret_cast<const float*>(v.scal + 12);
  h.f = hf[0]; h.m[0] = hf[1]; h.m[1] = hf[2]; h.m[2] = hf[3]; h.m[3] = hf[4];
  h.live = hf[5] != 0.f;
}
__device__ __forceinline__ void load_head(const TridiagView<double>& v, WHead<double>& h) {
  h.f = v.scal[4]; h.m[0] = v.scal[5]; h.m[1] = v.scal[6]; h.m[2] = v.scal[7]; h.m[3] = v.scal[8];
  h.live = h.f > 0.0;
}

// w at row r of column j from x (= the stored column before hreduce writes w):
// the head row j+1 takes f m, the others f x; no reflector gives 0.
template <typename R>
__device__ __forceinline__ void w_from_x(const WHead<R>& h, int r, int j, cplx<R>& wa, cplx<R>& wb) {
  if (!h.live) { wa = czero<cplx<R>>(); wb = czero<cplx<R>>(); return; }
  if (r == j + 1) {
    wa = mk(h.m[0], h.m[1]);
    wb = mk(h.m[2], h.m[3]);
  } else {
    wa = cscale(wa, h.f);
    wb = cscale(wb, h.f);
  }
}

// ----------------------------------------------------------------------------
// colupd: rows [j, n) of column j
// ----------------------------------------------------------------------------
// Row block `bid` (rows j + RB bid ..) of column j; writes the block's norm
// partials npart[2 bid], npart[2 bid + 1]. Returns false when do_update is 0
// (only y_{k-1} finished).
template <typename R, int NTH>
__device__ bool colupd_block(const TridiagView<R>& v, int p, int j, int k, int ncp, int do_update, int bid) {
  constexpr int NGR = NTH / RB;  // reflector groups
  using Z = cplx<R>;
  const int n = v.n;
  const int64_t ld = v.ld;
  Z* A = v.M;
  Z* B = v.M + n;
  const int r0 = j + bid * RB;
  const int tid = threadIdx.x;
  const int row = tid & (RB - 1);
  const int grp = tid >> 5;
  const int r = r0 + row;
  __shared__ Z s_sc[4 * NBMAX];     // per i: ya_i[j], yb_i[j], wa_i[j], wb_i[j]
  __shared__ Z s_red[NGR][RB][2];
  __shared__ double s_red_d[2][NTH / 32];

  // Every load that does not depend on c_{k-1} is issued first, so the kernel
  // waits about one memory latency instead of one per phase. Reflector i of
  // the panel contributes through (w_i, y_i); y_{k-1} = g - (c/2) w_{k-1} is
  // formed once c is known.
  const bool live = r < n;
  // (1) y_{k-1} on this CTA's rows: w_{k-1} and g
  Z fwa = czero<Z>(), fwb = czero<Z>(), fga = czero<Z>(), fgb = czero<Z>();
  if (k > 0 && grp == 0 && live) {
    fwa = A[r + (int64_t)(j - 1) * ld]; fwb = B[r + (int64_t)(j - 1) * ld];
    fga = v.ga[r]; fgb = v.gb[r];
  }
  // (2) row-j scalars of reflector tid
  Z cwa = czero<Z>(), cwb = czero<Z>(), cya = czero<Z>(), cyb = czero<Z>();
  if (do_update && tid < k) {
    cwa = A[j + (int64_t)(p + tid) * ld]; cwb = B[j + (int64_t)(p + tid) * ld];
    if (tid == k - 1) { cya = v.ga[j]; cyb = v.gb[j]; }
    else { cya = v.Ya[j + (int64_t)tid * v.ldy]; cyb = v.Yb[j + (int64_t)tid * v.ldy]; }
  }
  // (3) this row's entries of the group's first two reflectors (i = grp, grp + NGR)
  Z pw[2][2], py[2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = grp + u * NGR;
    pw[u][0] = pw[u][1] = py[u][0] = py[u][1] = czero<Z>();
    if (do_update && live && i < k) {
      pw[u][0] = A[r + (int64_t)(p + i) * ld]; pw[u][1] = B[r + (int64_t)(p + i) * ld];
      if (i == k - 1) { py[u][0] = v.ga[r]; py[u][1] = v.gb[r]; }
      else { py[u][0] = v.Ya[r + (int64_t)i * v.ldy]; py[u][1] = v.Yb[r + (int64_t)i * v.ldy]; }
    }
  }
  // (4) the column itself
  Z x0a = czero<Z>(), x0b = czero<Z>();
  if (do_update && grp == 0 && live) { x0a = A[r + (int64_t)j * ld]; x0b = B[r + (int64_t)j * ld]; }
  // (5) c_{k-1} = sum of the previous column's partials (deterministic order)
  double cl = 0.0;
  if (k > 0)
    for (int i = tid; i < ncp; i += NTH) cl += v.cpart[i];
  const double csum = (k > 0) ? block_sum(cl, s_red_d[0]) : 0.0;
  const R half_c = (R)(0.5 * csum);

  // finish y_{k-1} = g - (c/2) w_{k-1} on this CTA's rows (rows >= j)
  if (k > 0 && grp == 0 && live) {
    v.Ya[r + (int64_t)(k - 1) * v.ldy] = csub(fga, cscale(fwa, half_c));
    v.Yb[r + (int64_t)(k - 1) * v.ldy] = csub(fgb, cscale(fwb, half_c));
  }
  if (!do_update) return false;

  // scalars at row j for every previous reflector of the panel (k < NBMAX = 128 <= NTH)
  if (tid < k) {
    if (tid == k - 1) { cya = csub(cya, cscale(cwa, half_c)); cyb = csub(cyb, cscale(cwb, half_c)); }
    s_sc[4 * tid + 0] = cya; s_sc[4 * tid + 1] = cyb; s_sc[4 * tid + 2] = cwa; s_sc[4 * tid + 3] = cwb;
  }
  __syncthreads();

  Z da = czero<Z>(), db = czero<Z>();
  auto contrib = [&](int i, Z wa, Z wb, Z ya, Z yb) {
    const Z sya = s_sc[4 * i + 0], syb = s_sc[4 * i + 1], swa = s_sc[4 * i + 2], swb = s_sc[4 * i + 3];
    if (i == k - 1) { ya = csub(ya, cscale(wa, half_c)); yb = csub(yb, cscale(wb, half_c)); }
    // A part: wa conj(ya_j) + conj(wb) yb_j + ya conj(wa_j) + conj(yb) wb_j
    cfmacb(da, wa, sya); cfmac(da, wb, syb); cfmacb(da, ya, swa); cfmac(da, yb, swb);
    // B part: wb conj(ya_j) - conj(wa) yb_j + yb conj(wa_j) - conj(ya) wb_j
    cfmacb(db, wb, sya); cfmac(db, cneg(wa), syb); cfmacb(db, yb, swa); cfmac(db, cneg(ya), swb);
  };
  if (live) {
    if (grp < k) contrib(grp, pw[0][0], pw[0][1], py[0][0], py[0][1]);
    if (grp + NGR < k) contrib(grp + NGR, pw[1][0], pw[1][1], py[1][0], py[1][1]);
    for (int i = grp + 2 * NGR; i < k; i += NGR) {  // panels wider than 2 NGR
      const Z wa = A[r + (int64_t)(p + i) * ld], wb = B[r + (int64_t)(p + i) * ld];
      Z ya, yb;
      if (i == k - 1) { ya = v.ga[r]; yb = v.gb[r]; }
      else { ya = v.Ya[r + (int64_t)i * v.ldy]; yb = v.Yb[r + (int64_t)i * v.ldy]; }
      contrib(i, wa, wb, ya, yb);
    }
  }
  s_red[grp][row][0] = da;
  s_red[grp][row][1] = db;
  __syncthreads();

  Z xa = czero<Z>(), xb = czero<Z>();
  if (grp == 0 && r < n) {
    Z ta = s_red[0][row][0], tb = s_red[0][row][1];
    for (int g2 = 1; g2 < NGR; ++g2) { ta = cadd(ta, s_red[g2][row][0]); tb = cadd(tb, s_red[g2][row][1]); }
    xa = csub(x0a, ta);
    xb = csub(x0b, tb);
    A[r + (int64_t)j * ld] = xa;
    B[r + (int64_t)j * ld] = xb;
    if (r == j) v.d[j] = (double)xa.x;
    if (r == j + 1) {
      v.scal[0] = (double)xa.x; v.scal[1] = (double)xa.y;
      v.scal[2] = (double)xb.x; v.scal[3] = (double)xb.y;
      __threadfence();  // before this CTA's arrival is counted
    }
  }
  if constexpr (std::is_same<R, float>::value) {
    // the rows lie in warp 0; plain squares (see reflector_head<float>)
    if (tid < 32) {
      double ss = 0.0;
      if (r < n && r > j) {
        const double a0 = xa.x, a1 = xa.y, b0 = xb.x, b1 = xb.y;
        ss = fma(a0, a0, a1 * a1) + fma(b0, b0, b1 * b1);
      }
      ss = warp_sum(ss);
      if (tid == 0) v.npart[2 * bid + 1] = ss;
    }
  } else {
    double sc = 0.0;  // local max-abs of x (rows >= j+1)
    if (grp == 0 && r < n && r > j)
      sc = fmax(fmax(fabs((double)xa.x), fabs((double)xa.y)), fmax(fabs((double)xb.x), fabs((double)xb.y)));
    // scaled sum of squares (LAPACK lassq style, combined across CTAs in reflect)
    const double bmax = block_max(sc, s_red_d[0]);
    double ss = 0.0;
    if (grp == 0 && r < n && r > j && bmax > 0.0) {
      const double inv = 1.0 / bmax;
      const double a0 = xa.x * inv, a1 = xa.y * inv, b0 = xb.x * inv, b1 = xb.y * inv;
      ss = a0 * a0 + a1 * a1 + b0 * b0 + b1 * b1;
    }
    const double bss = block_sum(ss, s_red_d[1]);
    if (tid == 0) {
      v.npart[2 * bid + 0] = bmax;
      v.npart[2 * bid + 1] = bss;
    }
  }
  return true;
}

template <typename R>
__global__ void __launch_bounds__(NT) k_colupd(TridiagView<R> v, int p, int j, int k, int ncp, int do_update) {
  pdl_wait();  // launched with launch_pdl: the previous kernel's results first
  if (!colupd_block<R, NT>(v, p, j, k, ncp, do_update, (int)blockIdx.x)) return;
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(v.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  // every CTA's partials (and x_1) are visible: form the reflector head once
  __threadfence();
  reflector_head(v, j, gridDim.x);
  if (threadIdx.x == 0) *v.counter = 0u;
}

// ----------------------------------------------------------------------------
// dot partials of w (rows [j+1, n)) against the panel's previous reflectors
// and aux vectors, DR rows per CTA (warp = 32 rows, lane = row):
//   <y_i,w> = ya^H wa + yb^H wb,  [y_i,w] = ya^T wb - yb^T wa,  same for w_i.
// The warps' sums meet in `scratch` (4 warps x k x 4) and the CTA writes one
// partial per (i, product).
// ----------------------------------------------------------------------------
constexpr int DR = 128;       // rows per dot-partial CTA
template <typename R>
__device__ void panel_dots(const TridiagView<R>& v, int p, int j, int k, int b, int ndot, cplx<R>* scratch) {
  using Z = cplx<R>;
  const int n = v.n;
  const int64_t ld = v.ld;
  const Z* A = v.M;
  const Z* B = v.M + n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gr = j + 1 + b * DR + warp * 32 + lane;
  const bool live = gr < n;
  WHead<R> h;
  Z xa = czero<Z>(), xb = czero<Z>();
  if (live) {
    load_head(v, h);
    xa = A[gr + (int64_t)j * ld];
    xb = B[gr + (int64_t)j * ld];
  }
  Z ya[4], yb[4], qa[4], qb[4];
  for (int i0 = 0; i0 < k; i0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      ya[u] = yb[u] = qa[u] = qb[u] = czero<Z>();
      if (live && i < k) {
        ya[u] = v.Ya[gr + (int64_t)i * v.ldy]; yb[u] = v.Yb[gr + (int64_t)i * v.ldy];
        qa[u] = A[gr + (int64_t)(p + i) * ld]; qb[u] = B[gr + (int64_t)(p + i) * ld];
      }
    }
    if (i0 == 0 && live) w_from_x<R>(h, gr, j, xa, xb);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      if (i >= k) break;
      Z d1 = czero<Z>(), d2 = czero<Z>(), d3 = czero<Z>(), d4 = czero<Z>();
      cfmac(d1, ya[u], xa); cfmac(d1, yb[u], xb);
      cfma(d2, ya[u], xb); cfma(d2, cneg(yb[u]), xa);
      cfmac(d3, qa[u], xa); cfmac(d3, qb[u], xb);
      cfma(d4, qa[u], xb); cfma(d4, cneg(qb[u]), xa);
      d1.x = warp_sum(d1.x); d1.y = warp_sum(d1.y);
      d2.x = warp_sum(d2.x); d2.y = warp_sum(d2.y);
      d3.x = warp_sum(d3.x); d3.y = warp_sum(d3.y);
      d4.x = warp_sum(d4.x); d4.y = warp_sum(d4.y);
      if (lane == 0) {
        Z* o = scratch + ((int64_t)warp * k + i) * 4;
        o[0] = d1; o[1] = d2; o[2] = d3; o[3] = d4;
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 4 * k; t += blockDim.x) {
    Z acc = scratch[t];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) acc = cadd(acc, scratch[w * 4 * k + t]);
    v.dpart[((int64_t)b * v.nbmax + (t >> 2)) * 4 + (t & 3)] = acc;
  }
  // the last dot CTA to finish sums all ndot partials into dots (fixed order:
  // nsplit threads per output over interleaved partials, then combined in order)
  __threadfence();
  __shared__ unsigned s_ticket;
  __syncthreads();
  if (threadIdx.x == 0) s_ticket = atomicAdd(v.counter + 1, 1u);
  __syncthreads();
  if (s_ticket != (unsigned)(ndot - 1)) return;
  __threadfence();
  const int no = 4 * k;
  if (no > (int)blockDim.x) {  // panels wider than 32: one thread per output
    for (int o = threadIdx.x; o < no; o += blockDim.x) {
      Z d = czero<Z>();
#pragma unroll 8
      for (int c = 0; c < ndot; ++c) d = cadd(d, __ldcg(v.dpart + ((int64_t)c * v.nbmax + (o >> 2)) * 4 + (o & 3)));
      v.dots[o] = d;
    }
  } else {
    const int nsplit = (int)blockDim.x / no;
    const int t = threadIdx.x % no, sp = threadIdx.x / no;
    Z acc = czero<Z>();
    if (sp < nsplit) {
#pragma unroll 8
      for (int c = sp; c < ndot; c += nsplit)
        acc = cadd(acc, __ldcg(v.dpart + ((int64_t)c * v.nbmax + (t >> 2)) * 4 + (t & 3)));
    }
    __syncthreads();  // scratch is free again
    scratch[threadIdx.x] = acc;
    __syncthreads();
    if ((int)threadIdx.x < no) {
      Z d = scratch[threadIdx.x];
      for (int u = 1; u < nsplit; ++u) d = cadd(d, scratch[u * no + threadIdx.x]);
      v.dots[threadIdx.x] = d;
    }
  }
  if (threadIdx.x == 0) v.counter[1] = 0u;
}

// ----------------------------------------------------------------------------
// hemv: quaternion Hermitian mat-vec of the panel-start trailing matrix.
//   Region rows/cols [b0, n); lower-triangle 32x32 tiles, one warp per tile,
//   after the first ndot CTAs, which form the panel dot partials. b0 is j + 1,
//   or the even row below it where pairs of rows are read at once (PAIR: FP32,
//   even n, 16-byte loads); row b0 < j + 1 then carries w = 0 and its output is
//   not read.
//   Lane (tr, tc) = (lane & 7, lane >> 3) owns four rows and eight columns of
//   the tile, read straight into registers; each element is used for its row
//   and its (conjugate-)transposed column, and the lanes' sums meet by halving
//   exchanges. Per row block and source block one partial (ga, gb) per row is
//   stored. A diagonal tile reads both triangles from the lower one and forms row
//   products only.
//   Bound: the matrix is read once per column (HBM above ~n = 3600, L2 below);
//   n = 4096, cold: column 0 134 MB in 31.8 us, column 2400 25 MB in 11.6 us. The
//   earlier form (tile in shared memory by TMA, a warp per product, products not
//   yet combined) was issue-bound at 1780 instructions of each of four warps per
//   tile against ~1300 of one here: 36.2 and 11.4 us, with twice the partial sums
//   for k_hreduce to read. Four CTAs per SM: 128 registers with a few spills in
//   the edge tiles beat 156 without (51.9 against 53.7 ms over the reduction).
// ----------------------------------------------------------------------------
constexpr int HT = 32;        // hemv tile edge
constexpr int HW = 4;         // tiles (warps) per CTA
template <typename R, bool PAIR>
__global__ void __launch_bounds__(32 * HW, sizeof(R) == 4 ? 4 : 2) k_hemv(TridiagView<R> v, int p, int j, int k, int ndot, int b0, int ntiles) {
  pdl_wait();  // launched with launch_pdl: the previous kernel's results first
  using Z = cplx<R>;
  // scratch of the dot CTAs (4 warps x k <= NBMAX x 4); the tile CTAs keep w of
  // their rows and columns there
  __shared__ __align__(16) Z s_buf[4 * NBMAX * 4];
  if ((int)blockIdx.x < ndot) {
    panel_dots(v, p, j, k, blockIdx.x, ndot, s_buf);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = (blockIdx.x - ndot) * HW + warp;
  if (t >= ntiles) return;
  const int n = v.n;
  const int64_t ld = v.ld;
  const Z* A = v.M;
  const Z* B = v.M + n;
  int I, J;
  tri_tile(t, I, J);
  const bool diag = (I == J);
  const int rbase = b0 + I * HT, cbase = b0 + J * HT;
  const int tr = lane & 7, tc = lane >> 3;
  // row i of this lane's four: pairs of consecutive rows in the PAIR form
  auto row_of = [&](int i) { return PAIR ? 16 * (i >> 1) + 2 * tr + (i & 1) : tr + 8 * i; };
  constexpr int CB = sizeof(R) == 4 ? 4 : 2;  // columns whose loads are in flight together
  Q4<R> m[CB][4];
  // inside the matrix and off the diagonal: unconditional loads from one base
  const bool inner = !diag && rbase + HT <= n;
  const Z* a0 = A + rbase + (int64_t)(cbase + tc) * ld;
  auto load_inner = [&](int c0) {
#pragma unroll
    for (int q = 0; q < CB; ++q) {
      const Z* a = a0 + (int64_t)(4 * (c0 + q)) * ld;
      if constexpr (PAIR) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(a + 16 * u + 2 * tr));
          const float4 y = __ldg(reinterpret_cast<const float4*>(a + n + 16 * u + 2 * tr));
          m[q][2 * u] = Q4<R>{x.x, x.y, y.x, y.y};
          m[q][2 * u + 1] = Q4<R>{x.z, x.w, y.z, y.w};
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const Z x = __ldg(a + tr + 8 * i), y = __ldg(a + n + tr + 8 * i);
          m[q][i] = Q4<R>{x.x, x.y, y.x, y.y};
        }
      }
    }
  };
  // elements of the diagonal tiles (above the diagonal from below it) and of the last row block
  auto load_edge = [&](int c0) {
#pragma unroll
    for (int q = 0; q < CB; ++q) {
      const int gc = cbase + tc + 4 * (c0 + q);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int gr = rbase + row_of(i);
        const int r = min(gr, n - 1), c = min(gc, n - 1);
        const bool low = r >= c;
        const int64_t o = low ? r + (int64_t)c * ld : c + (int64_t)r * ld;
        const Z x = __ldg(A + o), y = __ldg(B + o);
        // selects, not branches: the loads are in flight together
        const bool in = gr < n && gc < n, off = in && r != c;
        m[q][i].ax = in ? x.x : R(0);
        m[q][i].ay = off ? (low ? x.y : -x.y) : R(0);
        m[q][i].bx = off ? (low ? y.x : -y.x) : R(0);
        m[q][i].by = off ? (low ? y.y : -y.y) : R(0);
      }
    }
  };
  if (inner) load_inner(0); else load_edge(0);
  // w on the tile's rows and columns: one of each per lane, shared in the warp
  Q4<R>* sw = reinterpret_cast<Q4<R>*>(s_buf) + warp * 2 * HT;
  WHead<R> h;
  load_head(v, h);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int g = (q ? cbase : rbase) + lane, gl = g < n ? g : n - 1;
    Z wa = A[gl + (int64_t)j * ld], wb = B[gl + (int64_t)j * ld];
    w_from_x<R>(h, g, j, wa, wb);
    if (g <= j || g >= n) { wa = czero<Z>(); wb = czero<Z>(); }
    q_store(sw + q * HT + lane, Q4<R>{wa.x, wa.y, wb.x, wb.y});
  }
  __syncwarp();
  R rs[16], cs[32];
#pragma unroll
  for (int q = 0; q < 16; ++q) rs[q] = R(0);
#pragma unroll
  for (int q = 0; q < 32; ++q) cs[q] = R(0);
#pragma unroll
  for (int c0 = 0; c0 < 8; c0 += CB) {
    if (c0 > 0) {
      if (inner) load_inner(c0); else load_edge(c0);
    }
#pragma unroll
    for (int q = 0; q < CB; ++q) {
      const Q4<R> wc = sw[HT + tc + 4 * (c0 + q)];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        row_prod(rs + 4 * i, m[q][i], wc);
        col_prod(cs + 4 * (c0 + q), m[q][i], sw[row_of(i)]);
      }
    }
  }
  Q4<R>* part = reinterpret_cast<Q4<R>*>(v.hpart);
  scatter_sum<16, 16, 8, R>(rs, lane);   // over the column lanes: lane tc is left with row tc
  q_store(part + ((int64_t)I * v.hblk + J) * HT + row_of(tc), Q4<R>{rs[0], rs[1], rs[2], rs[3]});
  if (!diag) {
    scatter_sum<32, 4, 1, R>(cs, lane);  // over the row lanes: lane tr is left with column tr
    q_store(part + ((int64_t)J * v.hblk + I) * HT + tc + 4 * tr, Q4<R>{cs[0], cs[1], cs[2], cs[3]});
  }
}

// ----------------------------------------------------------------------------
// hreduce: g = H_panelstart w - corrections, for rows [j+1, n); c partials;
//   w = f x written in place of x.
//   T is the hemv tile edge used for this column; nblk its number of blocks.
//   HRB rows per CTA; NSPL threads per (row, product) sum the hemv tile
//   partials (fixed split and combine order: deterministic). The panel dot
//   products come finished from the hemv grid (dots). All loads that do not
//   depend on one another are issued before the first is used.
// ----------------------------------------------------------------------------
constexpr int HRB = 8;                 // rows per CTA
template <typename R>
__global__ void __launch_bounds__(NT) k_hreduce(TridiagView<R> v, int p, int j, int k, int T, int nblk, int zero_mode,
                                                int sh) {
  pdl_wait();  // launched with launch_pdl: the previous kernel's results first
  constexpr int HNG = NT / HRB;           // reflector groups for the corrections
  constexpr int NSPL = NT / (2 * HRB);    // threads per (row, part) for the tile partials
  const int bid = (int)blockIdx.x;        // rows j + 1 + HRB bid ..
  using Z = cplx<R>;
  const int n = v.n;
  const int64_t ld = v.ld;
  Z* A = v.M;
  Z* B = v.M + n;
  const int r0 = j + 1;
  const int tid = threadIdx.x;
  const int row = tid & (HRB - 1), grp = tid / HRB;
  const int r = r0 + bid * HRB + row;
  __shared__ Z s_v[HRB][2];
  __shared__ Z s_dots[4 * NBMAX];
  __shared__ Z s_part[NSPL][2 * HRB];
  __shared__ Z s_red[HNG][HRB][2];
  // this row's x and the reflector head (w = f x is written in place at the end)
  WHead<R> h;
  Z xa = czero<Z>(), xb = czero<Z>();
  if (grp == 0 && r < n) {
    load_head(v, h);
    xa = A[r + (int64_t)j * ld];
    xb = B[r + (int64_t)j * ld];
  }
  // the group's first reflector (w_i, y_i) at this row, and the panel dots
  Z cwa = czero<Z>(), cwb = czero<Z>(), cya = czero<Z>(), cyb = czero<Z>(), dt = czero<Z>();
  if (!zero_mode) {
    if (r < n && grp < k) {
      cwa = A[r + (int64_t)(p + grp) * ld]; cwb = B[r + (int64_t)(p + grp) * ld];
      cya = v.Ya[r + (int64_t)grp * v.ldy]; cyb = v.Yb[r + (int64_t)grp * v.ldy];
    }
    if (tid < 4 * k) dt = v.dots[tid];
    // tile partials: output o = (row, ga or gb); split sp sums blocks S = sp, sp + NSPL, ...
    const int o = tid & (2 * HRB - 1), sp = tid / (2 * HRB);
    const int lr = bid * HRB + (o >> 1);
    Z s0 = czero<Z>(), s1 = czero<Z>(), s2 = czero<Z>(), s3 = czero<Z>();
    if (r0 + lr < n) {
      const int Rb = (lr + sh) / T, off = (lr + sh) % T;  // the hemv tile grid starts sh rows above r0
      const Z* base = v.hpart + (((int64_t)Rb * v.hblk) * T + off) * 2 + (o & 1);
      const int64_t stride = (int64_t)T * 2;
      int S = sp;
#pragma unroll 2
      for (; S + 3 * NSPL < nblk; S += 4 * NSPL) {
        const Z a0 = base[S * stride], a1 = base[(S + NSPL) * stride], a2 = base[(S + 2 * NSPL) * stride],
                a3 = base[(S + 3 * NSPL) * stride];
        s0 = cadd(s0, a0); s1 = cadd(s1, a1); s2 = cadd(s2, a2); s3 = cadd(s3, a3);
      }
      for (; S < nblk; S += NSPL) s0 = cadd(s0, base[S * stride]);
    }
    s_part[sp][o] = cadd(cadd(s0, s2), cadd(s1, s3));
    if (tid < 4 * k) s_dots[tid] = dt;
    for (int q = tid + NT; q < 4 * k; q += NT) s_dots[q] = v.dots[q];  // wide panels
  }
  __syncthreads();
  if (!zero_mode && tid < 2 * HRB) {
    Z t = s_part[0][tid];
#pragma unroll
    for (int u = 1; u < NSPL; ++u) t = cadd(t, s_part[u][tid]);
    s_v[tid >> 1][tid & 1] = t;
  }
  // deferred-update corrections, reflectors split over the groups
  Z ta = czero<Z>(), tb = czero<Z>();
  if (!zero_mode && r < n) {
    for (int i = grp; i < k; i += HNG) {
      Z wa = cwa, wb = cwb, ya = cya, yb = cyb;
      if (i != grp) {
        wa = A[r + (int64_t)(p + i) * ld]; wb = B[r + (int64_t)(p + i) * ld];
        ya = v.Ya[r + (int64_t)i * v.ldy]; yb = v.Yb[r + (int64_t)i * v.ldy];
      }
      const Z s1 = s_dots[4 * i + 0], s2 = s_dots[4 * i + 1], s3 = s_dots[4 * i + 2], s4 = s_dots[4 * i + 3];
      // ga -= wa s1 - conj(wb) s2 + ya s3 - conj(yb) s4
      // gb -= wb s1 + conj(wa) s2 + yb s3 + conj(ya) s4
      cfma(ta, wa, s1); cfmac(ta, cneg(wb), s2); cfma(ta, ya, s3); cfmac(ta, cneg(yb), s4);
      cfma(tb, wb, s1); cfmac(tb, wa, s2); cfma(tb, yb, s3); cfmac(tb, ya, s4);
    }
  }
  s_red[grp][row][0] = ta;
  s_red[grp][row][1] = tb;
  __syncthreads();
  double cp = 0.0;
  if (grp == 0 && r < n) {
    Z wa = xa, wb = xb;
    w_from_x<R>(h, r, j, wa, wb);
    A[r + (int64_t)j * ld] = wa;
    B[r + (int64_t)j * ld] = wb;
    Z ga = czero<Z>(), gb = czero<Z>();
    if (!zero_mode) {
      ga = s_v[row][0];
      gb = s_v[row][1];
      const int ng = k < HNG ? k : HNG;   // groups that hold a correction
      for (int g2 = 0; g2 < ng; ++g2) { ga = csub(ga, s_red[g2][row][0]); gb = csub(gb, s_red[g2][row][1]); }
      cp = (double)(wa.x * ga.x + wa.y * ga.y + wb.x * gb.x + wb.y * gb.y);
    }
    v.ga[r] = ga;
    v.gb[r] = gb;
  }
  if (tid < 32) {  // the rows lie in the first eight lanes
#pragma unroll
    for (int o = HRB / 2; o > 0; o >>= 1) cp += __shfl_xor_sync(0xffffffffu, cp, o);
    if (tid == 0) v.cpart[bid] = cp;
  }
}

// ----------------------------------------------------------------------------
// trailing update of the lower triangles of A (incl. diagonal) and B (strict)
// region [t0, n) x [t0, n), rank-4*nbp structured update.
// ----------------------------------------------------------------------------
constexpr int KC = 4;  // reflectors per smem stage (FP64)

// the rank-4 KC products of one K stage into the 4 x 4 complex micro-tiles
template <typename Z>
__device__ __forceinline__ void trail_stage(const Z (&sr)[4][KC][TB], const Z (&sc)[4][KC][TB], int tr, int tc,
                                            Z (&accA)[4][4], Z (&accB)[4][4]) {
#pragma unroll
  for (int kk = 0; kk < KC; ++kk) {
    Z rwa[4], rwb[4], rya[4], ryb[4], cwa[4], cwb[4], cya[4], cyb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      rwa[q] = sr[0][kk][4 * tr + q]; rwb[q] = sr[1][kk][4 * tr + q];
      rya[q] = sr[2][kk][4 * tr + q]; ryb[q] = sr[3][kk][4 * tr + q];
      cwa[q] = sc[0][kk][4 * tc + q]; cwb[q] = sc[1][kk][4 * tc + q];
      cya[q] = sc[2][kk][4 * tc + q]; cyb[q] = sc[3][kk][4 * tc + q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // A += wa conj(ya) + conj(wb) yb + ya conj(wa) + conj(yb) wb
        cfmacb(accA[q][c], rwa[q], cya[c]); cfmac(accA[q][c], rwb[q], cyb[c]);
        cfmacb(accA[q][c], rya[q], cwa[c]); cfmac(accA[q][c], ryb[q], cwb[c]);
        // B += wb conj(ya) - conj(wa) yb + yb conj(wa) - conj(ya) wb
        cfmacb(accB[q][c], rwb[q], cya[c]); cfmac(accB[q][c], cneg(rwa[q]), cyb[c]);
        cfmacb(accB[q][c], ryb[q], cwa[c]); cfmac(accB[q][c], cneg(rya[q]), cwb[c]);
      }
  }
}

// FP32: 64 x 32 tiles, 128 threads of 4 x 4 quaternion entries; packed FP32 instructions
// on pairs of rows, so that an entry pair's 32 products take 32 issue slots. All of a
// chunk's reflectors are staged at once (components apart, for the pairs), one barrier
// on each side; three CTAs per SM cover each other's staging and read-modify-write.
// Bound: the FP32 pipe (n = 4096: 3.4e11 multiply-adds, 9.3 ms). 64 x 64 tiles of 256
// threads, one CTA per SM, scalar: 20.5 ms, now 14.5.
constexpr int TF_R = 64, TF_C = 32, TF_K = 16;
using F32x2 = unsigned long long;
__device__ __forceinline__ void fma2(F32x2& acc, F32x2 a, F32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ F32x2 both(float v) {
  F32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float2 halves(F32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void copy_async4(float* smem, const float* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__global__ void __launch_bounds__(128, 3) k_trail_f32(TridiagView<float> v, int p, int nbp, int t0) {
  pdl_wait();
  // [reflector][component of wa, wb, ya, yb][row or column]
  __shared__ __align__(16) float sr[TF_K][8][TF_R];
  __shared__ __align__(16) float sc[TF_K][8][TF_C];
  const int n = v.n;
  const int64_t ld = v.ld;
  float2* A = v.M;
  float2* B = v.M + n;
  int I, J;
  tri_tile((int)(blockIdx.x >> 1), I, J);
  const int rb = t0 + I * TF_R, cb = t0 + J * TF_R + TF_C * (int)(blockIdx.x & 1);
  if (cb >= n) return;
  const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
  F32x2 acc[4][4][2];  // component, column, pair of rows
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[k][c][0] = acc[k][c][1] = 0ull;
  for (int k0 = 0; k0 < nbp; k0 += TF_K) {
    const int kt = min(TF_K, nbp - k0);
    if (k0) __syncthreads();
    // rows, then columns, by asynchronous copies of one component each: all in flight
    // at once (through registers their latency took as long as the products)
    auto source = [&](int vec, int kk) -> const float* {
      const int kc = k0 + kk;
      const float2* q = vec == 0 ? A + (int64_t)(p + kc) * ld : vec == 1 ? B + (int64_t)(p + kc) * ld
                      : vec == 2 ? v.Ya + (int64_t)kc * v.ldy : v.Yb + (int64_t)kc * v.ldy;
      return reinterpret_cast<const float*>(q);
    };
    {
      const int row = tid & (TF_R - 1), col = tid & (TF_C - 1);
      const int gr = 2 * min(rb + row, n - 1), gc = 2 * min(cb + col, n - 1);
#pragma unroll
      for (int vec = 0; vec < 4; ++vec) {
        for (int kk = tid / TF_R; kk < kt; kk += 128 / TF_R) {
          const float* src = source(vec, kk) + gr;
          copy_async4(&sr[kk][2 * vec][row], src);
          copy_async4(&sr[kk][2 * vec + 1][row], src + 1);
        }
        for (int kk = tid / TF_C; kk < kt; kk += 128 / TF_C) {
          const float* src = source(vec, kk) + gc;
          copy_async4(&sc[kk][2 * vec][col], src);
          copy_async4(&sc[kk][2 * vec + 1][col], src + 1);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
#pragma unroll 1
    for (int kk = 0; kk < kt; ++kk) {
      F32x2 r[8][2];
      float4 cv[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&sr[kk][s][4 * tr]);
        r[s][0] = q.x;
        r[s][1] = q.y;
        cv[s] = *reinterpret_cast<const float4*>(&sc[kk][s][4 * tc]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // w of the row with y of the column, then y of the row with w of the column
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          float x[4];
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const float4 q = cv[4 * (1 - t) + s];
            x[s] = c == 0 ? q.x : c == 1 ? q.y : c == 2 ? q.z : q.w;
          }
          const F32x2 ax = both(x[0]), ay = both(x[1]), bx = both(x[2]), by = both(x[3]);
          const F32x2 nay = both(-x[1]), nbx = both(-x[2]), nby = both(-x[3]);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const F32x2 rax = r[4 * t][h], ray = r[4 * t + 1][h], rbx = r[4 * t + 2][h], rby = r[4 * t + 3][h];
            fma2(acc[0][c][h], rax, ax); fma2(acc[1][c][h], ray, ax); fma2(acc[2][c][h], rbx, ax); fma2(acc[3][c][h], rby, ax);
            fma2(acc[0][c][h], ray, ay); fma2(acc[1][c][h], rax, nay); fma2(acc[2][c][h], rby, ay); fma2(acc[3][c][h], rbx, nay);
            fma2(acc[0][c][h], rbx, bx); fma2(acc[1][c][h], rby, nbx); fma2(acc[2][c][h], rax, nbx); fma2(acc[3][c][h], ray, bx);
            fma2(acc[0][c][h], rby, by); fma2(acc[1][c][h], rbx, by); fma2(acc[2][c][h], ray, nby); fma2(acc[3][c][h], rax, nby);
          }
        }
      }
    }
  }
  const bool whole = rb >= cb + TF_C && rb + TF_R <= n;
  const int gr = rb + 4 * tr;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int gc = cb + 4 * tc + c;
    if (gc >= n) continue;
    float2* pa = A + gr + (int64_t)gc * ld;
    float2* pb = B + gr + (int64_t)gc * ld;
    const float2 a0x = halves(acc[0][c][0]), a0y = halves(acc[1][c][0]), a1x = halves(acc[0][c][1]), a1y = halves(acc[1][c][1]);
    const float2 b0x = halves(acc[2][c][0]), b0y = halves(acc[3][c][0]), b1x = halves(acc[2][c][1]), b1y = halves(acc[3][c][1]);
    const float2 ua[4] = {{a0x.x, a0y.x}, {a0x.y, a0y.y}, {a1x.x, a1y.x}, {a1x.y, a1y.y}};
    const float2 ub[4] = {{b0x.x, b0y.x}, {b0x.y, b0y.y}, {b1x.x, b1y.x}, {b1x.y, b1y.y}};
    if (whole) {
      float2 x[4], y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { x[q] = pa[q]; y[q] = pb[q]; }
#pragma unroll
      for (int q = 0; q < 4; ++q) { pa[q] = csub(x[q], ua[q]); pb[q] = csub(y[q], ub[q]); }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (gr + q >= n || gr + q < gc) continue;
        pa[q] = csub(pa[q], ua[q]);
        if (gr + q > gc) pb[q] = csub(pb[q], ub[q]);
      }
    }
  }
}

template <typename R>
__global__ void __launch_bounds__(NT) k_trail(TridiagView<R> v, int p, int nbp, int t0) {
  pdl_wait();  // launched with launch_pdl: the previous kernel's results first
  using Z = cplx<R>;
  const int n = v.n;
  const int64_t ld = v.ld;
  Z* A = v.M;
  Z* B = v.M + n;
  const int t = blockIdx.x;
  int I, J;
  tri_tile(t, I, J);
  const int tid = threadIdx.x;
  const int tr = tid & 15, tc = tid >> 4;
  const int rb = t0 + I * TB, cb = t0 + J * TB;
  Z accA[4][4], accB[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int c = 0; c < 4; ++c) { accA[q][c] = czero<Z>(); accB[q][c] = czero<Z>(); }

  {
    // [vector: wa, wb, ya, yb][kk][row]
    __shared__ Z s_r[4][KC][TB];
    __shared__ Z s_c[4][KC][TB];
    for (int k0 = 0; k0 < nbp; k0 += KC) {
      __syncthreads();
      for (int e = tid; e < 4 * KC * TB; e += NT) {
        const int row = e % TB, kk = (e / TB) % KC, vec = e / (TB * KC);
        const int kg = k0 + kk;
        Z vr = czero<Z>(), vc = czero<Z>();
        if (kg < nbp) {
          const int gr = rb + row, gc = cb + row;
          if (gr < n) {
            if (vec == 0) vr = A[gr + (int64_t)(p + kg) * ld];
            else if (vec == 1) vr = B[gr + (int64_t)(p + kg) * ld];
            else if (vec == 2) vr = v.Ya[gr + (int64_t)kg * v.ldy];
            else vr = v.Yb[gr + (int64_t)kg * v.ldy];
          }
          if (gc < n) {
            if (vec == 0) vc = A[gc + (int64_t)(p + kg) * ld];
            else if (vec == 1) vc = B[gc + (int64_t)(p + kg) * ld];
            else if (vec == 2) vc = v.Ya[gc + (int64_t)kg * v.ldy];
            else vc = v.Yb[gc + (int64_t)kg * v.ldy];
          }
        }
        s_r[vec][kk][row] = vr;
        s_c[vec][kk][row] = vc;
      }
      __syncthreads();
      trail_stage<Z>(s_r, s_c, tr, tc, accA, accB);
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int gc = cb + 4 * tc + c;
    if (gc >= n) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int gr = rb + 4 * tr + q;
      if (gr >= n || gr < gc) continue;
      const int64_t o = gr + (int64_t)gc * ld;
      A[o] = csub(A[o], accA[q][c]);
      if (gr > gc) B[o] = csub(B[o], accB[q][c]);
    }
  }
}

// The same trailing update on the tensor cores (zq_tc32.cu), FP32 path, used
// only where ZQ_TC32_USES names it: the lower triangles of the (n - t0)^2
// trailing blocks of A and B take one rank-4 nbp product each,
//   A -= [Wa | conj(Wb) | Ya | conj(Yb)] [conj(Ya) | Yb | conj(Wa) | Wb]^T   (i >= j)
//   B -= [Wb | -conj(Wa) | Yb | -conj(Ya)] [conj(Ya) | Yb | conj(Wa) | Wb]^T (i > j)
// with W the panel's reflectors (stored in place, columns p..p+nbp-1) and Y
// its aux vectors, all read at rows t0.. (128 x 128 lower tiles only).
static Tc32Src trail_src(const float2* p, int64_t ld, int conj, float sign) {
  Tc32Src s{};
  s.p = reinterpret_cast<const float*>(p); s.ld = ld; s.kfast = 0; s.conj = conj; s.sign = sign;
  return s;
}
static int trail_tc32(const TridiagView<float>& v, int p, int nbp, int t0, cudaStream_t st) {
  const int n = v.n;
  const int64_t ld = v.ld;
  const float2* Wa = v.M + t0 + (int64_t)p * ld;
  const float2* Wb = v.M + n + t0 + (int64_t)p * ld;
  const float2* Ya = v.Ya + t0;
  const float2* Yb = v.Yb + t0;
  for (int half = 0; half < 2; ++half) {
    Tc32Args t{};
    t.cplx = 1; t.m = n - t0; t.n = n - t0; t.nseg = 4;
    // column operand, shared by both updates
    t.seg[0].b = trail_src(Ya, v.ldy, 1, 1.f);
    t.seg[1].b = trail_src(Yb, v.ldy, 0, 1.f);
    t.seg[2].b = trail_src(Wa, ld, 1, 1.f);
    t.seg[3].b = trail_src(Wb, ld, 0, 1.f);
    if (half == 0) {
      t.seg[0].a = trail_src(Wa, ld, 0, 1.f);
      t.seg[1].a = trail_src(Wb, ld, 1, 1.f);
      t.seg[2].a = trail_src(Ya, v.ldy, 0, 1.f);
      t.seg[3].a = trail_src(Yb, v.ldy, 1, 1.f);
    } else {
      t.seg[0].a = trail_src(Wb, ld, 0, 1.f);
      t.seg[1].a = trail_src(Wa, ld, 1, -1.f);
      t.seg[2].a = trail_src(Yb, v.ldy, 0, 1.f);
      t.seg[3].a = trail_src(Ya, v.ldy, 1, -1.f);
    }
    for (int q = 0; q < 4; ++q) t.seg[q].k = nbp;
    t.alpha = make_float2(-1.f, 0.f); t.beta = make_float2(1.f, 0.f);
    t.C = reinterpret_cast<float*>(v.M + (half ? n : 0) + t0 + (int64_t)t0 * ld);
    t.ldc = ld;
    t.tri = half ? 2 : 1;
    t.splits = 1;
    t.err = v.tc_err;
    if (int rc = tc32_gemm(t, st)) return rc;
  }
  return ZQ_OK;
}


// ----------------------------------------------------------------------------
// host driver
// ----------------------------------------------------------------------------
template <typename R>
int tridiagonalize(TridiagView<R> v, int nb, cudaStream_t st) {
  const int n = v.n;
  if (n <= 0) return ZQ_OK;
  if (nb > v.nbmax) nb = v.nbmax;
  if (nb < 1) nb = 1;
  ZQ_CUDA(cudaMemsetAsync(v.counter, 0, 2 * sizeof(unsigned), st));
  // FP32 with even n: rows are read in aligned pairs (A and B both start on a
  // 16-byte boundary in every column)
  const bool pair = std::is_same<R, float>::value && (n % 2) == 0 && (v.ld % 2) == 0 &&
                    (reinterpret_cast<uintptr_t>(v.M) % 16) == 0;
  int ncp = 0;  // number of c partials of the previous column
  // the last columns (all of them for orders that fit) run with the trailing
  // block held in shared memory
  const int rmax = resident_max<R>(v.ctas);
  for (int p = 0; p < n; p += nb) {
    if (n - p <= rmax) return tri_resident<R>(v, p, v.ctas, st);
    const int nbp = (nb < n - p) ? nb : (n - p);
    for (int k = 0; k < nbp; ++k) {
      const int j = p + k;
      const int L = n - 1 - j;
      const int ncta1 = ceil_div(n - j, RB);
      prof_begin(PC_PANEL, st);
      ZQ_CUDA(launch_pdl(k_colupd<R>, dim3(ncta1), dim3(NT), st, v, p, j, k, ncp, 1));
      count_launch();
      if (L < 1) { prof_end(PC_PANEL, st); ncp = 0; continue; }
      const int T = HT;
      const int b0 = pair ? ((j + 1) & ~1) : (j + 1);  // first row of the tile grid
      const int sh = (j + 1) - b0;
      const int nblk = ceil_div(n - b0, T);
      const int ndot = (k > 0 && L >= 2) ? ceil_div(L, DR) : 0;  // dot-partial CTAs of the hemv grid
      prof_end(PC_PANEL, st);
      if (L >= 2) {
        prof_begin(PC_HEMV, st);
        const int ntiles = nblk * (nblk + 1) / 2;
        const dim3 grid(ceil_div(ntiles, HW) + ndot);
        if constexpr (std::is_same<R, float>::value) {
          if (pair) ZQ_CUDA(launch_pdl(k_hemv<R, true>, grid, dim3(32 * HW), st, v, p, j, k, ndot, b0, ntiles));
          else ZQ_CUDA(launch_pdl(k_hemv<R, false>, grid, dim3(32 * HW), st, v, p, j, k, ndot, b0, ntiles));
        } else {
          ZQ_CUDA(launch_pdl(k_hemv<R, false>, grid, dim3(32 * HW), st, v, p, j, k, ndot, b0, ntiles));
        }
        count_launch();
        prof_end(PC_HEMV, st);
      }
      prof_begin(PC_PANEL, st);
      const int nhr = ceil_div(L, HRB);
      ZQ_CUDA(launch_pdl(k_hreduce<R>, dim3(nhr), dim3(NT), st, v, p, j, k, T, nblk, L < 2 ? 1 : 0, sh));
      count_launch();
      prof_end(PC_PANEL, st);
      ncp = nhr;
    }
    const int t0 = p + nbp;
    if (t0 < n) {
      // finish y of the panel's last reflector (rows >= t0), then update
      prof_begin(PC_PANEL, st);
      ZQ_CUDA(launch_pdl(k_colupd<R>, dim3(ceil_div(n - t0, RB)), dim3(NT), st, v, p, t0, nbp, ncp, 0));
      count_launch();
      prof_end(PC_PANEL, st);
      const int nblk = ceil_div(n - t0, TB);
      prof_begin(PC_TRAIL, st);
      if constexpr (std::is_same<R, float>::value) {
        if (v.tc_err && fp32_products_on_tensor_cores(TC_USE_TRAIL)) {
          if (int rc = trail_tc32(v, p, nbp, t0, st)) return rc;
          prof_end(PC_TRAIL, st);
          ncp = 0;
          continue;
        }
      }
      if constexpr (std::is_same<R, float>::value)
        ZQ_CUDA(launch_pdl(k_trail_f32, dim3(nblk * (nblk + 1)), dim3(128), st, v, p, nbp, t0));
      else
        ZQ_CUDA(launch_pdl(k_trail<R>, dim3(nblk * (nblk + 1) / 2), dim3(NT), st, v, p, nbp, t0));
      count_launch();
      prof_end(PC_TRAIL, st);
      ncp = 0;
    }
  }
  return ZQ_OK;
}

template <typename R>
size_t tridiag_workspace_bytes(int n, int nbmax) {
  using Z = cplx<R>;
  const size_t hblk = (size_t)ceil_div(n > 0 ? n : 1, 32);
  size_t b = 0;
  b += sizeof(Z) * (2 * (size_t)n * nbmax);          // Ya, Yb
  b += sizeof(Z) * (2 * (size_t)n);                   // ga, gb
  b += sizeof(Z) * ((hblk + 2) * (hblk + 2) * 32 * 2);  // hpart
  b += sizeof(Z) * (hblk * nbmax * 4);                // dpart
  b += sizeof(Z) * (4 * (size_t)nbmax);               // dots
  b += sizeof(double) * (2 * hblk + 16);              // npart (2 hblk), scal
  b += sizeof(double) * ((size_t)ceil_div(n > 0 ? n : 1, HRB) + 1);  // cpart (one per hreduce CTA)
  b += sizeof(unsigned) * 8;                          // counters (colupd, dots)
  b += resident_workspace_bytes(n, sizeof(R));
  return b + 17 * 256;
}

template <typename R>
TridiagView<R> tridiag_bind(void* ws, cplx<R>* M, int n, int64_t ld, int nbmax, double* d, double* e, double* tau) {
  using Z = cplx<R>;
  TridiagView<R> v{};
  const int hblk = ceil_div(n > 0 ? n : 1, 32);
  char* p = reinterpret_cast<char*>(ws);
  auto take = [&](size_t bytes) { char* q = p; p += (bytes + 255) & ~(size_t)255; return q; };
  v.M = M; v.n = n; v.ld = ld; v.nbmax = nbmax; v.ldy = n > 0 ? n : 1; v.hblk = hblk;
  v.Ya = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)n * nbmax));
  v.Yb = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)n * nbmax));
  v.ga = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)n));
  v.gb = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)n));
  v.hpart = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)(hblk + 2) * (hblk + 2) * 32 * 2));
  v.dpart = reinterpret_cast<Z*>(take(sizeof(Z) * (size_t)hblk * nbmax * 4));
  v.dots = reinterpret_cast<Z*>(take(sizeof(Z) * 4 * (size_t)nbmax));
  v.npart = reinterpret_cast<double*>(take(sizeof(double) * 2 * hblk));
  v.cpart = reinterpret_cast<double*>(take(sizeof(double) * ((size_t)ceil_div(n > 0 ? n : 1, HRB) + 1)));
  v.scal = reinterpret_cast<double*>(take(sizeof(double) * 16));
  v.counter = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * 8));
  v.rws = take(resident_workspace_bytes(n, sizeof(R)));
  v.ctas = resident_ctas(n, true);
  v.d = d; v.e = e; v.tau = tau;
  return v;
}

template size_t tridiag_workspace_bytes<double>(int, int);
template size_t tridiag_workspace_bytes<float>(int, int);
template TridiagView<double> tridiag_bind<double>(void*, cplx<double>*, int, int64_t, int, double*, double*, double*);
template TridiagView<float> tridiag_bind<float>(void*, cplx<float>*, int, int64_t, int, double*, double*, double*);

template int tridiagonalize<double>(TridiagView<double>, int, cudaStream_t);
template int tridiagonalize<float>(TridiagView<float>, int, cudaStream_t);

}  // namespace zq
