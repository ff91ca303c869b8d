// Batches of matrices of order up to 32: one warp per matrix, which stays in
// shared memory from the first load to the last store.
//
// Reference: the steps of ts::zquatev (zquatev.cc:42-100) once per matrix; it has
// no batched entry point.
//
// What bounds it: the FP64 pipe. An instruction holds its SM quadrant's pipe for
// 64 cycles whether one lane is active or 32, so the work is laid out by lanes:
//   1. reduction: the matrix is kept with both triangles, H w takes a lane per row
//      (several lanes per row once the trailing block has at most 16 rows), the
//      rank-2 update a lane per entry of the lower triangle, mirrored on the store;
//   2. phases and QL: serial chains, so one warp of the CTA runs them for all the
//      CTA's matrices, a lane each; the rotations of some sweeps are recorded, then
//      every warp applies those of its matrix to the rows of Z, a lane per row;
//   3. back-transform: a lane per eigenvector (several once n <= 16), so the inner
//      products with a reflector need no exchange between lanes.
// 2000 matrices of order 19: 2.1 ms (8.3 ms with a lane per row in every step, a
// matrix in global memory and the QL chain in one lane of each warp); of order 8 0.44
// ms (1.6), of order 32 11.4 ms (35, a CTA per matrix), where 39 KB of shared memory
// each leave four matrices to an SM.
#include "zq_batched.h"
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_quat.cuh"
#include "zq_recip.cuh"

namespace zq {
namespace {

constexpr int SMALL_WARPS = 8;  // matrices per CTA at most

// Shared memory of one matrix, in doubles (nmax sets the offsets, n the row strides):
//   planes of A and B, ld = n | 1 so rows and columns both miss each other's banks;
//     later X in the same place, with Z in the last quarter until X is formed
//   w and y; the recorded rotations during QL
//   d, the couplings, their quaternions, the phases
//   the rotations' columns (bytes), the order of the eigenvalues (bytes)
struct SmallOffsets {
  int v, d, off, e4, phi, idx, perm, total;
};
__host__ __device__ inline SmallOffsets small_offsets(int n) {
  SmallOffsets o;
  o.v = 4 * n * (n | 1);
  o.d = o.v + 8 * n;
  o.off = o.d + n;
  o.e4 = o.off + n;
  o.phi = o.e4 + 4 * n;
  o.idx = o.phi + 4 * n;
  o.perm = o.idx + (4 * n + 7) / 8;
  o.total = (o.perm + (n + 7) / 8 + 1) & ~1;
  return o;
}

__device__ __forceinline__ int exponent_of(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// the range of recip_sqrt
__device__ __forceinline__ bool mid_range(double q) {
  const int e = exponent_of(q);
  return e > 123 && e < 1923;
}

// |off[k]| negligible beside |d[k]| + |d[k + 1]|; the exponents settle most cases
__device__ __forceinline__ bool small_coupling(const double* d, const double* off, int k) {
  const int e = exponent_of(off[k]), e0 = exponent_of(d[k]), e1 = exponent_of(d[k + 1]);
  if (e > 30 && e + 51 >= (e0 > e1 ? e0 : e1)) return false;
  const double o = fabs(off[k]);
  return o <= 1.1102230246251565e-16 * (fabs(d[k]) + fabs(d[k + 1])) || o < 1e-300;
}

// the smallest power of two >= v (v in 1 .. 32)
__device__ __forceinline__ int lanes_for(int v) { return v <= 1 ? 1 : 1 << (32 - __clz(v - 1)); }

__device__ __forceinline__ Q4<double> q_of(const double2* a, const double2* b, int i) {
  const double2 x = a[i], y = b[i];
  return Q4<double>{x.x, x.y, y.x, y.y};
}

// Load [A; B] (lower triangles) and reduce it to tridiagonal form; the reflectors go
// to the columns of the matrix in global memory. Returns the scale: the matrix is
// brought to largest entry in [1, 2) (subnormal numbers to 2^-52 and more), so no sum
// of squares needs its own.
__device__ double small_reduce(double2* A, double2* B, int64_t gld, int n, double* s, const SmallOffsets& o, int lane) {
  const int ld = n | 1;
  double2* ma = reinterpret_cast<double2*>(s);
  double2* mb = ma + n * ld;
  double2* wa = reinterpret_cast<double2*>(s + o.v);
  double2 *wb = wa + n, *ya = wb + n, *yb = ya + n;
  double *d = s + o.d, *e4 = s + o.e4;
  unsigned long long top = 0;
  for (int c = 0; c < n; ++c) {
    if (lane >= c && lane < n) {
      double2 a = A[lane + c * gld], b = B[lane + c * gld];
      if (lane == c) { a.y = 0.0; b = make_double2(0.0, 0.0); }
      ma[c * ld + lane] = a;
      mb[c * ld + lane] = b;
      ma[lane * ld + c] = cconj(a);
      mb[lane * ld + c] = lane == c ? b : cneg(b);
      const unsigned long long u = absmax_bits(a), v = absmax_bits(b);
      const unsigned long long t = u > v ? u : v;
      top = t > top ? t : top;
    }
  }
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, top, k);
    top = t > top ? t : top;
  }
  int ex = (int)(top >> 52);
  const bool finite = ex < 2047;
  // a zero matrix stays as it is; one of subnormal numbers comes as near as 2^1022 takes it
  ex = top == 0ull ? 1023 : (ex < 1 ? 1 : (ex > 2045 ? 2045 : ex));
  // (a matrix that holds an Inf or a NaN becomes NaN as a whole)
  const double scale = __hiloint2double(ex << 20, 0);
  const double inv = finite ? __hiloint2double((2046 - ex) << 20, 0) : __longlong_as_double(0x7ff8000000000000ll);
  __syncwarp();
  for (int t = lane; t < n * ld; t += 32) {
    const double2 a = ma[t], b = mb[t];
    ma[t] = cscale(a, inv);
    mb[t] = cscale(b, inv);
  }
  __syncwarp();
  for (int j = 0; j < n; ++j) {
    const int L = n - 1 - j, r0 = j + 1;
    if (lane == 0) d[j] = ma[j * ld + j].x;
    if (L < 1) break;
    Q4<double> x = q_zero<double>();
    if (lane < L) x = q_of(ma + j * ld + r0, mb + j * ld + r0, lane);
    if (L == 1) {  // one row left: the entry itself is the coupling
      if (lane == 0) {
        e4[4 * j] = x.ax; e4[4 * j + 1] = x.ay; e4[4 * j + 2] = x.bx; e4[4 * j + 3] = x.by;
        A[r0 + j * gld] = make_double2(0.0, 0.0);
        B[r0 + j * gld] = make_double2(0.0, 0.0);
      }
      continue;
    }
    const double x2 = fma(x.ax, x.ax, x.ay * x.ay) + fma(x.bx, x.bx, x.by * x.by);
    const int LP = lanes_for(L);
    double ss = x2;
    for (int k = LP >> 1; k > 0; k >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, k);
    ss = __shfl_sync(0xffffffffu, ss, 0);
    const double q2 = __shfl_sync(0xffffffffu, x2, 0);
    // the scalars of zq_resident.cu: with g = |x||x_1| and t = |x|/|x_1|, f = 1 / sqrt(ss + g),
    // the head of w is f (1 + t) x_1 and the coupling -t x_1; columns below 1e-75 of
    // the matrix are left as they are
    double f = 0.0;
    Q4<double> w = q_zero<double>(), e = w;
    if (!(ss < 1e-150)) {
      const double g2 = ss * q2;
      if (g2 > 1e-300) {
        const double rg = rsqrt(g2), t = ss * rg;
        f = rsqrt(fma(g2, rg, ss));
        const double h = lane == 0 ? fma(f, t, f) : f;
        w = Q4<double>{x.ax * h, x.ay * h, x.bx * h, x.by * h};
        e = Q4<double>{-t * x.ax, -t * x.ay, -t * x.bx, -t * x.by};
      } else {  // |x_1| too small to matter: the head is 1
        f = rsqrt(ss);
        w = lane == 0 ? Q4<double>{1.0, 0.0, 0.0, 0.0} : Q4<double>{x.ax * f, x.ay * f, x.bx * f, x.by * f};
        e = Q4<double>{-ss * f, 0.0, 0.0, 0.0};
      }
    }
    if (lane == 0) { e4[4 * j] = e.ax; e4[4 * j + 1] = e.ay; e4[4 * j + 2] = e.bx; e4[4 * j + 3] = e.by; }
    if (lane < L) {
      wa[lane] = make_double2(w.ax, w.ay);
      wb[lane] = make_double2(w.bx, w.by);
      A[r0 + lane + j * gld] = wa[lane];
      B[r0 + lane + j * gld] = wb[lane];
    }
    __syncwarp();
    if (f == 0.0) continue;
    // g = H w: LP lanes per group, a row each; the groups share the columns
    const int row = lane & (LP - 1), P = 32 / LP, rr = row < L ? row : L - 1;
    double g[4] = {0.0, 0.0, 0.0, 0.0};
    {
      const double2 *pa = ma + r0 * ld + r0 + rr, *pb = mb + r0 * ld + r0 + rr;
#pragma unroll 2
      for (int c = lane / LP; c < L; c += P) row_prod(g, q_of(pa, pb, c * ld), q_of(wa, wb, c));
    }
    for (int k = LP; k < 32; k <<= 1) {
#pragma unroll
      for (int u = 0; u < 4; ++u) g[u] += __shfl_xor_sync(0xffffffffu, g[u], k);
    }
    double cp = 0.0;
    const Q4<double> wr = q_of(wa, wb, rr);
    if (row < L) cp = fma(wr.ax, g[0], wr.ay * g[1]) + fma(wr.bx, g[2], wr.by * g[3]);
    for (int k = LP >> 1; k > 0; k >>= 1) cp += __shfl_xor_sync(0xffffffffu, cp, k);
    const double hc = -0.5 * cp;
    if (lane < L) {
      ya[lane] = make_double2(fma(hc, wr.ax, g[0]), fma(hc, wr.ay, g[1]));
      yb[lane] = make_double2(fma(hc, wr.bx, g[2]), fma(hc, wr.by, g[3]));
    }
    __syncwarp();
    // M -= w y^H + y w^H, a lane per entry of the lower triangle: column p (L - p
    // entries) and column L - 1 - p (p + 1 entries) make one run of L + 1
    const int items = (L + 1) * ((L + 1) / 2);
    const float rl = 1.0f / (float)(L + 1);
    for (int t = lane; t < items; t += 32) {
      int p = (int)(((float)t + 0.5f) * rl), q = t - p * (L + 1);
      int c = p, r = p + q;
      if (q >= L - p) {
        c = L - 1 - p;
        r = c + q - (L - p);
        if (c == p) continue;  // the middle column of an odd L stands alone
      }
      const Q4<double> u = rank2(q_of(wa, wb, r), q_of(ya, yb, r), q_of(wa, wb, c), q_of(ya, yb, c));
      const int lo = (r0 + c) * ld + r0 + r, up = (r0 + r) * ld + r0 + c;
      double2 a = ma[lo], b = mb[lo];
      a.x -= u.ax; a.y -= u.ay; b.x -= u.bx; b.y -= u.by;
      if (r == c) { a.y = 0.0; b = make_double2(0.0, 0.0); }
      ma[lo] = a;
      mb[lo] = b;
      if (r != c) { ma[up] = cconj(a); mb[up] = cneg(b); }
    }
    __syncwarp();
  }
  return scale;
}

// Moduli and unit phases of the couplings (one lane)
__device__ void small_phases(int n, double* s, const SmallOffsets& o) {
  const double* e4 = s + o.e4;
  double *off = s + o.off, *phi = s + o.phi;
  Q4<double> f{1.0, 0.0, 0.0, 0.0};
  for (int k = 0;; ++k) {
    phi[4 * k] = f.ax; phi[4 * k + 1] = f.ay; phi[4 * k + 2] = f.bx; phi[4 * k + 3] = f.by;
    if (k + 1 >= n) break;
    const Q4<double> e{e4[4 * k], e4[4 * k + 1], e4[4 * k + 2], e4[4 * k + 3]};
    const double q = fma(e.ax, e.ax, e.ay * e.ay) + fma(e.bx, e.bx, e.by * e.by);
    if (q <= 1e-280) {
      off[k] = 0.0;
      f = Q4<double>{1.0, 0.0, 0.0, 0.0};
      continue;
    }
    off[k] = sqrt(q);
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    row_prod(v, e, f);
    const double r = rsqrt(fma(v[0], v[0], v[1] * v[1]) + fma(v[2], v[2], v[3] * v[3]));
    f = Q4<double>{v[0] * r, v[1] * r, v[2] * r, v[3] * r};
  }
  off[n - 1] = 0.0;
}

struct QlState { int l, iter, bad; };

// Implicit QL sweeps with Wilkinson shifts on (d, off) by one lane, until the
// rotation buffer might not hold the next sweep or the matrix is done (q.l == n).
// Returns the number of rotations recorded: (c, s) and the column idx they act on
// together with idx + 1.
__device__ int small_sweeps(int n, double* s, const SmallOffsets& o, QlState& q) {
  double *d = s + o.d, *off = s + o.off;
  double2* rot = reinterpret_cast<double2*>(s + o.v);
  unsigned char* idx = reinterpret_cast<unsigned char*>(s + o.idx);
  const int cap = 4 * n;
  int cnt = 0;
  while (q.l < n) {
    const int l = q.l;
    int m = l;
    while (m < n - 1 && !small_coupling(d, off, m)) ++m;
    if (m == l || q.iter >= 60) {
      if (m != l) ++q.bad;
      ++q.l;
      q.iter = 0;
      continue;
    }
    if (cnt + m - l > cap) break;
    ++q.iter;
    const double el = off[l], dl = d[l];
    double g = (d[l + 1] - dl) / (2.0 * el);
    const double ag = fabs(g), r1 = ag < 1e140 ? sqrt(fma(g, g, 1.0)) : ag;
    double dn = d[m];
    g = dn - dl + el / (g + copysign(r1, g));
    double sn = 1.0, c = 1.0, p = 0.0;
    bool early = false;
    for (int i = m - 1; i >= l; --i) {
      const double ei = off[i], di = d[i];
      const double ff = sn * ei, bb = c * ei, qq = fma(ff, ff, g * g);
      double r;
      if (mid_range(qq)) {
        const double y = recip_sqrt(qq);
        r = qq * y; sn = ff * y; c = g * y;
      } else {
        r = hypot(ff, g);
        if (r == 0.0) { off[i + 1] = 0.0; d[i + 1] = dn - p; off[m] = 0.0; early = true; break; }
        sn = ff / r; c = g / r;
      }
      off[i + 1] = r;
      g = dn - p;
      const double t = fma(di - g, sn, 2.0 * (c * bb));
      p = sn * t;
      d[i + 1] = g + p;
      g = fma(c, t, -bb);
      dn = di;
      rot[cnt] = make_double2(c, sn);
      idx[cnt] = (unsigned char)i;
      ++cnt;
    }
    if (!early) { d[l] = dn - p; off[l] = g; off[m] = 0.0; }
  }
  return cnt;
}

// X = Phi Z in ascending order, the reflectors applied backwards, the result and its
// conjugate partner stored
__device__ void small_back(double2* A, double2* B, int64_t gld, double* eig, int n, double scale, double* s,
                           const SmallOffsets& o, int lane) {
  const int ld = n | 1;
  double2* xa = reinterpret_cast<double2*>(s);
  double2* xb = xa + n * ld;
  const double* z = s + 3 * n * ld;
  double2* wa = reinterpret_cast<double2*>(s + o.v);
  double2* wb = wa + n;
  const double *d = s + o.d, *phi = s + o.phi;
  unsigned char* perm = reinterpret_cast<unsigned char*>(s + o.perm);
  if (lane < n) perm[lane] = (unsigned char)lane;
  __syncwarp();
  if (lane < n) {
    const double v = d[lane];
    int rank = 0;
    for (int q = 0; q < n; ++q) rank += (d[q] < v) || (d[q] == v && q < lane);
    perm[rank] = (unsigned char)lane;
  }
  __syncwarp();
  if (lane < n) eig[lane] = d[perm[lane]] * scale;
  // row r of X ends below row r + 1 of Z, so the rows may be formed in place in order
  const int from = lane < n ? perm[lane] : 0;
  for (int r = 0; r < n; ++r) {
    const double v = z[r * ld + from];
    __syncwarp();
    if (lane < n) {
      xa[r * ld + lane] = make_double2(phi[4 * r] * v, phi[4 * r + 1] * v);
      xb[r * ld + lane] = make_double2(phi[4 * r + 2] * v, phi[4 * r + 3] * v);
    }
    __syncwarp();
  }
  // x <- x - w <w, x> - w' [w, x], w' = (-conj(wb), conj(wa)): NP lanes per group, a
  // column each; the groups share the rows
  const int NP = lanes_for(n), P = 32 / NP, col = lane & (NP - 1), cc = col < n ? col : n - 1, grp = lane / NP;
  double2 na = make_double2(0.0, 0.0), nb = na;
  auto fetch = [&](int j) {
    if (j >= 0 && lane < n - 1 - j) { na = A[j + 1 + lane + j * gld]; nb = B[j + 1 + lane + j * gld]; }
  };
  fetch(n - 3);
  for (int j = n - 3; j >= 0; --j) {
    const int L = n - 1 - j;
    if (lane < L) { wa[lane] = na; wb[lane] = nb; }
    __syncwarp();
    fetch(j - 1);
    double2 c1 = make_double2(0.0, 0.0), c2 = c1;
    double2 *pa = xa + (j + 1) * ld + cc, *pb = xb + (j + 1) * ld + cc;
#pragma unroll 2
    for (int i = grp; i < L; i += P) {
      const double2 a = wa[i], b = wb[i], va = pa[i * ld], vb = pb[i * ld];
      cfmac(c1, a, va); cfmac(c1, b, vb);
      cfma(c2, a, vb); cfma(c2, cneg(b), va);
    }
    for (int k = NP; k < 32; k <<= 1) {
      c1.x += __shfl_xor_sync(0xffffffffu, c1.x, k); c1.y += __shfl_xor_sync(0xffffffffu, c1.y, k);
      c2.x += __shfl_xor_sync(0xffffffffu, c2.x, k); c2.y += __shfl_xor_sync(0xffffffffu, c2.y, k);
    }
    c1 = cneg(c1);
    c2 = cneg(c2);
#pragma unroll 2
    for (int i = grp; i < L; i += P) {
      const double2 a = wa[i], b = wb[i];
      double2 va = pa[i * ld], vb = pb[i * ld];
      cfma(va, a, c1); cfmac(va, cneg(b), c2);
      cfma(vb, b, c1); cfmac(vb, a, c2);
      if (col < n) { pa[i * ld] = va; pb[i * ld] = vb; }
    }
    __syncwarp();
  }
  for (int c = 0; c < n; ++c) {
    if (lane < n) {
      const double2 u = xa[lane * ld + c], v = xb[lane * ld + c];
      A[lane + c * gld] = u;
      B[lane + c * gld] = v;
      A[lane + (n + c) * gld] = make_double2(-v.x, v.y);
      B[lane + (n + c) * gld] = make_double2(u.x, -u.y);
    }
  }
  __syncwarp();
}

struct SmallArgs {
  const BatchTask* tasks;
  int count;
  int* counter;  // work counter (zeroed before the launch)
  double2* D;
  double* eig;
  int* info;     // per task: 0 ok, > 0 QL non-convergence
  SmallOffsets o;
  int nmax;
  BatchTask one;  // the only task where tasks is null (no counter, no info)
};

__global__ void __launch_bounds__(SMALL_WARPS * 32, 2) k_small(SmallArgs a) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_first;
  __shared__ int s_n[SMALL_WARPS], s_cnt[SMALL_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  // CTAs that share an SM run their chains in different quadrants
  const int chain = (int)blockIdx.x % warps;
  double* s = smem + warp * a.o.total;
  int pass = 0;
  for (;;) {
    if (threadIdx.x == 0 && a.tasks) s_first = atomicAdd(a.counter, warps);
    if (threadIdx.x == 0 && !a.tasks) s_first = pass++;
    __syncthreads();
    const int t = s_first + warp;
    if (s_first >= a.count) return;
    BatchTask tk{};
    if (t < a.count) tk = a.tasks ? a.tasks[t] : a.one;
    int n = tk.n;
    if (n > a.nmax) {  // not within the launch's limit: reported, not solved
      if (lane == 0 && a.info) a.info[tk.out_slot] = -1;
      n = 0;
    }
    if (lane == 0) s_n[warp] = n;
    const int64_t gld = tk.ld;
    double2* A = tk.Dp ? tk.Dp : a.D + tk.off;
    double2* B = A + n;
    double scale = 1.0;
    if (n > 0) {
      scale = small_reduce(A, B, gld, n, s, a.o, lane);
      __syncwarp();
      double* z = s + 3 * n * (n | 1);
      for (int r = 0; r < n; ++r)
        if (lane < n) z[r * (n | 1) + lane] = lane == r ? 1.0 : 0.0;
    }
    __syncthreads();
    QlState q{0, 0, 0};
    double* sl = smem + lane * a.o.total;  // the chain's matrix of this lane
    const bool own = warp == chain && lane < warps;
    const int nl = own ? s_n[lane] : 0;
    if (nl > 0) small_phases(nl, sl, a.o);
    __syncwarp();
    for (;;) {
      if (own) s_cnt[lane] = nl > 0 ? small_sweeps(nl, sl, a.o, q) : 0;
      __syncwarp();
      const int more = __syncthreads_or(own && q.l < nl);
      if (lane < n) {  // this matrix's rotations, a row of Z per lane
        const double2* rot = reinterpret_cast<const double2*>(s + a.o.v);
        const unsigned char* idx = reinterpret_cast<const unsigned char*>(s + a.o.idx);
        double* zr = s + 3 * n * (n | 1) + lane * (n | 1);
        const int cnt = s_cnt[warp];
        int cur = -1;
        double carry = 0.0;
        for (int k = 0; k < cnt; ++k) {
          const int i = idx[k];
          const double2 cs = rot[k];
          if (i + 1 != cur) {  // the next sweep starts: column i + 1 anew
            if (cur >= 0) zr[cur] = carry;
            carry = zr[i + 1];
          }
          const double v = zr[i];
          zr[i + 1] = fma(cs.y, v, cs.x * carry);
          carry = fma(cs.x, v, -(cs.y * carry));
          cur = i;
        }
        if (cur >= 0) zr[cur] = carry;
      }
      if (!more) break;
      __syncthreads();  // the rotations are read
    }
    __syncwarp();
    if (own && nl > 0 && a.info) a.info[a.tasks[s_first + lane].out_slot] = q.bad;
    if (n > 0) small_back(A, B, gld, tk.Ep ? tk.Ep : a.eig + tk.eoff, n, scale, s, a.o, lane);
    __syncthreads();  // s_first, s_n and the matrices are free
  }
}

}  // namespace

int small_solve(double2* D, int64_t ld, int n, double* eig, cudaStream_t st) {
  SmallArgs a{};
  a.count = 1;
  a.o = small_offsets(n);
  a.nmax = n;
  a.one.Dp = D; a.one.Ep = eig; a.one.n = n; a.one.ld = (int)ld;
  k_small<<<1, 32, sizeof(double) * (size_t)a.o.total, st>>>(a);
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int small_launch(const BatchTask* tasks, int count, int nmax, int* dev_counter, double2* D, double* eig, int ctas,
                 int* dev_info, cudaStream_t st) {
  if (count <= 0) return ZQ_OK;
  if (nmax < 1 || nmax > SMALL_MAX) { set_error_message("batch: order outside the warp solver's range"); return ZQ_ERR_ARG; }
  int dev = 0, sms = 0, optin = 0;
  ZQ_CUDA(cudaGetDevice(&dev));
  ZQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ZQ_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  SmallArgs a{};
  a.tasks = tasks;
  a.count = count;
  a.counter = dev_counter;
  a.D = D;
  a.eig = eig;
  a.info = dev_info;
  a.o = small_offsets(nmax);
  a.nmax = nmax;
  // CTAs per SM as asked for (at least two: a CTA's chain leaves the other quadrants to
  // its neighbour), as many matrices each as then fit, fewer if the batch has not enough
  const int per_sm = ctas / sms < 2 ? 2 : ctas / sms;
  const size_t bytes = sizeof(double) * (size_t)a.o.total;
  int warps = (int)(((size_t)optin / per_sm - 2048) / bytes);
  const int spread = ceil_div(count, per_sm * sms);
  if (warps > spread) warps = spread;
  if (warps > SMALL_WARPS) warps = SMALL_WARPS;
  if (warps < 1) warps = 1;
  int grid = ceil_div(count, warps);
  if (grid > per_sm * sms) grid = per_sm * sms;
  ZQ_CUDA(cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 2048));
  ZQ_CUDA(cudaMemsetAsync(dev_counter, 0, sizeof(int), st));
  k_small<<<grid, warps * 32, bytes * warps, st>>>(a);
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace zq
