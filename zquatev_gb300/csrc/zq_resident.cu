// Quaternion tridiagonalisation with the matrix resident in shared memory.
//
// Same reduction and outputs as zq_tridiag.cu (one quaternion reflector per
// column; reference blocked.cc:45-546, unblocked.cc:44-131): d, the quaternion
// subdiagonal e, tau, and w_j stored in column j below the diagonal. Here the
// lower triangles of A and B are loaded once, as T x T tiles dealt round robin
// over the shared memories of a group of G co-resident CTAs, and stay there:
// per column every tile takes the previous column's rank-2 update and the
// mat-vec with the current reflector in one sweep, and only vectors travel
// between the CTAs (through L2), with two group barriers per column:
//
//   sweep j    tiles -= w_{j-1} y_{j-1}^H + y_{j-1} w_{j-1}^H (structured), then the
//              tile's products with w_j and their part of c = w_j^H H w_j; column
//              j + 1 is published
//      -- barrier --
//   rows       g = H w_j from the tile partials of the CTA's share of the rows,
//              y_j = g - (c/2) w_j, and column j + 1 brought up to date there,
//              with its norm partials (every CTA also sums row j + 1 for itself)
//      -- barrier --
//              every CTA forms reflector j + 1 from the norm partials
//
// Why: the per-column kernels of zq_tridiag.cu cost ~22 us (FP32) to ~75 us
// (FP64) per column in launches, memory round trips and FP64 work on few SMs,
// at orders where the arithmetic takes a few; and GB300's FP64 pipe (2 FMA per
// clock per SM) makes the split of the FP64 work over all SMs matter more than
// operand reuse, hence small tiles. Reduction before and after: FP64 n = 384
// 29 -> 4.9 ms, n = 750 60 -> 18 ms (7.2 ms of FP64 pipe time); FP32 n = 1023
// 23.5 -> 8.4 ms. What remains per column (FP32, n = 750, cycles): reflector
// scalars 1400, vectors 1250, sweep 2400, c 1000, rows 2450, column 860, norms
// 780, barriers 3100 + 2500 (2540 in isolation): chains of L2 round trips and
// dependent instructions.
//
// Tile work: one warp per tile, lane (tr, tc) = (lane & 7, lane >> 3) owns
// rows tr + 8 i and columns tc + 4 q of the tile, stored so that a lane only
// touches its own 16-byte-aligned slots (no bank conflicts, no barriers around
// the tiles). The lanes' row and column products meet by a halving exchange
// (each step every lane keeps half of its values), so the sums cost about one
// add per value. A diagonal tile holds both triangles and forms row products
// only.
//
// Tiles are dealt in the order of their columns from the last one back, so
// that the live tiles of every stage are spread evenly.
//
// A group of one CTA per SM is one cooperative launch and meets at a counter; that
// wait is bounded (when it runs out, the abort flag and the caller's error flag are
// raised, NaN is left in d, and all CTAs return). A cluster meets at its hardware
// barrier, which has no limit and needs none: its CTAs are scheduled together and
// all pass the same barriers.
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_quat.cuh"
#include "zq_resident.h"

#include <algorithm>
#include <atomic>
#include <functional>
#include <queue>
#include <vector>

namespace zq {
namespace {

constexpr int RT_THREADS = 256;
constexpr int RT_WARPS = RT_THREADS / 32;
constexpr int RT_CLUSTER = 16;  // largest cluster
constexpr int RT_SMEM_MAX = 227 * 1024 - 3 * 1024;  // dynamic shared memory per CTA (static part below 3 KB)

// a lane's tile slot e: FP32 one 16-byte slot, FP64 two 16-byte planes
template <int EL> __device__ __forceinline__ Q4<float> t_load(const float* t, int e, int lane) {
  const float4 v = reinterpret_cast<const float4*>(t)[e * 32 + lane];
  return Q4<float>{v.x, v.y, v.z, v.w};
}
template <int EL> __device__ __forceinline__ void t_store(float* t, int e, int lane, const Q4<float>& q) {
  reinterpret_cast<float4*>(t)[e * 32 + lane] = make_float4(q.ax, q.ay, q.bx, q.by);
}
template <int EL> __device__ __forceinline__ Q4<double> t_load(const double* t, int e, int lane) {
  const double2 u = reinterpret_cast<const double2*>(t)[e * 32 + lane];
  const double2 v = reinterpret_cast<const double2*>(t)[(EL + e) * 32 + lane];
  return Q4<double>{u.x, u.y, v.x, v.y};
}
template <int EL> __device__ __forceinline__ void t_store(double* t, int e, int lane, const Q4<double>& q) {
  reinterpret_cast<double2*>(t)[e * 32 + lane] = make_double2(q.ax, q.ay);
  reinterpret_cast<double2*>(t)[(EL + e) * 32 + lane] = make_double2(q.bx, q.by);
}

// Signs (bit q set: minus) of the four products that make component k of
//   the rank-2 term     sum_q w_r[k^q] y_c[q]   + + + + | + - - + | + + - - | + - + -
//   a row product       sum_q m[k^q] w_c[q]     + - - - | + + + - | + - + + | + + - +
//   a column product    sum_q m[k^q] w_r[q]     + + + + | - + - + | - + + - | - - + +
__device__ __forceinline__ unsigned quat_signs(unsigned table, int k) { return (table >> (4 * k)) & 15u; }
constexpr unsigned SIGNS_RANK2 = 0xAC60u, SIGNS_ROW = 0x428Eu, SIGNS_COL = 0x3950u;
__device__ __forceinline__ double flip(double v, unsigned neg) {
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)(neg & 1u) << 63));
}

// tile t in dealing order: column blocks from the last one back
__device__ __forceinline__ void rt_tile(int t, int nt, int& I, int& J) {
  int a, b;
  tri_tile(t, a, b);
  J = nt - 1 - a;
  I = J + b;
}

// Barrier of one group (bounded). ctr only grows; `target` is this CTA's count.
__device__ __forceinline__ bool group_barrier(unsigned* ctr, unsigned& target, int G, unsigned* abt, int* err,
                                              long long limit, int* s_ok) {
  __syncthreads();
  if (G > 1) {
    if (threadIdx.x == 0) {
      target += (unsigned)G;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      unsigned v;
      int ok = 1, spins = 0;
      const int every = limit < 100000 ? 0 : 63;  // polls between looks at the clock, less one
      const long long t0 = clock64();
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if ((int)(v - target) >= 0) break;
        if ((++spins & every) == 0) {
          if (*reinterpret_cast<volatile unsigned*>(abt)) { ok = 0; break; }
          if (clock64() - t0 > limit) {
            atomicExch(abt, 1u);
            if (err) atomicExch(err, 1);
            ok = 0;
            break;
          }
        }
      }
      *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
  }
  return true;
}

__device__ __forceinline__ void cluster_barrier() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ double pow2_biased(int be) {
  return be < 1 ? 0.0 : __longlong_as_double((long long)be << 52);
}

// Sums of the vector phases. FP64 data: doubles. FP32 data: unevaluated pairs of
// floats (hi + lo, ~48 bits; Dekker/Knuth two-sums and FMA products): the FP64 pipe
// takes ~75 cycles per dependent instruction here, a pair's sum ~30. What follows from
// them is rounded to 24 bits (f, h, c / 2) or describes data that are (e); against sums
// in double the first correction of the refinement is the same (its maximum, 33 random
// matrices of n = 60 to 2500: geometric mean of the ratios 1.00).
struct Pair { float hi, lo; };
__device__ __forceinline__ Pair sum2(Pair a, Pair b) {
  const float s = a.hi + b.hi, t = s - a.hi;
  const float e = ((a.hi - (s - t)) + (b.hi - t)) + (a.lo + b.lo);
  const float h = s + e;
  return Pair{h, e - (h - s)};
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  const float p = a.hi * b.hi;
  const float e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p)));
  const float h = p + e;
  return Pair{h, e - (h - p)};
}
// 1 / sqrt(a) by one Newton step from the approximate instruction
__device__ __forceinline__ Pair rsqrt2(Pair a) {
  const float y = rsqrtf(a.hi), p = y * y;
  const Pair u = mul2(a, Pair{p, fmaf(y, y, -p)});
  const float d = (1.f - u.hi) - u.lo;
  return Pair{y, 0.5f * y * d};
}
template <typename R> struct AccOf { using type = double; };
template <> struct AccOf<float> { using type = Pair; };
template <typename R> using Acc = typename AccOf<R>::type;
__device__ __forceinline__ double acc_add(double a, double b) { return a + b; }
__device__ __forceinline__ Pair acc_add(Pair a, Pair b) { return sum2(a, b); }
__device__ __forceinline__ double acc_shfl(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ Pair acc_shfl(Pair v, int o) {
  return Pair{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}
__device__ __forceinline__ void acc_square(double& s, double x) { s = fma(x, x, s); }
__device__ __forceinline__ void acc_square(Pair& s, float x) {
  const float p = x * x;
  s = sum2(s, Pair{p, fmaf(x, x, -p)});
}
__device__ __forceinline__ double acc_value(double x) { return x; }
__device__ __forceinline__ Pair acc_value(float x) { return Pair{x, 0.f}; }
__device__ __forceinline__ double acc_double(double v) { return v; }
__device__ __forceinline__ double acc_double(Pair v) { return (double)v.hi + (double)v.lo; }
__device__ __forceinline__ double acc_half(double v) { return 0.5 * v; }
__device__ __forceinline__ float acc_half(Pair v) { return 0.5f * (v.hi + v.lo); }
__device__ __forceinline__ void acc_store(double* p, double v) { *p = v; }
__device__ __forceinline__ void acc_store(double* p, Pair v) { *reinterpret_cast<float2*>(p) = make_float2(v.hi, v.lo); }
__device__ __forceinline__ void acc_load(const double* p, double& v) { v = __ldcg(p); }
__device__ __forceinline__ void acc_load(const double* p, Pair& v) {
  const float2 t = __ldcg(reinterpret_cast<const float2*>(p));
  v = Pair{t.x, t.y};
}
template <int FROM, int TO, typename V> __device__ __forceinline__ V acc_lanes(V v) {
#pragma unroll
  for (int o = FROM; o >= TO; o >>= 1) v = acc_add(v, acc_shfl(v, o));
  return v;
}
// Sum of `count` accumulators written by other CTAs, by one warp; every lane gets it.
template <typename R>
__device__ __forceinline__ Acc<R> warp_gather(const double* p, int count, int lane) {
  Acc<R> s{};
  for (int i = lane; i < count; i += 128) {  // four loads in flight
    Acc<R> v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = Acc<R>{};
      if (i + 32 * u < count) acc_load(p + i + 32 * u, v[u]);
    }
    s = acc_add(s, acc_add(acc_add(v[0], v[1]), acc_add(v[2], v[3])));
  }
  return acc_lanes<16, 1>(s);
}

// The reflector's scalars from ss = |x|^2 and q2 = |x_1|^2 (in units of the scaled
// matrix): g = sqrt(ss q2) = |x||x_1|, s = |x| / |x_1| = ss / g, f = 1 / sqrt(ss + g),
// h = f (1 + s). False: |x_1| is too small beside |x| to matter (below 1e-75, FP32
// 1e-15), the head is taken as 1 and f = 1 / |x|.
// Columns below tiny_column (|x| under 1e-75 of the matrix, FP32 1e-14) are left as
// they are (f = 0, e = 0), so no product here leaves the range of normal numbers.
__device__ __forceinline__ bool tiny_column(double ss) { return ss < 1e-150; }
__device__ __forceinline__ bool tiny_column(Pair ss) { return ss.hi < 1e-28f; }
__device__ __forceinline__ bool reflector_scalars(double ss, double q2, double& f, double& h, double& s) {
  const double t = ss * q2;
  if (!(t > 1e-300)) { f = rsqrt(ss); return false; }
  const double rg = rsqrt(t);
  s = ss * rg;
  f = rsqrt(fma(t, rg, ss));
  h = fma(f, s, f);
  return true;
}
__device__ __forceinline__ bool reflector_scalars(Pair ss, Pair q2, float& f, float& h, Pair& s) {
  // an even power of two brings ss into [1, 4): q2 <= ss keeps its bits
  const int e = ((int)(__float_as_uint(ss.hi) >> 23) - 127) & ~1;
  const float sc = __uint_as_float((unsigned)(127 - e) << 23), sr = __uint_as_float((unsigned)(127 - e / 2) << 23);
  const Pair a{ss.hi * sc, ss.lo * sc};
  const Pair t = mul2(a, Pair{q2.hi * sc, q2.lo * sc});
  if (!(t.hi > 1e-30f)) {
    const Pair r = rsqrt2(a);
    f = (r.hi + r.lo) * sr;
    return false;
  }
  const Pair rg = rsqrt2(t);
  s = mul2(a, rg);
  const Pair r = rsqrt2(sum2(mul2(t, rg), a));
  const Pair hh = sum2(mul2(r, s), r);
  f = (r.hi + r.lo) * sr;
  h = (hh.hi + hh.lo) * sr;
  return true;
}
__device__ __forceinline__ unsigned mag_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned long long mag_bits(double v) { return abs_bits(v); }
__device__ __forceinline__ double mag_value(unsigned b) { return (double)__uint_as_float(b); }
__device__ __forceinline__ double mag_value(unsigned long long b) { return bits_to_double(b); }

// CTAs that own rows in the vector phases: enough to spread the sums, few
// enough that one warp gathers their partials in one or two steps
template <typename R> __host__ __device__ __forceinline__ int row_ctas(int G) {
  const int most = sizeof(R) == 8 ? 96 : 32;
  return G < most ? G : most;
}

// One matrix reduced by the group (CL: the group is one cluster). Returns
// false when a wait ran out.
//
// An FP64 instruction holds its SM quadrant's pipe for 64 cycles whatever the
// number of lanes, so the vector phases keep one real component per lane (the
// four lanes of a row exchange theirs by shuffles). The matrix is scaled by a
// power of two once (largest entry in [1, 2)), so no sum of squares needs a scale
// of its own; FP32 columns whose squares vanish are 1e-19 of the matrix.
//
// Between two barriers an exchanged array is written or read by other CTAs, never
// both: a CTA that runs ahead must not overwrite what another has yet to read. The
// phases and what they touch:
//   load     writes cpart (largest magnitudes)
//   column 0 reads cpart; writes x, npart, q2
//   sweep    reads x, y, npart, q2; writes col, part, cpart (parts of c)
//   rows     reads col, part, cpart, and x of the CTA's own rows; writes x, y, npart, q2
template <typename R, int T, int LPR, bool CL>
__device__ bool reduce_matrix(const TriTask<R>& tk, const TriGroup<R>& gr, int rank, int G, unsigned char* smem,
                              unsigned& target, int* err, long long limit) {
  constexpr int RR = T / 8, CC = T / 4, EL = RR * CC;  // rows, columns and entries per lane
  constexpr int NRV = RR * 4 / 4;                      // row sums a lane ends with (4 column lanes)
  constexpr int NCV = CC * 4 / 8;                      // column sums a lane ends with (8 row lanes)
  constexpr int TILE = T * T * 4;                      // reals per tile
  __shared__ R s_head[8];                              // f, f m (4)
  __shared__ double s_red[RT_WARPS];
  __shared__ double s_cw[RT_WARPS];                    // the warps' parts of c
  __shared__ R s_hc;                                   // c / 2
  __shared__ R s_team[2][4][32];                       // row sums of the warps that share a tile
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tr = lane & 7, tc = lane >> 3;
  const int n = tk.n, k0 = tk.k0, m = n - k0;
  const int64_t ld = tk.ld;
  cplx<R>* A = tk.M + k0 + (int64_t)k0 * ld;
  cplx<R>* B = A + n;
  const int nt = (m + T - 1) / T;
  const int ntiles = nt * (nt + 1) / 2;
  const int mine = ntiles > rank ? (ntiles - rank + G - 1) / G : 0;
  const int NR = row_ctas<R>(G);
  auto barrier = [&]() {
    if constexpr (CL) {
      cluster_barrier();
      return true;
    } else {
      return group_barrier(gr.counter, target, G, gr.abort, err, limit, &s_ok);
    }
  };

  // shared memory: tiles | w (previous, current) | y | own rows (w, g, x) | needed blocks
  R* tiles = reinterpret_cast<R*>(smem);
  const int cap = (ntiles + G - 1) / G;
  Q4<R>* wbuf[2];
  wbuf[0] = reinterpret_cast<Q4<R>*>(tiles + (size_t)cap * TILE);
  wbuf[1] = wbuf[0] + m;
  Q4<R>* ys = wbuf[1] + m;
  const int rmax = (m + NR - 1) / NR;
  R* own_w = reinterpret_cast<R*>(ys + m);
  R* own_g = own_w + 4 * rmax;          // and g at row j + 1 in the row after the CTA's
  R* own_x = own_g + 4 * (rmax + 1);
  unsigned char* need = reinterpret_cast<unsigned char*>(own_x + 4 * rmax);

  // load the tiles; clear the vectors; mark the row blocks this CTA's tiles touch
  for (int b = tid; b < nt; b += RT_THREADS) need[b] = 0;
  for (int r = tid; r < m; r += RT_THREADS) { wbuf[0][r] = q_zero<R>(); wbuf[1][r] = q_zero<R>(); ys[r] = q_zero<R>(); }
  __syncthreads();
  decltype(mag_bits(R(0))) mb = 0;
  for (int q = warp; q < mine; q += RT_WARPS) {
    int I, J;
    rt_tile(rank + q * G, nt, I, J);
    if (lane == 0) { need[I] = 1; need[J] = 1; }
    R* tl = tiles + (size_t)q * TILE;
#pragma unroll 4
    for (int e = 0; e < EL; ++e) {
      const int r = I * T + tr + 8 * (e % RR), c = J * T + tc + 4 * (e / RR);
      Q4<R> v = q_zero<R>();
      if (r < m && c < m) {
        const bool low = r >= c;
        const int64_t o = low ? r + (int64_t)c * ld : c + (int64_t)r * ld;
        const cplx<R> a = A[o], b = B[o];
        v = low ? Q4<R>{a.x, a.y, b.x, b.y} : Q4<R>{a.x, -a.y, -b.x, -b.y};
        if (r == c) { v.ay = 0; v.bx = 0; v.by = 0; }
        mb = max(mb, max(max(mag_bits(v.ax), mag_bits(v.ay)), max(mag_bits(v.bx), mag_bits(v.by))));
      }
      t_store<EL>(tl, e, lane, v);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
  if (lane == 0) s_red[warp] = mag_value(mb);
  __syncthreads();
  if (tid == 0) {
    unsigned long long b = 0;
    for (int q = 0; q < RT_WARPS; ++q) b = max(b, abs_bits(s_red[q]));
    gr.cpart[rank] = bits_to_double(b);
  }
  if (!barrier()) return false;
  double scale = 1.0;
  bool finite = true;
  {
    unsigned long long b = 0;
    for (int i = lane; i < G; i += 32) b = max(b, abs_bits(__ldcg(gr.cpart + i)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    const int be = (int)(b >> 52);
    finite = be < 2047;
    // FP32 data: the scale and its inverse stay normal numbers of R
    const int lim = sizeof(R) == 8 ? 1022 : 126;
    if (b != 0) scale = pow2_biased(be < 1023 - lim ? 1023 - lim : (be > 1023 + lim ? 1023 + lim : be));
  }
  // (a matrix that holds an Inf or a NaN becomes NaN as a whole: at the scale of its
  // largest entry its numbers would vanish and leave a finite result)
  const R inv = (R)(finite ? bits_to_double((2046ull << 52) - (unsigned long long)__double_as_longlong(scale))
                           : __longlong_as_double(0x7ff8000000000000ll));
  for (int q = warp; q < mine; q += RT_WARPS) {
    R* tl = tiles + (size_t)q * TILE;
#pragma unroll 4
    for (int e = 0; e < EL; ++e) {
      Q4<R> v = t_load<EL>(tl, e, lane);
      v.ax *= inv; v.ay *= inv; v.bx *= inv; v.by *= inv;
      t_store<EL>(tl, e, lane, v);
    }
  }
  // this CTA's rows: its share of [j, m) for the column j being formed
  int rows0 = 0, nrows = 0;
  auto partition = [&](int j) {
    const int per = (m - j + NR - 1) / NR;
    rows0 = j + rank * per;
    nrows = (rank >= NR || rows0 >= m) ? 0 : (rows0 + per < m ? per : m - rows0);
  };
  // |x|^2 of the own rows below the diagonal of column j (ss: a part per thread),
  // and |x_1|^2 for everybody (row j + 1; x: this thread's first component)
  auto publish_norms = [&](int j, R x, Acc<R> ss) {
    const int items = 4 * nrows;
    if (warp * 32 < items || warp == 0) ss = acc_lanes<16, 1>(ss);
    if (items > 32) {
      if (lane == 0) acc_store(s_red + warp, warp * 32 < items ? ss : Acc<R>{});
      __syncthreads();
      if (warp == 0) {
        ss = Acc<R>{};
        if (lane < RT_WARPS) {
          if constexpr (sizeof(R) == 8) ss = s_red[lane];
          else { const float2 t = reinterpret_cast<const float2*>(s_red)[lane]; ss = Pair{t.x, t.y}; }
        }
        ss = acc_lanes<RT_WARPS / 2, 1>(ss);
      }
    }
    if (tid == 0 && rank < NR) acc_store(gr.npart + rank, ss);
    const int i1 = j + 1 - rows0;  // row j + 1 among the own rows: the first or the second
    if (warp == 0 && i1 >= 0 && i1 < nrows) {
      Acc<R> q{};
      acc_square(q, x);
      q = acc_lanes<2, 1>(q);
      if (tid == 4 * i1) acc_store(gr.q2, q);
    }
  };
  // column 0 as it is
  partition(0);
  {
    Acc<R> ss{};
    R x0 = R(0);
    for (int idx = tid; idx < ((4 * nrows + 31) & ~31); idx += RT_THREADS) {
      R x = R(0);
      if (idx < 4 * nrows) {
        const int r = rows0 + (idx >> 2), k = idx & 3;
        const R* src = reinterpret_cast<const R*>((k < 2 ? A : B) + r);
        x = src[k & 1] * inv;
        if (r == 0) { if (k) x = R(0); else tk.d[k0] = (double)x * scale; }
        own_x[idx] = x;
        reinterpret_cast<R*>(gr.x)[4 * r + k] = x;
        if (r > 0) acc_square(ss, x);
      }
      if (idx == tid) x0 = x;
    }
    publish_norms(0, x0, ss);
  }
  if (!barrier()) return false;

  for (int j = 0; j + 1 < m; ++j) {
    Q4<R>* wp = wbuf[(j & 1) ^ 1];
    Q4<R>* wn = wbuf[j & 1];
    // ------------------------------------------------ reflector j
    const bool last = m - 1 - j < 2;  // one row left: the entry itself is e
    if (warp == 0) {
      const R x1 = __ldcg(reinterpret_cast<const R*>(gr.x + j + 1) + (lane & 3));
      Acc<R> q2;
      acc_load(gr.q2, q2);
      const Acc<R> ss = warp_gather<R>(gr.npart, NR, lane);
      R f = R(0), h = R(0);
      bool unit = false;  // the head is 1
      if (!last && !tiny_column(ss)) {
        Acc<R> s{};
        unit = !reflector_scalars(ss, q2, f, h, s);
      }
      if (lane < 4) {
        s_head[1 + lane] = unit ? (lane == 0 ? R(1) : R(0)) : x1 * h;
        if (lane == 0) { s_head[0] = f; s_head[5] = unit ? R(1) : R(0); }
      }
    }
    // w and y_{j-1} of the blocks this CTA's tiles touch: up to RPT rows per thread
    // are held until the reflector is known
    constexpr int RPT = 4;
    const int rfrom = j >= 2 ? j - 2 : 0;
    Q4<R> xr[RPT];
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      const int r = rfrom + tid + RT_THREADS * u;
      xr[u] = q_zero<R>();
      if (r >= m || !need[r / T]) continue;
      if (r > j) xr[u] = q_ldcg(gr.x + r);
      ys[r] = j > 0 && r >= j ? q_ldcg(gr.y + r) : q_zero<R>();
    }
    __syncthreads();
    const R f = s_head[0];
    const Q4<R> w1{s_head[1], s_head[2], s_head[3], s_head[4]};  // w at row j + 1
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      const int r = rfrom + tid + RT_THREADS * u;
      if (r >= m || !need[r / T]) continue;
      const Q4<R> x = xr[u];
      wn[r] = r == j + 1 ? w1 : Q4<R>{x.ax * f, x.ay * f, x.bx * f, x.by * f};
    }
    for (int r = rfrom + tid + RT_THREADS * RPT; r < m; r += RT_THREADS) {
      if (!need[r / T]) continue;
      Q4<R> x = q_zero<R>();
      if (r > j) x = q_ldcg(gr.x + r);
      wn[r] = r == j + 1 ? w1 : Q4<R>{x.ax * f, x.ay * f, x.bx * f, x.by * f};
      ys[r] = j > 0 && r >= j ? q_ldcg(gr.y + r) : q_zero<R>();
    }
    __syncthreads();
    // e_j and tau_j: one warp, beside the sweep
    if (rank == G - 1 && warp == RT_WARPS - 1) {
      const R x1 = __ldcg(reinterpret_cast<const R*>(gr.x + j + 1) + (lane & 3));
      Acc<R> q2a;
      acc_load(gr.q2, q2a);
      const double q2 = acc_double(q2a), ss = acc_double(warp_gather<R>(gr.npart, NR, lane));
      if (lane < 4) {
        double e = x1;
        if (!last) {
          // |x| in the direction the reflector took; not a number stays visible
          if (!(ss >= 0.0)) e = ss;
          else if (!(f > R(0))) e = 0.0;
          else if (s_head[5] != R(0)) e = lane == 0 ? -ss * rsqrt(ss) : 0.0;
          else e = -ss * rsqrt(ss * q2) * (double)x1;
        }
        tk.e[4 * (size_t)(k0 + j) + lane] = e * scale;
        if (lane == 0) tk.tau[k0 + j] = f > R(0) ? 1.0 : 0.0;
      }
    }
    R cacc = R(0);  // this lane's part of c = w^H H w
    // ------------------------------------------------ sweep
    const int Jlo = (j + 1) / T;                       // first live column block
    const int live = (nt - Jlo) * (nt - Jlo + 1) / 2;  // tiles in dealing order
    // FP64 with few tiles left for the CTA: four warps share a tile (two columns
    // each, a component per lane), so that the SM's four quadrants work on it: a
    // tile takes 41 FP64 instructions of each of four warps instead of 146 of one
    bool teams = false;
    if constexpr (sizeof(R) == 8 && T == 8) teams = live <= 3 * G;
    if constexpr (sizeof(R) == 8 && T == 8) {
      if (teams) {
        const int team = warp >> 2, tw = warp & 3;
        const int r = lane >> 2, k = lane & 3;
        const unsigned s2 = quat_signs(SIGNS_RANK2, k), sr = quat_signs(SIGNS_ROW, k), sc = quat_signs(SIGNS_COL, k);
        for (int q = team; rank + q * G < live; q += 2) {
          int I, J;
          rt_tile(rank + q * G, nt, I, J);
          R* tl = tiles + (size_t)q * TILE;
          const bool diag = I == J;
          const int gr_ = I * T + r, rl = min(gr_, m - 1);
          const bool rin = gr_ < m;
          // row vectors: this lane's components of w and y, all of the new w
          const R wk = rin ? reinterpret_cast<const R*>(wp + rl)[k] : R(0);
          const R yk = rin ? reinterpret_cast<const R*>(ys + rl)[k] : R(0);
          Q4<R> nr = wn[rl];
          if (!rin) nr = q_zero<R>();
          R wx[4], yx[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            wx[u] = flip(__shfl_xor_sync(0xffffffffu, wk, u), s2 >> u);
            yx[u] = flip(__shfl_xor_sync(0xffffffffu, yk, u), s2 >> u);
          }
          const R nw[4] = {flip(nr.ax, sc), flip(nr.ay, sc >> 1), flip(nr.bx, sc >> 2), flip(nr.by, sc >> 3)};
          R rsum = R(0), csum[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int c = 2 * tw + u, gc = J * T + c, cl = min(gc, m - 1);
            Q4<R> wc = wp[cl], yc = ys[cl], nc = wn[cl];
            if (gc >= m) { wc = q_zero<R>(); yc = q_zero<R>(); nc = q_zero<R>(); }
            // the slot of (r, c) in the lanes' layout (t_load)
            R* e = tl + 2 * (((k >> 1) * EL + (c >> 2)) * 32 + r + 8 * (c & 3)) + (k & 1);
            R t0 = wx[0] * yc.ax, t1 = yx[0] * wc.ax;
            t0 = fma(wx[1], yc.ay, t0); t1 = fma(yx[1], wc.ay, t1);
            t0 = fma(wx[2], yc.bx, t0); t1 = fma(yx[2], wc.bx, t1);
            t0 = fma(wx[3], yc.by, t0); t1 = fma(yx[3], wc.by, t1);
            R v = *e - (t0 + t1);
            if (diag && r == c && k != 0) v = R(0);
            *e = v;
            if (gc == j + 1 && gr_ > j && rin) reinterpret_cast<R*>(gr.col + gr_)[k] = v;
            const R nq[4] = {flip(nc.ax, sr), flip(nc.ay, sr >> 1), flip(nc.bx, sr >> 2), flip(nc.by, sr >> 3)};
            R cs = R(0);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const R mq = __shfl_xor_sync(0xffffffffu, v, w);
              rsum = fma(mq, nq[w], rsum);
              cs = fma(mq, nw[w], cs);
            }
            csum[u] = cs;
          }
          s_team[team][tw][lane] = rsum;
          if (!diag) {
            // over the rows: lanes below 16 keep the first column, the others the second
            const bool up = lane & 16;
            R cs = (up ? csum[1] : csum[0]) + __shfl_xor_sync(0xffffffffu, up ? csum[0] : csum[1], 16);
            cs += __shfl_xor_sync(0xffffffffu, cs, 8);
            cs += __shfl_xor_sync(0xffffffffu, cs, 4);
            const int gc = J * T + 2 * tw + (lane >> 4);
            if ((lane & 12) == 0 && gc < m) reinterpret_cast<R*>(gr.part + (size_t)I * m + gc)[k] = cs;
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");
          if (tw == 0) {
            const R sum = (s_team[team][0][lane] + s_team[team][1][lane]) + (s_team[team][2][lane] + s_team[team][3][lane]);
            if (rin) reinterpret_cast<R*>(gr.part + (size_t)J * m + gr_)[k] = sum;
            const R nk = rin ? reinterpret_cast<const R*>(wn + rl)[k] : R(0);
            cacc = fma(diag ? nk : nk + nk, sum, cacc);  // an off-diagonal tile stands for its mirror too
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory");  // the sums are read
        }
      }
    }
    for (int q = warp; !teams && rank + q * G < live; q += RT_WARPS) {
      int I, J;
      rt_tile(rank + q * G, nt, I, J);
      R* tl = tiles + (size_t)q * TILE;
      const bool diag = I == J;
      const bool publish = J == Jlo && tc == (((j + 1) - J * T) & 3);
      const int pubq = ((j + 1) - J * T) >> 2;
      Q4<R> v[EL];
#pragma unroll
      for (int e = 0; e < EL; ++e) v[e] = t_load<EL>(tl, e, lane);
      R rs[RR * 4], cs[CC * 4];
#pragma unroll
      for (int k = 0; k < RR * 4; ++k) rs[k] = R(0);
#pragma unroll
      for (int k = 0; k < CC * 4; ++k) cs[k] = R(0);
      Q4<R> wr[RR], yr[RR], nr[RR];
#pragma unroll
      for (int i = 0; i < RR; ++i) {
        const int r0 = I * T + tr + 8 * i, r = min(r0, m - 1);
        wr[i] = wp[r]; yr[i] = ys[r]; nr[i] = wn[r];
        if (r0 >= m) { wr[i] = q_zero<R>(); yr[i] = q_zero<R>(); nr[i] = q_zero<R>(); }
      }
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        const int cc = J * T + tc + 4 * c, cl = min(cc, m - 1);
        Q4<R> wc = wp[cl], yc = ys[cl], nc = wn[cl];
        if (cc >= m) { wc = q_zero<R>(); yc = q_zero<R>(); nc = q_zero<R>(); }
#pragma unroll
        for (int i = 0; i < RR; ++i) {
          const int e = c * RR + i;
          const Q4<R> u = rank2(wr[i], yr[i], wc, yc);
          v[e].ax -= u.ax; v[e].ay -= u.ay; v[e].bx -= u.bx; v[e].by -= u.by;
          if (diag && tr + 8 * i == tc + 4 * c) { v[e].ay = 0; v[e].bx = 0; v[e].by = 0; }
          row_prod(rs + 4 * i, v[e], nc);
          col_prod(cs + 4 * c, v[e], nr[i]);
          t_store<EL>(tl, e, lane, v[e]);
          if (publish && c == pubq) {
            const int r = I * T + tr + 8 * i;
            if (r > j && r < m) q_store(gr.col + r, v[e]);
          }
        }
      }
      // row sums over the four column lanes, column sums over the eight row lanes
      scatter_sum<RR * 4, 16, 8, R>(rs, lane);
      {
        // column lane tc is left with values [tc NRV, (tc + 1) NRV) of (row, component)
        const int k = tc * NRV;
        const int r = I * T + tr + 8 * (k / 4);
        if (r < m) {
          R* o = reinterpret_cast<R*>(gr.part + (size_t)J * m + r) + (k & 3);
          const R* wv = reinterpret_cast<const R*>(wn + r) + (k & 3);
          R cp = R(0);
#pragma unroll
          for (int q2 = 0; q2 < NRV; ++q2) {
            o[q2] = rs[q2];
            cp = fma(wv[q2], rs[q2], cp);
          }
          cacc += diag ? cp : cp + cp;  // an off-diagonal tile stands for its mirror too
        }
      }
      if (!diag) {
        scatter_sum<CC * 4, 4, 1, R>(cs, lane);
        const int k = tr * NCV;
        const int c = J * T + tc + 4 * (k / 4);
        if (c < m) {
          R* o = reinterpret_cast<R*>(gr.part + (size_t)I * m + c) + (k & 3);
#pragma unroll
          for (int q2 = 0; q2 < NCV; ++q2) o[q2] = cs[q2];
        }
      }
    }
    // w_j in place of column j (this CTA's rows of the partition that formed it)
    for (int idx = tid; idx < 4 * nrows; idx += RT_THREADS) {
      const int r = rows0 + (idx >> 2), k = idx & 3;
      if (r <= j) continue;
      R* dst = reinterpret_cast<R*>((k < 2 ? A : B) + r + (int64_t)j * ld);
      dst[k & 1] = r == j + 1 ? s_head[1 + k] : own_x[idx] * f;
    }
    // this CTA's part of c
    {
      const Acc<R> c = acc_lanes<16, 1>(acc_value(cacc));
      if (lane == 0) acc_store(s_cw + warp, c);
      __syncthreads();
      if (warp == 0) {
        Acc<R> t{};
        if (lane < RT_WARPS) {
          if constexpr (sizeof(R) == 8) t = s_cw[lane];
          else { const float2 u = reinterpret_cast<const float2*>(s_cw)[lane]; t = Pair{u.x, u.y}; }
        }
        t = acc_lanes<RT_WARPS / 2, 1>(t);
        if (lane == 0) acc_store(gr.cpart + rank, t);
      }
    }
    if (!barrier()) return false;
    // ------------------------------------------------ rows: g, y_j and column j + 1
    const int p = j + 1;
    partition(p);
    if (nrows > 0) {
      if (warp == RT_WARPS - 1) {
        const Acc<R> c = warp_gather<R>(gr.cpart, G, lane);
        if (lane == 0) s_hc = acc_half(c);
      }
      constexpr int RPW = 32 / LPR;               // rows per warp and pass
      const int sl = lane & (LPR - 1);
      const int k = sl / (LPR / 4);               // component this lane ends with
      const bool rep = (sl & (LPR / 4 - 1)) == 0;  // one lane of those holding it
      // the CTA's rows, and row p once more for its own use
      for (int i0 = warp * RPW; i0 <= nrows; i0 += RT_WARPS * RPW) {
        const int i = i0 + lane / LPR;
        const bool in = i <= nrows;
        const int r = i < nrows ? rows0 + i : p;
        R s[4] = {R(0), R(0), R(0), R(0)};
        R x = R(0);
        if (in) {
          if (i < nrows) x = __ldcg(reinterpret_cast<const R*>(gr.x + r) + k);
#pragma unroll 4
          for (int b = Jlo + sl; b < nt; b += LPR) {
            const Q4<R> t = q_ldcg(gr.part + (size_t)b * m + r);
            s[0] += t.ax; s[1] += t.ay; s[2] += t.bx; s[3] += t.by;
          }
        }
        scatter_sum<4, LPR / 2, LPR / 4, R>(s, lane);
#pragma unroll
        for (int o = LPR / 8; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
        if (in && rep) {
          own_g[4 * i + k] = s[0];
          if (i < nrows) own_w[4 * i + k] = r == p ? s_head[1 + k] : x * f;
        }
      }
    }
    {
      Acc<R> ss{};
      R xfirst = R(0);
      const int k = tid & 3;
      R col = R(0);
      if (tid < 4 * nrows) col = __ldcg(reinterpret_cast<const R*>(gr.col + rows0) + tid);
      __syncthreads();
      if (nrows > 0) {
        const R g1 = own_g[4 * nrows + k];
        const R hc = s_hc;
        const R wk1 = s_head[1 + k];
        const R yk1 = g1 - hc * wk1;
        // this lane's signs of the structured products
        const bool n1 = k & 1, n2 = k == 1 || k == 2, n3 = k >= 2;
        R wc[4], yc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          wc[q] = __shfl_sync(0xffffffffu, wk1, q);
          yc[q] = __shfl_sync(0xffffffffu, yk1, q);
        }
        if (n1) { wc[1] = -wc[1]; yc[1] = -yc[1]; }
        if (n2) { wc[2] = -wc[2]; yc[2] = -yc[2]; }
        if (n3) { wc[3] = -wc[3]; yc[3] = -yc[3]; }
        for (int idx = tid; idx < ((4 * nrows + 31) & ~31); idx += RT_THREADS) {
          const bool in = idx < 4 * nrows;
          const int r = rows0 + (idx >> 2);
          if (in && idx != tid) col = __ldcg(reinterpret_cast<const R*>(gr.col + rows0) + idx);
          const R w = in ? own_w[idx] : R(0), g = in ? own_g[idx] : R(0);
          const R y = g - hc * w;
          R u = w * yc[0], t = y * wc[0];
#pragma unroll
          for (int q = 1; q < 4; ++q) {
            u = fma(__shfl_xor_sync(0xffffffffu, w, q), yc[q], u);
            t = fma(__shfl_xor_sync(0xffffffffu, y, q), wc[q], t);
          }
          R x = R(0);
          if (in) {
            x = col - (u + t);
            if (r == p) { if (k) x = R(0); else tk.d[k0 + p] = (double)x * scale; }
            own_x[idx] = x;
            reinterpret_cast<R*>(gr.x)[4 * r + k] = x;
            reinterpret_cast<R*>(gr.y)[4 * r + k] = y;
            if (r > p) acc_square(ss, x);
          }
          if (idx == tid) xfirst = x;
        }
      }
      publish_norms(p, xfirst, ss);
    }
    if (!barrier()) return false;
  }
  if (rank == 0 && tid == 0 && m > 0) {
    double* e = tk.e + 4 * (size_t)(n - 1);
    e[0] = e[1] = e[2] = e[3] = 0.0;
    tk.tau[n - 1] = 0.0;
  }
  return true;
}

template <typename R, int T, bool CL>
__global__ void __launch_bounds__(RT_THREADS, 1) k_tri_resident(const TriArgs<R> a) {
  extern __shared__ __align__(16) unsigned char rt_smem[];
  constexpr int LPR = sizeof(R) == 8 ? 32 : 8;
  const int group = blockIdx.x / a.G, rank = blockIdx.x % a.G;
  const TriGroup<R> gr = tri_group<R>(a.ws + (size_t)group * a.ws_stride, a.G, a.m_max, T);
  unsigned target = 0;
  if constexpr (CL) {
    // a queue of matrices: each cluster's first CTA takes one for all of them
    __shared__ int s_task;
    for (int it = 0; a.tasks; ++it) {
      if (rank == 0 && threadIdx.x == 0) gr.slot[it & 1] = atomicAdd(a.queue, 1);
      cluster_barrier();
      if (threadIdx.x == 0) s_task = __ldcg(gr.slot + (it & 1));
      __syncthreads();
      const int t = s_task;
      if (t >= a.ntasks) return;
      TriTask<R> tk = a.tasks[t];
      if (!tk.M) tk.M = a.base + tk.off;
      if (tk.n > 0) reduce_matrix<R, T, LPR, true>(tk, gr, rank, a.G, rt_smem, target, a.err, a.limit);
      __syncthreads();
    }
  }
  if (!reduce_matrix<R, T, LPR, CL>(a.one, gr, rank, a.G, rt_smem, target, a.err, a.limit) && rank == 0 && threadIdx.x == 0)
    a.one.d[a.one.k0] = __longlong_as_double(0x7ff8000000000000ll);
}

template <typename R>
size_t rt_smem_bytes(int m, int T, int G) {
  const int nt = (m + T - 1) / T, ntiles = nt * (nt + 1) / 2;
  const size_t cap = (size_t)((ntiles + G - 1) / G);
  const int NR = row_ctas<R>(G);
  return cap * T * T * 4 * sizeof(R) + sizeof(Q4<R>) * (3 * (size_t)m + 3 * (size_t)((m + NR - 1) / NR) + 1) + (size_t)nt + 16;
}

// shared-memory opt-in (and clusters above eight CTAs), once per device and kernel
template <typename R, int T, bool CL>
int rt_attr() {
  static std::atomic<unsigned long long> set{0};
  int dev = 0;
  ZQ_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(set.load() & bit)) {
    ZQ_CUDA(cudaFuncSetAttribute(k_tri_resident<R, T, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM_MAX));
    if (CL) ZQ_CUDA(cudaFuncSetAttribute(k_tri_resident<R, T, CL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set.fetch_or(bit);
  }
  return ZQ_OK;
}

template <typename R, int T, bool CL>
int rt_launch(const TriArgs<R>& a, int ctas, size_t smem, cudaStream_t st) {
  if (int rc = rt_attr<R, T, CL>()) return rc;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(RT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if (CL) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)a.G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ZQ_CUDA(cudaLaunchKernelEx(&cfg, k_tri_resident<R, T, CL>, a));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

// clusters of G CTAs with all of the shared memory that run at once on this device
template <typename R, int T>
int clusters_at_once(int G) {
  static std::atomic<int> known[64][RT_CLUSTER + 1];
  int dev = 0;
  if (G < 1 || G > RT_CLUSTER || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int k = known[dev][G].load();
  if (k == 0) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)G);
    cfg.blockDim = dim3(RT_THREADS);
    cfg.dynamicSmemBytes = RT_SMEM_MAX;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (rt_attr<R, T, true>() != ZQ_OK ||
        cudaOccupancyMaxActiveClusters(&clusters, k_tri_resident<R, T, true>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    k = clusters + 1;
    known[dev][G].store(k);
  }
  return k - 1;
}

}  // namespace

namespace {
// Tile edge: FP64 sweeps are bound by the FP64 pipe (an instruction holds its SM
// quadrant for 64 cycles), so small tiles spread them over more warps (n = 750:
// 24.0 ms with 8, 28.5 ms with 16); FP32 sweeps at 16 (n = 1023: 16.6 ms, 17.6
// with 8, 18.6 with 32).
template <typename R> constexpr int rt_tile_edge() { return sizeof(R) == 8 ? 8 : 16; }
// Up to this order one cluster of 16 CTAs does the reduction: its hardware
// barrier takes ~1000 cycles against ~2400 through L2, which outweighs having
// fewer SMs for the tiles (FP32, n = 300: 8.0 against 8.6 ms for the whole
// solve; FP64, n = 64: 4.85 against 4.99 ms), and matrices of different streams
// reduce side by side.
template <typename R> constexpr int rt_cluster_max() { return sizeof(R) == 8 ? 64 : 448; }
}  // namespace

int sm_count() {
  static std::atomic<int> sms[64];
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if ((v = sms[dev].load())) return v;
  int coop = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  sms[dev].store(v);
  return v;
}

template <typename R>
bool resident_fits(int m, int ctas) {
  if (m < 1 || ctas < 1) return false;
  constexpr int T = rt_tile_edge<R>();
  const int nt = (m + T - 1) / T, ntiles = nt * (nt + 1) / 2;
  return rt_smem_bytes<R>(m, T, ctas < ntiles ? ctas : ntiles) <= (size_t)RT_SMEM_MAX;
}

template <typename R>
int resident_max(int ctas) {
  if (ctas < 1) return 0;
  int lo = 0, hi = RESIDENT_MMAX;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (resident_fits<R>(mid, ctas)) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename R>
int tri_resident(const TridiagView<R>& v, int k0, int ctas, cudaStream_t st) {
  const int m = v.n - k0;
  constexpr int T = rt_tile_edge<R>();
  const int nt = (m + T - 1) / T, ntiles = nt * (nt + 1) / 2;
  const bool cl = m <= rt_cluster_max<R>() && clusters_at_once<R, T>(RT_CLUSTER) > 0;
  const int most = cl ? RT_CLUSTER : ctas;
  const int G = most < ntiles ? most : ntiles;
  TriArgs<R> a{};
  a.one = TriTask<R>{v.M, v.n, k0, v.ld, v.d, v.e, v.tau, 0};
  a.G = G; a.m_max = m;
  a.ws = reinterpret_cast<unsigned char*>(v.rws);
  a.ws_stride = 0;
  a.err = v.tc_err;
  a.limit = pipeline_wait_cycles();
  ZQ_CUDA(cudaMemsetAsync(v.rws, 0, 64, st));  // counter, abort flag
  const size_t smem = rt_smem_bytes<R>(m, T, G);
  return cl ? rt_launch<R, T, true>(a, G, smem, st) : rt_launch<R, T, false>(a, G, smem, st);
}

int resident_ctas(int n, bool alone) {
  const int sms = sm_count();
  // beside other solves: a quarter of the SMs where that is enough
  return !alone && n <= resident_max<float>(sms / 4) && n <= resident_max<double>(sms / 4) ? sms / 4 : sms;
}

size_t resident_workspace_bytes(int n, size_t real_bytes) {
  const int m = n < RESIDENT_MMAX ? n : RESIDENT_MMAX;
  return tri_group_bytes(1024, m, 8, real_bytes);
}

// Time of a queue (largest order first) on clusters of G, in clock cycles: per
// column ~12000 outside the sweep, and the sweep's tiles in rounds of one per SM
// quadrant at 9700 (146 FP64 instructions of 64 cycles and latencies); each
// matrix goes to the cluster that is free first. 0: G cannot hold the largest.
static double tri_queue_cycles(const int* orders, int count, int G) {
  constexpr int T = rt_tile_edge<double>();
  const int clusters = clusters_at_once<double, T>(G);
  if (count < 1 || clusters < 1 || rt_smem_bytes<double>(orders[0], T, G) > (size_t)RT_SMEM_MAX) return 0.0;
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (int q = 0; q < clusters; ++q) free_at.push(0.0);
  double end = 0.0, cost = 0.0;
  for (int i = 0; i < count; ++i) {
    if (i == 0 || orders[i] != orders[i - 1]) {
      cost = 0.0;
      for (int a = (orders[i] + T - 1) / T; a > 0; --a) {
        const int tiles = a * (a + 1) / 2;
        cost += T * (12000.0 + 9700.0 * ((tiles + 4 * G - 1) / (4 * G)));
      }
    }
    const double t = free_at.top() + cost;
    free_at.pop();
    free_at.push(t);
    end = std::max(end, t);
  }
  return end;
}

int tri_queue_cluster(const int* orders, int count, double* cycles) {
  int best = 0;
  double least = 0.0;
  for (int G = 1; G <= RT_CLUSTER; ++G) {
    const double c = tri_queue_cycles(orders, count, G);
    if (c > 0.0 && (best == 0 || c < least)) { best = G; least = c; }
  }
  if (cycles) *cycles = least;
  return best;
}

static size_t tri_queue_stride(int G, int m_max) {
  return (tri_group_bytes(G, m_max, rt_tile_edge<double>(), sizeof(double)) + 255) & ~(size_t)255;
}
static int tri_queue_groups(int G) { return std::max(1, clusters_at_once<double, rt_tile_edge<double>()>(G)); }

size_t tri_queue_bytes(int G, int m_max, int ntasks) {
  return tri_queue_stride(G, m_max) * std::min(ntasks, tri_queue_groups(G));
}

int tri_queue(const TriTask<double>* tasks, int ntasks, double2* base, int m_max, int G, void* ws, int* queue,
              cudaStream_t st) {
  if (ntasks <= 0) return ZQ_OK;
  constexpr int T = rt_tile_edge<double>();
  TriArgs<double> a{};
  a.tasks = tasks; a.ntasks = ntasks; a.base = base; a.queue = queue;
  a.G = G; a.m_max = m_max;
  a.ws = reinterpret_cast<unsigned char*>(ws);
  a.ws_stride = tri_queue_stride(G, m_max);
  const int groups = std::min(ntasks, tri_queue_groups(G));
  ZQ_CUDA(cudaMemsetAsync(queue, 0, sizeof(int), st));
  return rt_launch<double, T, true>(a, groups * G, rt_smem_bytes<double>(m_max, T, G), st);
}

template bool resident_fits<float>(int, int);
template bool resident_fits<double>(int, int);
template int resident_max<float>(int);
template int resident_max<double>(int);
template int tri_resident<float>(const TridiagView<float>&, int, int, cudaStream_t);
template int tri_resident<double>(const TridiagView<double>&, int, int, cudaStream_t);

}  // namespace zq
