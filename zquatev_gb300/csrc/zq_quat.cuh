// Quaternion entries as four reals, and their structured products.
#pragma once

#include <cuda_runtime.h>

namespace zq {

// four reals: (a.x, a.y, b.x, b.y) of a quaternion entry
template <typename R> struct alignas(16) Q4 { R ax, ay, bx, by; };

template <typename R> __device__ __forceinline__ Q4<R> q_zero() { return Q4<R>{R(0), R(0), R(0), R(0)}; }
__device__ __forceinline__ Q4<float> q_ldcg(const Q4<float>* p) {
  const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
  return Q4<float>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Q4<double> q_ldcg(const Q4<double>* p) {
  const double2 u = __ldcg(reinterpret_cast<const double2*>(p)), v = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return Q4<double>{u.x, u.y, v.x, v.y};
}
__device__ __forceinline__ void q_store(Q4<float>* p, const Q4<float>& q) {
  *reinterpret_cast<float4*>(p) = make_float4(q.ax, q.ay, q.bx, q.by);
}
__device__ __forceinline__ void q_store(Q4<double>* p, const Q4<double>& q) {
  reinterpret_cast<double2*>(p)[0] = make_double2(q.ax, q.ay);
  reinterpret_cast<double2*>(p)[1] = make_double2(q.bx, q.by);
}
// the structured rank-2 term at (r, c): row vectors (w, y)_r, column vectors (w, y)_c
//   A: wa_r conj(ya_c) + conj(wb_r) yb_c + ya_r conj(wa_c) + conj(yb_r) wb_c
//   B: wb_r conj(ya_c) - conj(wa_r) yb_c + yb_r conj(wa_c) - conj(ya_r) wb_c
template <typename R>
__device__ __forceinline__ Q4<R> rank2(const Q4<R>& wr, const Q4<R>& yr, const Q4<R>& wc, const Q4<R>& yc) {
  Q4<R> t;
  t.ax = wr.ax * yc.ax; t.ax = fma(wr.ay, yc.ay, t.ax);
  t.ay = wr.ay * yc.ax; t.ay = fma(-wr.ax, yc.ay, t.ay);
  t.bx = wr.bx * yc.ax; t.bx = fma(wr.by, yc.ay, t.bx);
  t.by = wr.by * yc.ax; t.by = fma(-wr.bx, yc.ay, t.by);
  t.ax = fma(wr.bx, yc.bx, t.ax); t.ax = fma(wr.by, yc.by, t.ax);
  t.ay = fma(wr.bx, yc.by, t.ay); t.ay = fma(-wr.by, yc.bx, t.ay);
  t.bx = fma(-wr.ax, yc.bx, t.bx); t.bx = fma(-wr.ay, yc.by, t.bx);
  t.by = fma(-wr.ax, yc.by, t.by); t.by = fma(wr.ay, yc.bx, t.by);
  t.ax = fma(yr.ax, wc.ax, t.ax); t.ax = fma(yr.ay, wc.ay, t.ax);
  t.ay = fma(yr.ay, wc.ax, t.ay); t.ay = fma(-yr.ax, wc.ay, t.ay);
  t.bx = fma(yr.bx, wc.ax, t.bx); t.bx = fma(yr.by, wc.ay, t.bx);
  t.by = fma(yr.by, wc.ax, t.by); t.by = fma(-yr.bx, wc.ay, t.by);
  t.ax = fma(yr.bx, wc.bx, t.ax); t.ax = fma(yr.by, wc.by, t.ax);
  t.ay = fma(yr.bx, wc.by, t.ay); t.ay = fma(-yr.by, wc.bx, t.ay);
  t.bx = fma(-yr.ax, wc.bx, t.bx); t.bx = fma(-yr.ay, wc.by, t.bx);
  t.by = fma(-yr.ax, wc.by, t.by); t.by = fma(yr.ay, wc.bx, t.by);
  return t;
}
// g_r += M(r, c) w_c:  ga += a wa - conj(b) wb,  gb += b wa + conj(a) wb
template <typename R>
__device__ __forceinline__ void row_prod(R* g, const Q4<R>& m, const Q4<R>& w) {
  g[0] = fma(m.ax, w.ax, g[0]); g[0] = fma(-m.ay, w.ay, g[0]); g[0] = fma(-m.bx, w.bx, g[0]); g[0] = fma(-m.by, w.by, g[0]);
  g[1] = fma(m.ax, w.ay, g[1]); g[1] = fma(m.ay, w.ax, g[1]); g[1] = fma(-m.bx, w.by, g[1]); g[1] = fma(m.by, w.bx, g[1]);
  g[2] = fma(m.bx, w.ax, g[2]); g[2] = fma(-m.by, w.ay, g[2]); g[2] = fma(m.ax, w.bx, g[2]); g[2] = fma(m.ay, w.by, g[2]);
  g[3] = fma(m.bx, w.ay, g[3]); g[3] = fma(m.by, w.ax, g[3]); g[3] = fma(m.ax, w.by, g[3]); g[3] = fma(-m.ay, w.bx, g[3]);
}
// g_c += M(c, r) w_r from the stored (r, c):  ga += conj(a) wa + conj(b) wb,  gb += -b wa + a wb
template <typename R>
__device__ __forceinline__ void col_prod(R* g, const Q4<R>& m, const Q4<R>& w) {
  g[0] = fma(m.ax, w.ax, g[0]); g[0] = fma(m.ay, w.ay, g[0]); g[0] = fma(m.bx, w.bx, g[0]); g[0] = fma(m.by, w.by, g[0]);
  g[1] = fma(m.ax, w.ay, g[1]); g[1] = fma(-m.ay, w.ax, g[1]); g[1] = fma(m.bx, w.by, g[1]); g[1] = fma(-m.by, w.bx, g[1]);
  g[2] = fma(-m.bx, w.ax, g[2]); g[2] = fma(m.by, w.ay, g[2]); g[2] = fma(m.ax, w.bx, g[2]); g[2] = fma(-m.ay, w.by, g[2]);
  g[3] = fma(-m.bx, w.ay, g[3]); g[3] = fma(-m.by, w.ax, g[3]); g[3] = fma(m.ax, w.by, g[3]); g[3] = fma(m.ay, w.bx, g[3]);
}
// v[0..N) summed over the lanes that differ in the bits of MASK, MASK/2, ..., LOW:
// each step halves the values a lane keeps; returns in v[0..N / lanes)
template <int N, int MASK, int LOW, typename R>
__device__ __forceinline__ void scatter_sum(R* v, int lane) {
  if constexpr (MASK >= LOW) {
    const bool up = lane & MASK;
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
      const R keep = up ? v[N / 2 + k] : v[k], send = up ? v[k] : v[N / 2 + k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
    }
    scatter_sum<N / 2, MASK / 2, LOW, R>(v, lane);
  }
}

}  // namespace zq
