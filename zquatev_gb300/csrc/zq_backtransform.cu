// Back-transformation and output assembly.
//
// Reference: zquatev.cc:74-98 -- band extraction + zhbev, U = Q0 Z and
// V = Q1 Z by zgemm3m (zquatev.cc:86-90), the explicit Q0/Q1 accumulated
// during the panels (blocked.cc:477-544), and the symmetry fill of the right
// half (zquatev.cc:92-98).
//
// Here Q is never accumulated during the reduction. After the tridiagonal is
// known:
//   1. phase_reduce: the quaternion subdiagonal e_k is made real by unit
//      quaternions phi with phi_{k+1} = e_k phi_k / |e_k|, so that
//      phi_{k+1}^H e_k phi_k = |e_k| (exact similarity, FP64);
//   2. form_q: X = Q * [diag(alpha); diag(beta)] (the left half of Q Phi) by
//      applying the stored reflectors backwards in compact-WY blocks,
//      Q_blk = I - V T V^H, with the structured 2x2-block T built from the
//      Gram matrix of the block's reflectors. Only the trailing (L x L)
//      sub-blocks that can be non-zero are touched (zungtr-style);
//   3. apply_z: (U; V) = X Z with the REAL eigenvector matrix Z of the
//      real tridiagonal; complex X is read as a real array with twice the
//      rows, so this is one real DGEMM;
//   4. symmetry_fill: D[:, n:] = (-conj(V); conj(U)).
#include "zq_common.cuh"
#include "zq_kernels.h"
#include "zq_tc32.h"

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace zq {

// Quaternion phases: phi_0 = 1, phi_{k+1} = u_k phi_k with u_k = e_k / |e_k|
// (phi reset to 1 where e_k = 0), i.e. a segmented prefix product of unit
// quaternions. One CTA: each thread takes a contiguous chunk, a Hillis-Steele
// scan over the 1024 chunk products combines them (quaternion products are
// associative), then every thread rewrites its chunk; each phi is normalised
// when written.
struct Quat { double a0, a1, b0, b1; int reset; };
// q(a1, b1) q(a2, b2) = q(a1 a2 - conj(b1) b2, b1 a2 + conj(a1) b2)
__device__ __forceinline__ Quat qmul(const Quat& x, const Quat& y) {
  Quat r;
  r.a0 = (x.a0 * y.a0 - x.a1 * y.a1) - (x.b0 * y.b0 + x.b1 * y.b1);
  r.a1 = (x.a0 * y.a1 + x.a1 * y.a0) - (x.b0 * y.b1 - x.b1 * y.b0);
  r.b0 = (x.b0 * y.a0 - x.b1 * y.a1) + (x.a0 * y.b0 + x.a1 * y.b1);
  r.b1 = (x.b0 * y.a1 + x.b1 * y.a0) + (x.a0 * y.b1 - x.a1 * y.b0);
  r.reset = 0;
  return r;
}
// later o earlier (segmented: a reset in `later` drops `earlier`)
__device__ __forceinline__ Quat qcombine(const Quat& later, const Quat& earlier) {
  if (later.reset) return later;
  Quat r = qmul(later, earlier);
  r.reset = earlier.reset;
  return r;
}
__device__ __forceinline__ Quat qunit_of(const double* e, int k, double& nrm) {
  double ea0 = e[4 * k], ea1 = e[4 * k + 1], eb0 = e[4 * k + 2], eb1 = e[4 * k + 3], back = 1.0;
  // entries whose squares leave the range of doubles are brought to [1, 2) first
  const unsigned long long t0 = abs_bits(ea0) > abs_bits(ea1) ? abs_bits(ea0) : abs_bits(ea1);
  const unsigned long long t1 = abs_bits(eb0) > abs_bits(eb1) ? abs_bits(eb0) : abs_bits(eb1);
  const int ex = (int)((t0 > t1 ? t0 : t1) >> 52);
  if (ex > 0 && ex < 2046 && (ex < 1023 - 450 || ex > 1023 + 450)) {
    const double sc = __hiloint2double((2046 - ex) << 20, 0);
    back = __hiloint2double(ex << 20, 0);
    ea0 *= sc; ea1 *= sc; eb0 *= sc; eb1 *= sc;
  }
  nrm = sqrt(ea0 * ea0 + ea1 * ea1 + eb0 * eb0 + eb1 * eb1);
  Quat u;
  if (nrm > 0.0) { const double s = 1.0 / nrm; u.a0 = ea0 * s; u.a1 = ea1 * s; u.b0 = eb0 * s; u.b1 = eb1 * s; u.reset = 0; }
  else { u.a0 = 1.0; u.a1 = 0.0; u.b0 = 0.0; u.b1 = 0.0; u.reset = 1; }
  nrm *= back;
  return u;
}
// Few threads: an FP64 instruction holds its SM quadrant for 64 cycles a warp, so
// the scan's steps cost by the warps that take part (1024 threads at any order:
// 59 us at n = 23, 78 us at n = 750; now 8 and 41 us).
constexpr int PH_T = 256;
__global__ void __launch_bounds__(PH_T) k_phase(const double* e, int n, double* offd, double* phi, const DcMat* mats) {
  pdl_wait();
  __shared__ Quat s_q[PH_T];
  if (mats) {
    const DcMat mt = mats[blockIdx.x];
    n = mt.n;
    e += 4 * (int64_t)mt.p; offd += mt.p; phi += 4 * (int64_t)mt.p;
  }
  const int t = threadIdx.x, T = blockDim.x;
  const int m = n - 1;                      // number of u_k
  const int per = (m + T - 1) / T;
  const int k0 = t * per, k1 = (k0 + per < m) ? k0 + per : m;
  Quat acc{1.0, 0.0, 0.0, 0.0, 0};
  for (int k = k0; k < k1; ++k) {
    double nrm;
    const Quat u = qunit_of(e, k, nrm);
    acc = qcombine(u, acc);
  }
  s_q[t] = acc;
  __syncthreads();
  for (int off = 1; off < T && off * per < m; off <<= 1) {
    Quat v = s_q[t];
    if (t >= off) v = qcombine(v, s_q[t - off]);
    __syncthreads();
    s_q[t] = v;
    __syncthreads();
  }
  // exclusive prefix of this chunk = inclusive prefix of the previous one
  Quat run = (t > 0) ? s_q[t - 1] : Quat{1.0, 0.0, 0.0, 0.0, 0};
  if (t == 0) { phi[0] = 1.0; phi[1] = 0.0; phi[2] = 0.0; phi[3] = 0.0; }
  for (int k = k0; k < k1; ++k) {
    double nrm;
    const Quat u = qunit_of(e, k, nrm);
    offd[k] = nrm;
    run = qcombine(u, run);
    const double s = 1.0 / sqrt(run.a0 * run.a0 + run.a1 * run.a1 + run.b0 * run.b0 + run.b1 * run.b1);
    phi[4 * (k + 1) + 0] = run.a0 * s; phi[4 * (k + 1) + 1] = run.a1 * s;
    phi[4 * (k + 1) + 2] = run.b0 * s; phi[4 * (k + 1) + 3] = run.b1 * s;
  }
}

static int phase_threads(int n) { return n <= 32 ? 32 : (n <= 256 ? 64 : (n <= 1024 ? 128 : PH_T)); }

int phase_reduce(const double* e, int n, double* offd, double* phi, cudaStream_t st) {
  if (n <= 0) return ZQ_OK;
  ZQ_CUDA(launch_pdl_smem(k_phase, dim3(1), dim3(phase_threads(n)), 0, st, e, n, offd, phi, nullptr));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int phase_reduce_forest(const double* e, const DcMat* mats, int count, int nmax, double* offd, double* phi,
                        cudaStream_t st) {
  if (count <= 0) return ZQ_OK;
  ZQ_CUDA(launch_pdl_smem(k_phase, dim3(count), dim3(phase_threads(nmax)), 0, st, e, nmax, offd, phi, mats));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

// X = [diag(alpha); diag(beta)]
template <typename Z>
__global__ void k_init_x(Z* X, int64_t ldx, int n, const double* phi) {
  pdl_wait();
  const int64_t total = (int64_t)2 * n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t % (2 * n));
    const int c = (int)(t / (2 * n));
    Z v = czero<Z>();
    if (r == c) { v.x = phi[4 * c]; v.y = phi[4 * c + 1]; }
    else if (r == n + c) { v.x = phi[4 * c + 2]; v.y = phi[4 * c + 3]; }
    X[r + (int64_t)c * ldx] = v;
  }
}

// pack the block's reflectors: Wa[r, i] = A(p+1+r, p+i) for r >= i, else 0 (same for B)
template <typename Z>
__global__ void k_pack_w(const Z* M, int64_t ldm, int n, int p, int kb, int L, Z* Wa, Z* Wb) {
  pdl_wait();
  const int64_t total = (int64_t)L * kb;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t % L), i = (int)(t / L);
    Z va = czero<Z>(), vb = va;
    if (r >= i) {
      const int64_t o = (p + 1 + r) + (int64_t)(p + i) * ldm;
      va = M[o];
      vb = M[n + o];
    }
    Wa[r + (int64_t)i * L] = va;
    Wb[r + (int64_t)i * L] = vb;
  }
}

// T (kb x kb quaternion, upper triangular) from G1 = <w_i, w_l>, G2 = [w_i, w_l]:
//   T[k][k] = 1,  T[i][k] = - sum_{i<=l<k} T[i][l] q(G1[l][k], G2[l][k])
// One CTA of 1024 threads: thread (i, g) sums the l = i+g, i+g+16, ... terms of
// column k; the 16 partials of each row are reduced in shared memory.
constexpr int BT_G = 16;
template <typename Z>
__global__ void __launch_bounds__(1024) k_build_t(const Z* G1, const Z* G2, int kb, Z* Ta, Z* Tb) {
  pdl_wait();
  const int tid = threadIdx.x;
  const int i = tid & 63, g = tid >> 6;
  __shared__ Z red[BT_G][64][2];
  for (int t = tid; t < kb * kb; t += blockDim.x) { Ta[t] = czero<Z>(); Tb[t] = czero<Z>(); }
  __syncthreads();
  for (int k = 0; k < kb; ++k) {
    Z sa = czero<Z>(), sb = sa;
    if (i < k) {
      for (int l = i + g; l < k; l += BT_G) {
        const Z ta = Ta[i + l * kb], tb = Tb[i + l * kb];
        const Z g1 = G1[l + k * kb], g2 = G2[l + k * kb];
        // q(ta, tb) q(g1, g2) = q(ta g1 - conj(tb) g2, tb g1 + conj(ta) g2)
        cfma(sa, ta, g1); cfmac(sa, cneg(tb), g2);
        cfma(sb, tb, g1); cfmac(sb, ta, g2);
      }
    }
    red[g][i][0] = sa;
    red[g][i][1] = sb;
    __syncthreads();
    if (g == 0) {
      if (i < k) {
        Z ta = czero<Z>(), tb = ta;
        for (int q = 0; q < BT_G; ++q) { ta = cadd(ta, red[q][i][0]); tb = cadd(tb, red[q][i][1]); }
        Ta[i + k * kb] = cneg(ta);
        Tb[i + k * kb] = cneg(tb);
      } else if (i == k) {
        Z one = czero<Z>();
        one.x = 1;
        Ta[k + k * kb] = one;
        Tb[k + k * kb] = czero<Z>();
      }
    }
    __syncthreads();
  }
}

// split-K partial buffer of the Q formation (complex elements)
static int64_t fq_pcap(int n, int nbq) { return (int64_t)64 * nbq * (n > 64 ? n : 64); }

// Most K blocks (16 complex terms each) per split of the tensor-core W^H X
// product (env ZQ_FORMQ_KSPLIT; 0: only as many splits as fill the GPU). Each
// split accumulates in tensor memory, whose FP32 sums truncate; the splits are
// added in FP32 by the reduce. 8 blocks keep the refinement's second-step
// correction at 6.2e-8 at n2 = 8192 (one accumulation per output: 2.6e-7).
static int formq_kblocks_per_split() {
  static const int v = [] {
    const char* s = getenv("ZQ_FORMQ_KSPLIT");
    return s ? atoi(s) : 8;
  }();
  return v;
}

size_t form_q_workspace_bytes(int n, int nbq) {
  // Wa, Wb (n x nbq), G1, G2, Ta, Tb (nbq^2), C1e, C1o, C2e, C2o (nbq x n), split-K partials
  return sizeof(double2) * ((size_t)2 * n * nbq + 4 * (size_t)nbq * nbq + 4 * (size_t)nbq * n + (size_t)fq_pcap(n, nbq)) + 256;
}

// ----------------------------------------------------------------------------
// FP32: W, T and V = W T^H of every block in four launches
//
// They depend on the reflectors alone, not on X. One block after another (a pack,
// two Gram products of 64 x 64 outputs with their split sums, and the T recurrence
// on one SM, ~150 us a block on a second stream) they bound the whole formation up
// to n ~ 2000; all blocks at once they take as long as one. With V = W T^H the update
// is X -= W (V^H X): the two small products T (W^H X) between the large ones are gone
// too, and the two halves of the update share a launch. n = 750: 1.88 -> 0.98 ms,
// n = 4096: 31 -> 26 ms. (V = W T on the other side of the update is as fast, but the
// refinement's corrections grow by a third: 3.0e-8 -> 4.0e-8 at n = 4096.)
//
// W and V of a block start at row `pb` (of zeros: reflector pb begins one row
// lower) and have an even leading dimension, so that the tensor-core product reads
// W and X in 16-byte pieces.
// ----------------------------------------------------------------------------
constexpr int FQ_NB = 64;        // reflectors per block
// rows of W per partial Gram sum: few enough CTAs' worth for small orders (n = 512: 16
// CTAs of 256 rows took 89 us)
__host__ __device__ inline int fq_rows(int n) { return n <= 1024 ? 64 : 256; }
struct FqBlocks {
  const float2* M; int64_t ldm;
  int n, nref, nblocks;
  float2 *W, *V;                 // per block: the a parts (ld x kb), then the b parts
  float4 *part, *T;              // per block: partial Gram sums (chunks x 64 x 64), T (64 x 64, T[i + 64 k])
};
__host__ __device__ inline int fq_ld(int n, int b) { return (n - FQ_NB * b + 1) & ~1; }
__host__ __device__ inline int64_t fq_off(int n, int b) {  // complex elements before block b
  return (int64_t)2 * FQ_NB * ((int64_t)b * fq_ld(n, 0) - (int64_t)FQ_NB * b * (b - 1) / 2);
}
__host__ __device__ inline int fq_chunks(int n, int b) { return (n - FQ_NB * b + fq_rows(n) - 1) / fq_rows(n); }
__host__ __device__ inline int fq_kb(int nref, int b) { return nref - FQ_NB * b < FQ_NB ? nref - FQ_NB * b : FQ_NB; }
// bytes of W, V, T and the partial sums
static size_t fq_bytes(int n, int nblocks) {
  return 2 * sizeof(float2) * (size_t)fq_off(n, nblocks) +
         sizeof(float4) * FQ_NB * FQ_NB * (size_t)nblocks * (1 + fq_chunks(n, 0));
}

__global__ void __launch_bounds__(256) k_fq_pack(FqBlocks q) {
  pdl_wait();
  const int b = blockIdx.y, pb = FQ_NB * b, kb = fq_kb(q.nref, b), ld = fq_ld(q.n, b), rows = q.n - pb;
  float2* wa = q.W + fq_off(q.n, b);
  float2* wb = wa + (int64_t)ld * kb;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ld * kb; t += gridDim.x * blockDim.x) {
    const int r = t % ld, i = t / ld;
    float2 a = make_float2(0.f, 0.f), c = a;
    if (r > i && r < rows) {
      const int64_t o = pb + r + (int64_t)(pb + i) * q.ldm;
      a = q.M[o];
      c = q.M[q.n + o];
    }
    wa[t] = a;
    wb[t] = c;
  }
}

// Gram sums of one chunk of rows: quaternion <w_i, w_l> = (conj(wa_i) wa_l + conj(wb_i) wb_l,
// wa_i wb_l - wb_i wa_l), 4 x 4 of them per thread
__global__ void __launch_bounds__(256) k_fq_gram(FqBlocks q) {
  pdl_wait();
  const int b = blockIdx.y, ch = blockIdx.x;
  const int pb = FQ_NB * b, kb = fq_kb(q.nref, b), ld = fq_ld(q.n, b), rows = q.n - pb;
  if (ch * fq_rows(q.n) >= rows) return;
  __shared__ float4 w[32][FQ_NB + 1];
  const float2* wa = q.W + fq_off(q.n, b);
  const float2* wb = wa + (int64_t)ld * kb;
  const int tl = threadIdx.x & 15, ti = threadIdx.x >> 4;
  float4 acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int r1 = min((ch + 1) * fq_rows(q.n), rows);
  for (int r0 = ch * fq_rows(q.n); r0 < r1; r0 += 32) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; ++u) {  // a warp per column, a lane per row
      const int i = (threadIdx.x >> 5) + 8 * u, r = r0 + (threadIdx.x & 31);
      float2 a = make_float2(0.f, 0.f), c = a;
      if (i < kb && r < r1) { a = wa[r + (int64_t)i * ld]; c = wb[r + (int64_t)i * ld]; }
      w[threadIdx.x & 31][i] = make_float4(a.x, a.y, c.x, c.y);
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < 32; ++r) {
      float4 x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) { x[u] = w[r][ti + 16 * u]; y[u] = w[r][tl + 16 * u]; }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float4& g = acc[u][v];
          const float4 p = x[u], s = y[v];
          g.x = fmaf(p.x, s.x, g.x); g.x = fmaf(p.y, s.y, g.x); g.x = fmaf(p.z, s.z, g.x); g.x = fmaf(p.w, s.w, g.x);
          g.y = fmaf(p.x, s.y, g.y); g.y = fmaf(-p.y, s.x, g.y); g.y = fmaf(p.z, s.w, g.y); g.y = fmaf(-p.w, s.z, g.y);
          g.z = fmaf(p.x, s.z, g.z); g.z = fmaf(-p.y, s.w, g.z); g.z = fmaf(-p.z, s.x, g.z); g.z = fmaf(p.w, s.y, g.z);
          g.w = fmaf(p.x, s.w, g.w); g.w = fmaf(p.y, s.z, g.w); g.w = fmaf(-p.z, s.y, g.w); g.w = fmaf(-p.w, s.x, g.w);
        }
    }
  }
  float4* out = q.part + ((int64_t)b * fq_chunks(q.n, 0) + ch) * FQ_NB * FQ_NB;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) out[(ti + 16 * u) + FQ_NB * (tl + 16 * v)] = acc[u][v];
}

// T from the Gram sums, a CTA per block: T[k][k] = 1, T[i][k] = - sum_{i<=l<k} T[i][l] q(G[l][k]).
// Thread (i, g) sums the terms l = i + g, i + g + 16, ... of column k.
constexpr int FQ_T_SMEM = 2 * FQ_NB * FQ_NB * (int)sizeof(float4);
__global__ void __launch_bounds__(1024) k_fq_t(FqBlocks q) {
  pdl_wait();
  extern __shared__ float4 fq_sm[];
  float4* g = fq_sm;                  // G[l + 64 k]
  float4* tt = g + FQ_NB * FQ_NB;     // T[i + 64 k]
  __shared__ float4 red[BT_G][FQ_NB];
  const int b = blockIdx.x, kb = fq_kb(q.nref, b), chunks = fq_chunks(q.n, b);
  const int tid = threadIdx.x, i = tid & 63, s = tid >> 6;
  const float4* part = q.part + (int64_t)b * fq_chunks(q.n, 0) * FQ_NB * FQ_NB;
  for (int t = tid; t < FQ_NB * FQ_NB; t += blockDim.x) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < chunks; ++c) {
      const float4 u = part[(int64_t)c * FQ_NB * FQ_NB + t];
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    g[t] = v;
    tt[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  for (int k = 0; k < kb; ++k) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < k) {
      for (int l = i + s; l < k; l += BT_G) {
        // q(ta, tb) q(g1, g2) = q(ta g1 - conj(tb) g2, tb g1 + conj(ta) g2)
        const float4 t = tt[i + FQ_NB * l], v = g[l + FQ_NB * k];
        a.x += t.x * v.x - t.y * v.y - t.z * v.z - t.w * v.w;
        a.y += t.x * v.y + t.y * v.x - t.z * v.w + t.w * v.z;
        a.z += t.z * v.x - t.w * v.y + t.x * v.z + t.y * v.w;
        a.w += t.z * v.y + t.w * v.x + t.x * v.w - t.y * v.z;
      }
    }
    red[s][i] = a;
    __syncthreads();
    if (s == 0) {
      if (i < k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int u = 0; u < BT_G; ++u) { const float4 r = red[u][i]; v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w; }
        tt[i + FQ_NB * k] = make_float4(-v.x, -v.y, -v.z, -v.w);
      } else if (i == k) {
        tt[i + FQ_NB * k] = make_float4(1.f, 0.f, 0.f, 0.f);
      }
    }
    __syncthreads();
  }
  for (int t = tid; t < FQ_NB * FQ_NB; t += blockDim.x) q.T[(int64_t)b * FQ_NB * FQ_NB + t] = tt[t];
}

// V = W S, S = T^H, for 64 rows of a block: Va = Wa Sa - conj(Wb) Sb, Vb = Wb Sa + conj(Wa) Sb
constexpr int FQ_V_SMEM = 2 * FQ_NB * FQ_NB * (int)sizeof(float4);
__global__ void __launch_bounds__(256) k_fq_v(FqBlocks q) {
  pdl_wait();
  extern __shared__ float4 fq_sm[];
  float4* w = fq_sm;                  // W[r + 64 i]
  float4* tt = w + FQ_NB * FQ_NB;     // S[i + 64 c], the conjugate of T[c + 64 i]
  const int b = blockIdx.y, pb = FQ_NB * b, kb = fq_kb(q.nref, b), ld = fq_ld(q.n, b);
  const int r0 = FQ_NB * blockIdx.x;
  if (r0 >= q.n - pb) return;
  const float2* wa = q.W + fq_off(q.n, b);
  const float2* wb = wa + (int64_t)ld * kb;
  float2* va = q.V + fq_off(q.n, b);
  float2* vb = va + (int64_t)ld * kb;
  for (int t = threadIdx.x; t < FQ_NB * FQ_NB; t += blockDim.x) {
    const int r = r0 + (t & 63), i = t >> 6;
    float2 a = make_float2(0.f, 0.f), c = a;
    if (r < ld && i < kb) { a = wa[r + (int64_t)i * ld]; c = wb[r + (int64_t)i * ld]; }
    w[t] = make_float4(a.x, a.y, c.x, c.y);
    const float4 v = q.T[(int64_t)b * FQ_NB * FQ_NB + i + FQ_NB * (t & 63)];
    tt[(t & 63) + FQ_NB * i] = make_float4(v.x, -v.y, -v.z, -v.w);
  }
  __syncthreads();
  const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;
  float4 acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int i = 0; i < kb; ++i) {
    float4 x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { x[u] = w[tr + 16 * u + FQ_NB * i]; y[u] = tt[i + FQ_NB * (tc + 16 * u)]; }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        float4& o = acc[u][v];
        const float4 p = x[u], s = y[v];
        o.x = fmaf(p.x, s.x, o.x); o.x = fmaf(-p.y, s.y, o.x); o.x = fmaf(-p.z, s.z, o.x); o.x = fmaf(-p.w, s.w, o.x);
        o.y = fmaf(p.x, s.y, o.y); o.y = fmaf(p.y, s.x, o.y); o.y = fmaf(-p.z, s.w, o.y); o.y = fmaf(p.w, s.z, o.y);
        o.z = fmaf(p.z, s.x, o.z); o.z = fmaf(-p.w, s.y, o.z); o.z = fmaf(p.x, s.z, o.z); o.z = fmaf(p.y, s.w, o.z);
        o.w = fmaf(p.z, s.y, o.w); o.w = fmaf(p.w, s.x, o.w); o.w = fmaf(p.x, s.w, o.w); o.w = fmaf(-p.y, s.z, o.w);
      }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = r0 + tr + 16 * u, c = tc + 16 * v;
      if (r >= ld || c >= kb) continue;
      const float4 o = acc[u][v];
      va[r + (int64_t)c * ld] = make_float2(o.x, o.y);
      vb[r + (int64_t)c * ld] = make_float2(o.z, o.w);
    }
}

// Operand source of the tensor-core product (zq_tc32.cu) over a complex64 array.
static Tc32Src tsrc(const float2* p, int64_t ld, int kfast, int conj = 0, float sign = 1.f) {
  Tc32Src s{};
  s.p = reinterpret_cast<const float*>(p); s.ld = ld; s.kfast = kfast; s.conj = conj; s.sign = sign;
  return s;
}

// X = Q Phi in FP32, the blocks' W and V prepared together (big: fq_bytes of scratch)
static int form_q_batched(const float2* M, int64_t ldm, int n, float2* X, int64_t ldx, void* ws, void* big,
                          cudaStream_t st, int* tc_err) {
  const bool use_tc = tc_err && fp32_products_on_tensor_cores(TC_USE_FORMQ);      // C1 = V^H X (inner L)
  const bool use_tc_x = tc_err && fp32_products_on_tensor_cores(TC_USE_FORMQ_X);  // X -= W C1 (inner 64)
  FqBlocks q{};
  q.M = M; q.ldm = ldm; q.n = n; q.nref = n - 2; q.nblocks = ceil_div(n - 2, FQ_NB);
  q.W = reinterpret_cast<float2*>(big);
  q.V = q.W + fq_off(n, q.nblocks);
  q.T = reinterpret_cast<float4*>(q.V + fq_off(n, q.nblocks));
  q.part = q.T + (size_t)q.nblocks * FQ_NB * FQ_NB;
  {
    static std::atomic<unsigned long long> attr_set{0};  // per device
    int dev = 0;
    ZQ_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(attr_set.load() & bit)) {
      ZQ_CUDA(cudaFuncSetAttribute(k_fq_t, cudaFuncAttributeMaxDynamicSharedMemorySize, FQ_T_SMEM));
      ZQ_CUDA(cudaFuncSetAttribute(k_fq_v, cudaFuncAttributeMaxDynamicSharedMemorySize, FQ_V_SMEM));
      attr_set.fetch_or(bit);
    }
  }
  const int px = ceil_div(n * FQ_NB, 256 * 8);
  ZQ_CUDA(launch_pdl_smem(k_fq_pack, dim3(px, q.nblocks), dim3(256), 0, st, q));
  ZQ_LAUNCH_CHECK();
  ZQ_CUDA(launch_pdl_smem(k_fq_gram, dim3(fq_chunks(n, 0), q.nblocks), dim3(256), 0, st, q));
  ZQ_LAUNCH_CHECK();
  ZQ_CUDA(launch_pdl_smem(k_fq_t, dim3(q.nblocks), dim3(1024), FQ_T_SMEM, st, q));
  ZQ_LAUNCH_CHECK();
  ZQ_CUDA(launch_pdl_smem(k_fq_v, dim3(ceil_div(n, FQ_NB), q.nblocks), dim3(256), FQ_V_SMEM, st, q));
  ZQ_LAUNCH_CHECK();
  float2* C1 = reinterpret_cast<float2*>(ws);  // [C1e; C1o], 2 kb x L
  float2* Pk = C1 + (size_t)2 * FQ_NB * n;
  const int64_t pcap = fq_pcap(n, FQ_NB);
  const float2 one = make_float2(1.f, 0.f), zero = make_float2(0.f, 0.f), mone = make_float2(-1.f, 0.f);
  for (int b = q.nblocks - 1; b >= 0; --b) {
    const int pb = FQ_NB * b, kb = fq_kb(q.nref, b), ld = fq_ld(n, b), rows = n - pb, L = n - 1 - pb;
    const float2 *Wa = q.W + fq_off(n, b), *Wb = Wa + (int64_t)ld * kb;
    const float2 *Va = q.V + fq_off(n, b), *Vb = Va + (int64_t)ld * kb;
    // rows from pb (zero in W and V), columns from pb + 1
    float2* Xas = X + pb + (int64_t)(pb + 1) * ldx;
    float2* Xbs = Xas + n;
    float2 *C1e = C1, *C1o = C1 + kb;
    const int64_t ldc1 = 2 * kb;
    ZgemmArgsT<float> g{};
    g.P = Pk; g.pcap = pcap;
    // C1e = Va^H Xa_sub + Vb^H Xb_sub ; C1o = Va^T Xb_sub - Vb^T Xa_sub   (kb x L)
    if (use_tc) {
      // both halves in one tensor-core product, formed transposed so that the
      // long inner dimension is contiguous in X and V:
      //   [C1e; C1o]^T (L x 2kb) = [Xa_sub^T | Xb_sub^T] [[conj(Va), -Vb]; [conj(Vb), Va]]
      // stored as C1 = [C1e; C1o] (2kb x L, ld 2kb)
      Tc32Args t{};
      t.cplx = 1; t.m = L; t.n = 2 * kb; t.nseg = 2;
      t.seg[0].a = tsrc(Xas, ldx, 1);
      t.seg[0].b = tsrc(Va, ld, 1, 1);
      t.seg[0].b2 = tsrc(Vb, ld, 1, 0, -1.f);
      t.seg[0].nsplit = kb; t.seg[0].k = rows;
      t.seg[1].a = tsrc(Xbs, ldx, 1);
      t.seg[1].b = tsrc(Vb, ld, 1, 1);
      t.seg[1].b2 = tsrc(Va, ld, 1);
      t.seg[1].nsplit = kb; t.seg[1].k = rows;
      t.alpha = one; t.beta = zero;
      t.C = reinterpret_cast<float*>(C1); t.ldc = ldc1; t.ctrans = 1;
      // split K over enough CTAs to fill the GPU (partials in the split-K buffer)
      const int tiles = ceil_div(L, 128), kblk = 2 * ceil_div(rows, 16);
      int splits = 1;
      while (tiles * splits < 2 * 152 && kblk / (2 * splits) >= 4 && (int64_t)(2 * splits) * L * 2 * kb <= pcap) splits *= 2;
      // shorter accumulations in tensor memory, summed in FP32 by the reduce
      if (const int per = formq_kblocks_per_split())
        while (kblk / splits > per && (int64_t)(2 * splits) * L * 2 * kb <= pcap) splits *= 2;
      t.splits = splits;
      t.P = reinterpret_cast<float*>(Pk);
      t.err = tc_err;
      prof_begin(PC_FORMQ_GEMM, st);
      const int rc = tc32_gemm(t, st);
      prof_end(PC_FORMQ_GEMM, st);
      if (rc) return rc;
    } else {
      g.m = kb; g.n = L; g.k1 = rows; g.k2 = rows;
      g.A1 = Va; g.lda1 = ld; g.B1 = Xas; g.ldb1 = ldx;
      g.A2 = Vb; g.lda2 = ld; g.B2 = Xbs; g.ldb2 = ldx;
      g.s2 = 1.f; g.alpha = one; g.beta = zero;
      g.C = C1e; g.ldc = ldc1;
      if (int rc = zgemm(OP_C, OP_N, OP_C, OP_N, g, 1, st)) return rc;
      g.A1 = Va; g.B1 = Xbs; g.A2 = Vb; g.B2 = Xas; g.s2 = -1.f; g.C = C1o;
      if (int rc = zgemm(OP_T, OP_N, OP_T, OP_N, g, 1, st)) return rc;
    }
    // Xa_sub -= Wa C1e - conj(Wb) C1o ; Xb_sub -= Wb C1e + conj(Wa) C1o   (rows x L)
    if (use_tc_x) {
      Tc32Args t{};
      t.cplx = 1; t.m = rows; t.n = L; t.nseg = 4; t.halves = 2;
      for (int half = 0; half < 2; ++half) {
        Tc32Seg* sg = t.seg + 2 * half;
        sg[0].a = tsrc(half ? Wb : Wa, ld, 0);
        sg[0].b = tsrc(C1e, ldc1, 1);
        sg[0].k = kb;
        sg[1].a = tsrc(half ? Wa : Wb, ld, 0, 1, half ? 1.f : -1.f);
        sg[1].b = tsrc(C1o, ldc1, 1);
        sg[1].k = kb;
      }
      t.alpha = mone; t.beta = one;
      t.C = reinterpret_cast<float*>(Xas); t.ldc = ldx; t.chalf = 2 * (int64_t)n;
      t.splits = 1;
      t.err = tc_err;
      prof_begin(PC_FORMQ_GEMM, st);
      const int rc = tc32_gemm(t, st);
      prof_end(PC_FORMQ_GEMM, st);
      if (rc) return rc;
      continue;
    }
    g = ZgemmArgsT<float>{};
    g.P = Pk; g.pcap = pcap;
    g.m = rows; g.n = L; g.k1 = kb; g.k2 = kb;
    g.A1 = Wa; g.lda1 = ld; g.B1 = C1e; g.ldb1 = ldc1;
    g.A2 = Wb; g.lda2 = ld; g.B2 = C1o; g.ldb2 = ldc1;
    g.s2 = -1.f; g.alpha = mone; g.beta = one;
    g.C = Xas; g.ldc = ldx;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
    g.A1 = Wb; g.A2 = Wa; g.s2 = 1.f; g.C = Xbs;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
  }
  return ZQ_OK;
}

template <typename R>
int form_q(const cplx<R>* M, int64_t ldm, int n, const double* phi, cplx<R>* X, int64_t ldx, int nbq, void* ws,
           cudaStream_t st, int* tc_err, void* big, size_t big_bytes) {
  using Z = cplx<R>;
  using Args = ZgemmArgsT<R>;
  if (n <= 0) return ZQ_OK;
  ZQ_CUDA(launch_pdl_smem(k_init_x<Z>, dim3(ceil_div(2 * n * n, 256) > 4096 ? 4096 : ceil_div(2 * n * n, 256)), dim3(256), 0, st, X, ldx, n, phi));
  ZQ_LAUNCH_CHECK();
  const int nref = n - 2;  // reflectors exist for columns 0..n-3
  if (nref <= 0) return ZQ_OK;
  const int nblocks = ceil_div(nref, nbq);
  if constexpr (std::is_same<R, float>::value) {
    if (nbq == FQ_NB && fq_bytes(n, nblocks) <= big_bytes)
      return form_q_batched(M, ldm, n, X, ldx, ws, big, st, tc_err);
  }
  Z* p = reinterpret_cast<Z*>(ws);
  Z* Wa = p; p += (size_t)n * nbq;
  Z* Wb = p; p += (size_t)n * nbq;
  Z* G1 = p; p += (size_t)nbq * nbq;
  Z* G2 = p; p += (size_t)nbq * nbq;
  Z* Ta = p; p += (size_t)nbq * nbq;
  Z* Tb = p; p += (size_t)nbq * nbq;
  Z* C1e = p; p += (size_t)nbq * n;
  Z* C1o = p; p += (size_t)nbq * n;
  Z* C2e = p; p += (size_t)nbq * n;
  Z* C2o = p; p += (size_t)nbq * n;
  Z* Pk = p;
  const int64_t pcap = fq_pcap(n, nbq);
  Z one = czero<Z>(), zero = czero<Z>(), mone = czero<Z>();
  one.x = 1; mone.x = -1;
  for (int bi = nblocks - 1; bi >= 0; --bi) {
    const int pb = bi * nbq;
    const int kb = (nbq < nref - pb) ? nbq : (nref - pb);
    const int L = n - 1 - pb;
    ZQ_CUDA(launch_pdl_smem(k_pack_w<Z>, dim3(ceil_div(L * kb, 256) > 2048 ? 2048 : ceil_div(L * kb, 256)), dim3(256), 0, st, M, ldm, n, pb, kb, L, Wa, Wb));
    ZQ_LAUNCH_CHECK();
    // G1 = Wa^H Wa + Wb^H Wb ; G2 = Wa^T Wb - Wb^T Wa   (kb x kb, inner L)
    Args g{};
    g.P = Pk; g.pcap = pcap;
    g.m = kb; g.n = kb; g.k1 = L; g.k2 = L;
    g.A1 = Wa; g.lda1 = L; g.B1 = Wa; g.ldb1 = L;
    g.A2 = Wb; g.lda2 = L; g.B2 = Wb; g.ldb2 = L;
    g.s2 = (R)1; g.alpha = one; g.beta = zero;
    g.C = G1; g.ldc = kb;
    if (int rc = zgemm(OP_C, OP_N, OP_C, OP_N, g, 1, st)) return rc;
    g.A1 = Wa; g.B1 = Wb; g.A2 = Wb; g.B2 = Wa; g.s2 = (R)-1; g.C = G2;
    if (int rc = zgemm(OP_T, OP_N, OP_T, OP_N, g, 1, st)) return rc;
    ZQ_CUDA(launch_pdl_smem(k_build_t<Z>, dim3(1), dim3(1024), 0, st, G1, G2, kb, Ta, Tb));
    ZQ_LAUNCH_CHECK();
    // C1e = Wa^H Xa_sub + Wb^H Xb_sub ; C1o = Wa^T Xb_sub - Wb^T Xa_sub   (kb x L)
    Z* Xas = X + (pb + 1) + (int64_t)(pb + 1) * ldx;
    Z* Xbs = Xas + n;
    g = Args{};
    g.P = Pk; g.pcap = pcap;
    g.m = kb; g.n = L; g.k1 = L; g.k2 = L;
    g.A1 = Wa; g.lda1 = L; g.B1 = Xas; g.ldb1 = ldx;
    g.A2 = Wb; g.lda2 = L; g.B2 = Xbs; g.ldb2 = ldx;
    g.s2 = (R)1; g.alpha = one; g.beta = zero;
    g.C = C1e; g.ldc = kb;
    if (int rc = zgemm(OP_C, OP_N, OP_C, OP_N, g, 1, st)) return rc;
    g.A1 = Wa; g.B1 = Xbs; g.A2 = Wb; g.B2 = Xas; g.s2 = (R)-1; g.C = C1o;
    if (int rc = zgemm(OP_T, OP_N, OP_T, OP_N, g, 1, st)) return rc;
    // C2e = Ta C1e - conj(Tb) C1o ; C2o = Tb C1e + conj(Ta) C1o   (kb x L)
    g = Args{};
    g.P = Pk; g.pcap = pcap;
    g.m = kb; g.n = L; g.k1 = kb; g.k2 = kb;
    g.A1 = Ta; g.lda1 = kb; g.B1 = C1e; g.ldb1 = kb;
    g.A2 = Tb; g.lda2 = kb; g.B2 = C1o; g.ldb2 = kb;
    g.s2 = (R)-1; g.alpha = one; g.beta = zero;
    g.C = C2e; g.ldc = kb;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
    g.A1 = Tb; g.A2 = Ta; g.s2 = (R)1; g.C = C2o;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
    // Xa_sub -= Wa C2e - conj(Wb) C2o ; Xb_sub -= Wb C2e + conj(Wa) C2o   (L x L)
    g = Args{};
    g.P = Pk; g.pcap = pcap;
    g.m = L; g.n = L; g.k1 = kb; g.k2 = kb;
    g.A1 = Wa; g.lda1 = L; g.B1 = C2e; g.ldb1 = kb;
    g.A2 = Wb; g.lda2 = L; g.B2 = C2o; g.ldb2 = kb;
    g.s2 = (R)-1; g.alpha = mone; g.beta = one;
    g.C = Xas; g.ldc = ldx;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
    g.A1 = Wb; g.A2 = Wa; g.s2 = (R)1; g.C = Xbs;
    if (int rc = zgemm(OP_N, OP_N, OP_R, OP_N, g, 1, st)) return rc;
  }
  return ZQ_OK;
}

template <typename R>
int apply_z(const cplx<R>* X, int64_t ldx, const R* Z, int64_t ldz, int n, cplx<R>* out, int64_t ldo,
            DgemmDescT<R>* dev_desc, cudaStream_t st, int* tc_err) {
  if (n <= 0) return ZQ_OK;
  if constexpr (std::is_same<R, float>::value) {
    if (tc_err && fp32_products_on_tensor_cores(TC_USE_APPLYZ)) {
      // one real product on the tensor cores: (4n x n) real view of X times Z
      Tc32Args t{};
      t.cplx = 0; t.m = 4 * n; t.n = n; t.nseg = 1;
      t.seg[0].a.p = reinterpret_cast<const float*>(X); t.seg[0].a.ld = 2 * ldx; t.seg[0].a.kfast = 0;
      t.seg[0].a.sign = 1.f;
      t.seg[0].b.p = Z; t.seg[0].b.ld = ldz; t.seg[0].b.kfast = 1; t.seg[0].b.sign = 1.f;
      t.seg[0].k = n;
      t.alpha = make_float2(1.f, 0.f); t.beta = make_float2(0.f, 0.f);
      t.C = reinterpret_cast<float*>(out); t.ldc = 2 * ldo;
      t.splits = 1;
      t.err = tc_err;
      prof_begin(PC_APPLYZ, st);
      const int rc = tc32_gemm(t, st);
      prof_end(PC_APPLYZ, st);
      return rc;
    }
  }
  DgemmDescT<R> d{};
  d.A = reinterpret_cast<const R*>(X); d.lda = 2 * ldx;
  d.B = Z; d.ldb = ldz;
  d.C = reinterpret_cast<R*>(out); d.ldc = 2 * ldo;
  d.m = 4 * n; d.n = n; d.k = n;
  d.alpha = 1; d.beta = 0;
  prof_begin(PC_APPLYZ, st);
  const int rc = dgemm_grouped<R>(&d, 1, dev_desc, st);
  prof_end(PC_APPLYZ, st);
  return rc;
}

template int form_q<double>(const cplx<double>*, int64_t, int, const double*, cplx<double>*, int64_t, int, void*, cudaStream_t, int*, void*, size_t);
template int form_q<float>(const cplx<float>*, int64_t, int, const double*, cplx<float>*, int64_t, int, void*, cudaStream_t, int*, void*, size_t);
template int apply_z<double>(const cplx<double>*, int64_t, const double*, int64_t, int, cplx<double>*, int64_t, DgemmDescT<double>*, cudaStream_t, int*);
template int apply_z<float>(const cplx<float>*, int64_t, const float*, int64_t, int, cplx<float>*, int64_t, DgemmDescT<float>*, cudaStream_t, int*);

__global__ void k_symfill(double2* D, int64_t ld, int n) {
  pdl_wait();
  const int64_t total = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(t % n), i = (int)(t / n);
    const double2 u = D[j + (int64_t)i * ld];
    const double2 v = D[n + j + (int64_t)i * ld];
    D[j + (int64_t)(n + i) * ld] = make_double2(-v.x, v.y);      // -conj(V)
    D[n + j + (int64_t)(n + i) * ld] = make_double2(u.x, -u.y);  // conj(U)
  }
}

int symmetry_fill(double2* D, int64_t ld, int n, cudaStream_t st) {
  if (n <= 0) return ZQ_OK;
  const int64_t total = (int64_t)n * n;
  const int blocks = (int)((total + 255) / 256 > 8192 ? 8192 : (total + 255) / 256);
  ZQ_CUDA(launch_pdl_smem(k_symfill, dim3(blocks), dim3(256), 0, st, D, ld, n));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

}  // namespace zq
