// FP64-accurate matrix products from integer residues on the 5th-generation
// tensor cores (the Ozaki scheme II: Ozaki, Uchino, Imamura, "Ozaki Scheme II:
// A GEMM-oriented emulation of floating-point matrix multiplication using an
// integer modular technique", 2025; here with bf16 residues and FP32
// accumulation).
//
//   * Every row of A (column of B) is scaled by a power of two above its
//     largest entry and rounded to integers of `bits` bits (55 for complex FP64
//     products, 60 for real ones).
//   * For each of L pairwise coprime moduli p <= 253 the integers are reduced to
//     symmetric residues, |r| <= 127: exact in bf16, products below 2^14, so
//     sums of 512 are exact in FP32; they are emptied into int32 and reduced
//     mod p.
//   * The product's integers (below P / 2, P the product of the moduli) follow
//     from their residues: X / P = frac(sum_l r_l c_l), c_l = inv_l / p_l in
//     96-bit fixed point, where the wrap-around of the integer sum is the frac.
//   * A complex product takes three real ones (re re, im im, (re + im)(re + im)):
//     residues of the sums are reduced again, so nothing is lost by the
//     subtraction, which happens in the fixed-point sums.
//
// Why: slicing into 7-bit digits (zq_ozaki.cu) takes 36 digit products of four
// real products each for the same accuracy; 16 moduli of three take a third of
// the tensor work (24 of 60 for the 35-bit step: 11 moduli). And every modulus
// is an independent product over the same tiles, so small matrices fill the
// GPU, where one CTA pair per tile ran all digit products in turn. Measured
// before and after: 8192 x 4096 x 4096 complex 28.9 -> 13.0 ms (k_crt_mma 7.5 ms,
// 1770 TFLOP/s executed; splitting 1.4, joining 1.2), 1500 x 1100 x 3000 1.61 ->
// 0.74 ms, 300 x 300 x 300 products of a solve 0.26 -> 0.10 ms each.
//
// k_crt_mma is persistent: each pair of CTAs (cta_group::2, 256 x 256 output
// tiles) takes jobs (modulus and product, tile); the roles of k_oz_umma's pairs
// (TMA producer, MMA issuer, eight drain warps; 6 stages of 32 KB, two TMEM
// accumulators) run through the jobs without draining the pipeline between
// them. All waits are bounded (zq_umma.cuh).
#include "zq_common.cuh"
#include "zq_crt.h"
#include "zq_umma.cuh"

#include <atomic>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <type_traits>

namespace zq {
namespace {

constexpr int CRT_MAX = 18;
constexpr int CRT_P[CRT_MAX] = {253, 251, 250, 249, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181};
// log2 of the product of the first l moduli, rounded down to 1/100
constexpr double CRT_LOG2[CRT_MAX + 1] = {0,     7.98,  15.95, 23.91, 31.87, 39.82, 47.73, 55.63, 63.50, 71.34,
                                          79.16, 86.96, 94.72, 102.45, 110.08, 117.70, 125.30, 132.87, 140.37};

constexpr int CB_M = 256, CB_N = 256, CB_K = 64;
constexpr int CB_CH = 512;            // K terms per exact FP32 accumulation
constexpr int CB_STAGES = 6;
constexpr uint32_t CB_HALF = 128 * CB_K * 2;   // one operand's 128 rows of a stage
constexpr uint32_t CB_STAGE = 2 * CB_HALF;
constexpr int CB_THREADS = 320;
constexpr int CB_SMEM = 1024 + CB_STAGES * CB_STAGE + 256 + 16384;  // slack: see UM_SMEM (zq_ozaki_umma.cu)
constexpr int CB_GROUP = 8;           // row tiles per group of the job order

// per modulus: 2^14, 2^28, 2^42, 2^56 mod p (symmetric), p, 1/p
struct CrtMod { float c1, c2, c3, c4, p, ip; };
struct CrtMods { CrtMod v[CRT_MAX]; };

constexpr int crt_sym(long long v, int p) {
  long long r = v % p;
  if (r > p / 2) r -= p;
  return (int)r;
}
constexpr CrtMods crt_mods() {
  CrtMods m{};
  for (int l = 0; l < CRT_MAX; ++l) {
    const int p = CRT_P[l];
    m.v[l].c1 = (float)crt_sym(1ll << 14, p);
    m.v[l].c2 = (float)crt_sym(1ll << 28, p);
    m.v[l].c3 = (float)crt_sym(1ll << 42, p);
    m.v[l].c4 = (float)crt_sym(1ll << 56, p);
    m.v[l].p = (float)p;
    m.v[l].ip = 1.0f / (float)p;
  }
  return m;
}
__constant__ CrtMods g_crt_mods = crt_mods();

// ------------------------------------------------------------------ residues
__device__ __forceinline__ float crt_rint(float v) { return __fadd_rn(__fadd_rn(v, 12582912.f), -12582912.f); }

// v 2^(bits - e) rounded to an integer, as four (56 bits) or five 14-bit limbs with its sign
template <int NL>
__device__ __forceinline__ void crt_limbs(double v, int e, int bits, float (&f)[NL]) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned neg = (unsigned)(b >> 32) & 0x80000000u;
  const int ex = (int)((b >> 52) & 0x7ff);
  unsigned long long mant = b & ((1ull << 52) - 1);
  if (ex != 0) mant |= 1ull << 52;
  const int sh = (ex == 0 ? 1 : ex) - 1075 - e + bits;
  unsigned long long V = 0;
  if (e > -1000 && mant != 0) {
    if (sh >= 0) V = sh < 11 ? mant << sh : 0;
    else if (sh > -55) V = (mant + (1ull << (-sh - 1))) >> (-sh);
  }
#pragma unroll
  for (int q = 0; q < NL; ++q)  // 0x4B000000 | d is 2^23 + d
    f[q] = __uint_as_float(__float_as_uint(__uint_as_float(0x4B000000u | ((unsigned)(V >> (14 * q)) & 0x3fffu)) - 8388608.f) ^ neg);
}
// symmetric residue of the limbs' integer (all steps exact: the sum is below 2^23, the
// fifth limb of 60 bits below 2^4)
template <int NL>
__device__ __forceinline__ float crt_residue(const float (&f)[NL], const CrtMod& m) {
  float x = fmaf(f[3], m.c3, fmaf(f[2], m.c2, fmaf(f[1], m.c1, f[0])));
  if constexpr (NL > 4) x = fmaf(f[4], m.c4, x);
  return fmaf(-crt_rint(x * m.ip), m.p, x);
}
__device__ __forceinline__ unsigned crt_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&v);
}

// Block: 32 operand rows x 64 K. The tile is read along whichever index is
// contiguous in memory and exchanged through shared memory; thread (row, 8 k)
// then writes 16 bytes per residue, 128 contiguous bytes per row. Three blocks an SM
// (signs kept in the limbs: 80 registers instead of 126) bring 1500 x 3000 entries to
// 48 planes in 121 us, 5.4 TB/s (two: 133 us); packed FP32 arithmetic, half the issue
// slots, or 8 x 256 tiles, 512 contiguous bytes, are no faster.
template <bool CPLX>
__global__ void __launch_bounds__(256, 3) k_crt_split(CrtSide s, bool is_a, int count, int count_pad, int Kp,
                                                   const int* __restrict__ exps, int bits, int moduli,
                                                   __nv_bfloat16* __restrict__ out) {
  pdl_wait();
  using E = typename std::conditional<CPLX, double2, double>::type;
  __shared__ E tile[32][65];  // padded: a column of the tile is read and written without conflicts too
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 64;
  auto element = [&](int idx, int k) {
    E v{};
    if (idx >= count) return v;
    const bool two = k >= s.K1;
    if (two) k -= s.K1;
    if (k >= (two ? s.K2 : s.K1)) return v;
    const int op = two ? s.op2 : s.op1;
    const int64_t ld = two ? s.ld2 : s.ld1;
    const E* X = reinterpret_cast<const E*>(two ? s.X2 : s.X1);
    const bool col = (op == OP_N || op == OP_R) == is_a;  // idx runs along a column of X
    v = __ldg(X + (col ? idx + (int64_t)k * ld : k + (int64_t)idx * ld));
    if constexpr (CPLX) {
      if (op == OP_R || op == OP_C) v.y = -v.y;
      if (two && is_a) { v.x *= s.s2; v.y *= s.s2; }
    }
    return v;
  };
  // position of (row, k) in the tile: the k within a group of eight is
  // exchanged with the group's number, so that both accesses avoid conflicts
  auto pos = [](int k) { return (k & 56) | ((k ^ (k >> 3)) & 7); };
  if ((s.op1 == OP_N || s.op1 == OP_R) == is_a) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = warp + 8 * u;
      tile[lane][pos(k)] = element(i0 + lane, k0 + k);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int r = warp + 8 * (u >> 1), k = lane + 32 * (u & 1);
      tile[r][pos(k)] = element(i0 + r, k0 + k);
    }
  }
  __syncthreads();
  const int g = lane & 7, r = warp * 4 + (lane >> 3);
  const int idx = i0 + r;
  const int e = idx < count ? exps[idx] : -1100;
  constexpr int NL = CPLX ? 4 : 5;  // complex products of up to 55 bits, real ones of 60
  float fr[8][NL], fi[CPLX ? 8 : 1][NL];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const E v = tile[r][8 * g + (u ^ g)];
    if constexpr (CPLX) {
      crt_limbs(v.x, e, bits, fr[u]);
      crt_limbs(v.y, e, bits, fi[u]);
    } else {
      crt_limbs(v, e, bits, fr[u]);
    }
  }
  const int64_t stride = (int64_t)count_pad * Kp;
  __nv_bfloat16* o = out + (int64_t)idx * Kp + k0 + 8 * g;
  for (int l = 0; l < moduli; ++l) {
    const CrtMod m = g_crt_mods.v[l];
    unsigned pr[4], pi[4], ps[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float a0 = crt_residue(fr[2 * h], m), a1 = crt_residue(fr[2 * h + 1], m);
      pr[h] = crt_pack(a0, a1);
      if constexpr (CPLX) {
        const float b0 = crt_residue(fi[2 * h], m), b1 = crt_residue(fi[2 * h + 1], m);
        pi[h] = crt_pack(b0, b1);
        const float s0 = a0 + b0, s1 = a1 + b1;
        ps[h] = crt_pack(fmaf(-crt_rint(s0 * m.ip), m.p, s0), fmaf(-crt_rint(s1 * m.ip), m.p, s1));
      }
    }
    *reinterpret_cast<uint4*>(o) = make_uint4(pr[0], pr[1], pr[2], pr[3]);
    o += stride;
    if constexpr (CPLX) {
      *reinterpret_cast<uint4*>(o) = make_uint4(pi[0], pi[1], pi[2], pi[3]);
      o += stride;
      *reinterpret_cast<uint4*>(o) = make_uint4(ps[0], ps[1], ps[2], ps[3]);
      o += stride;
    }
  }
}

// exponents (2^e above the largest magnitude) of a real operand's rows (A) or columns (B);
// CRT_NOT_FINITE where one of the values is Inf or NaN, which residues cannot carry: the
// product's row or column is then NaN (k_crt_join)
constexpr int CRT_NOT_FINITE = 5000;
__device__ __forceinline__ int crt_exponent(unsigned long long mb) {
  if (mb >= (0x7ffull << 52)) return CRT_NOT_FINITE;
  int e;
  frexp(bits_to_double(mb), &e);
  return e;
}
__global__ void k_crt_exp_init(int* e, int n) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] = -1100;
}
__global__ void __launch_bounds__(256) k_crt_exp_real(const double* __restrict__ X, int64_t ld, int count, int K, bool is_a,
                                                      int* __restrict__ exps) {
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long mb = 0;
  if (is_a) {  // rows: 32 per block column, 256 columns per block row
    const int r = blockIdx.x * 32 + lane;
    const int kend = min(K, (int)(blockIdx.y + 1) * 256);
    if (r < count)
      for (int k = blockIdx.y * 256 + warp; k < kend; k += 8) mb = max(mb, abs_bits(__ldg(X + r + (int64_t)k * ld)));
    __shared__ unsigned long long s[8][32];
    s[warp][lane] = mb;
    __syncthreads();
    if (warp == 0 && r < count) {
#pragma unroll
      for (int w = 1; w < 8; ++w) mb = max(mb, s[w][lane]);
      if (mb) atomicMax(exps + r, crt_exponent(mb));
    }
  } else {     // columns: one warp each
    const int c = blockIdx.x * 8 + warp;
    if (c >= count) return;
#pragma unroll 4
    for (int k = lane; k < K; k += 32) mb = max(mb, abs_bits(__ldg(X + k + (int64_t)c * ld)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    if (lane == 0 && mb) exps[c] = crt_exponent(mb);
  }
}

// ------------------------------------------------------------------ products
struct CrtMma {
  int mp, np, Kp, tm, tn, tiles, jobs, prods, lower;
  uint8_t* R;
  int* err;
  long long wait;
};

__device__ __forceinline__ void crt_job(const CrtMma& g, int job, int& z, int& bi, int& bj) {
  z = job / g.tiles;
  const int t = job - z * g.tiles;
  if (g.lower) { tri_tile(t, bi, bj); return; }
  const int per = CB_GROUP * g.tn, grp = t / per, first = grp * CB_GROUP;
  const int gm = (g.tm - first) < CB_GROUP ? (g.tm - first) : CB_GROUP;
  bi = first + (t % per) % gm;
  bj = (t % per) / gm;
}
// v mod p in [0, p), |v| < 2^30: the float quotient is at most one off
__device__ __forceinline__ int crt_mod(int v, int p, float ip) {
  int r = v - __float2int_rd((float)v * ip) * p;
  if (r < 0) r += p;
  if (r >= p) r -= p;
  return r;
}

__global__ void __launch_bounds__(CB_THREADS, 1)
    k_crt_mma(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const CrtMma g) {
  pdl_wait();
  extern __shared__ __align__(1024) unsigned char cb_raw[];
  const uint32_t raw = su32(cb_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  uint64_t* bars = reinterpret_cast<uint64_t*>(cb_raw + (ring - raw) + CB_STAGES * CB_STAGE);
  const uint32_t full0 = su32(bars), empty0 = full0 + 8 * CB_STAGES, accf0 = empty0 + 8 * CB_STAGES, acce0 = accf0 + 16,
                 done_bar = acce0 + 16;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  if (threadIdx.x == 0) {
    for (int s = 0; s < CB_STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accf0 + 8 * b, 1); mbar_init(acce0 + 8 * b, 16); }
    mbar_init(done_bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync();  // the peer's barriers are initialised before any remote arrival
  const uint32_t tmem = s_tmem;
  volatile int* abort = &s_abort;
  const int first = (int)(blockIdx.x >> 1), step = (int)(gridDim.x >> 1);
  const int Kp = g.Kp;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int ks = 0;
      bool ok = true;
      const uint32_t full_lead = mapa_shared(full0, 0);
      for (int job = first; job < g.jobs && ok; job += step) {
        int z, bi, bj;
        crt_job(g, job, z, bi, bj);
        const int ya = z * g.mp + bi * CB_M + (int)rank * 128, yb = z * g.np + bj * CB_N + (int)rank * 128;
        for (int k = 0; k < Kp; k += CB_K) {
          const int stage = ks % CB_STAGES, round = ks / CB_STAGES;
          if (!mbar_wait(empty0 + 8 * stage, (round & 1) ^ 1, abort, g.wait)) { ok = false; break; }
          const uint32_t sA = ring + stage * CB_STAGE;
          if (rank == 0) mbar_expect_tx(full0 + 8 * stage, 2 * CB_STAGE);
          tma_2d_pair(sA, &tmA, k, ya, full_lead + 8 * stage);
          tma_2d_pair(sA + CB_HALF, &tmB, k, yb, full_lead + 8 * stage);
          ++ks;
        }
      }
      // copies in flight finish before the CTA may exit (rank 1 is held at the
      // final cluster barrier until rank 0, which has the full barriers, is done;
      // after an abort abort_hold covers what the peer alone issued)
      if (rank == 0)
        for (int q = (ks > CB_STAGES ? ks - CB_STAGES : 0); q < ks; ++q)
          mbar_drain(full0 + 8 * (q % CB_STAGES), (q / CB_STAGES) & 1, 2000000LL);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0 && rank == 0) {
      int ks = 0, ci = 0;
      bool ok = true;
      for (int job = first; job < g.jobs && ok; job += step) {
        for (int cb = 0; cb < Kp && ok; cb += CB_CH) {
          const int ce = cb + CB_CH < Kp ? cb + CB_CH : Kp;
          const int buf = ci & 1;
          if (!mbar_wait(acce0 + 8 * buf, ((ci >> 1) & 1) ^ 1, abort, g.wait)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(buf * 256);
          for (int k = cb; k < ce; k += CB_K) {
            const int stage = ks % CB_STAGES, round = ks / CB_STAGES;
            if (!mbar_wait(full0 + 8 * stage, round & 1, abort, g.wait)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sA = ring + stage * CB_STAGE;
            const uint64_t ad = sw128_desc(sA), bd = sw128_desc(sA + CB_HALF);
#pragma unroll
            for (int q = 0; q < CB_K / 16; ++q)
              umma_bf16_pair(d, ad + 2 * q, bd + 2 * q, (k != cb || q > 0) ? 1u : 0u);
            umma_commit_pair_mc(empty0 + 8 * stage, (uint16_t)3);
            ++ks;
          }
          if (!ok) break;
          umma_commit_pair_mc(accf0 + 8 * buf, (uint16_t)3);
          ++ci;
        }
      }
      umma_commit_pair_mc(done_bar, (uint16_t)1);
      mbar_drain(done_bar, 0);
    }
  } else {
    // ------------------------------------------------------------ drain
    const int q = warp & 3;         // TMEM lane quarter this warp may access
    const int h = (warp - 2) >> 2;  // column half
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(128 * h);
    const uint32_t acce_lead = mapa_shared(acce0, 0);
    int v[128];
#pragma unroll
    for (int c = 0; c < 128; ++c) v[c] = 0;
    int ci = 0;
    bool ok = true;
    for (int job = first; job < g.jobs && ok; job += step) {
      int z, bi, bj;
      crt_job(g, job, z, bi, bj);
      const float pf = g_crt_mods.v[z / g.prods].p, ip = g_crt_mods.v[z / g.prods].ip;
      const int p = (int)pf;
      int nch = 0;
      for (int cb = 0; cb < Kp; cb += CB_CH) {
        const int buf = ci & 1;
        // warp-uniform outcome: the TMEM loads below are .sync.aligned
        const bool got = mbar_wait(accf0 + 8 * buf, (ci >> 1) & 1, abort, g.wait);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int gq = 0; gq < 8; ++gq) {
          uint32_t t[16];
          tmem_ld16(lane_base + (uint32_t)(buf * 256 + 16 * gq), t);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 16; ++c) v[16 * gq + c] += __float2int_rz(__uint_as_float(t[c]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank != 0) mbar_arrive_remote(acce_lead + 8 * buf);
          else mbar_arrive(acce0 + 8 * buf);
        }
        ++ci;
        if (++nch == 64) {  // 64 x 512 products stay below 2^29
          nch = 0;
#pragma unroll
          for (int c = 0; c < 128; ++c) v[c] = crt_mod(v[c], p, ip);
        }
      }
      if (!ok) break;
      uint8_t* o = g.R + ((int64_t)z * g.np + bj * CB_N + 128 * h) * g.mp + bi * CB_M + (int)rank * 128 + 32 * q + lane;
#pragma unroll
      for (int c = 0; c < 128; ++c) {
        o[(int64_t)c * g.mp] = (uint8_t)crt_mod(v[c], p, ip);
        v[c] = 0;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (s_abort) abort_hold();
  cluster_sync();  // both CTAs' MMAs and drains are finished before the collective release
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (threadIdx.x == 0 && s_abort) atomicExch(g.err, 1);
  cluster_sync();
}

// ------------------------------------------------------------ reconstruction
struct CrtJoin {
  uint32_t c[CRT_MAX][3];  // inv_l / p_l in 96-bit fixed point, low word first
  double pm;               // P = pm 2^pe, pm in [1, 2)
  int pe;
};

// the double nearest to (d / 2^96) P 2^E for a 96-bit two's complement d given
// by three 64-bit limbs of weight 2^0, 2^32, 2^64
__device__ __forceinline__ double crt_value(long long d0, long long d1, long long d2, double pm, int E) {
  uint32_t w0 = (uint32_t)d0;
  d1 += d0 >> 32;
  uint32_t w1 = (uint32_t)d1;
  d2 += d1 >> 32;
  uint32_t w2 = (uint32_t)d2;
  const unsigned neg = w2 >> 31;
  if (neg) {
    w0 = ~w0; w1 = ~w1; w2 = ~w2;
    if (++w0 == 0 && ++w1 == 0) ++w2;
  }
  const unsigned long long hi = ((unsigned long long)w2 << 32) | w1;
  if (hi == 0 && w0 == 0) return 0.0;
  const int lz = hi ? __clzll((long long)hi) : 64 + __clz((int)w0);
  unsigned long long m;
  if (lz >= 32) m = (lz < 64 ? hi << lz : 0ull) | ((unsigned long long)w0 << (lz - 32));
  else m = lz ? (hi << lz) | ((unsigned long long)w0 >> (32 - lz)) : hi;
  // m / 2^63 in [1, 2), rounded to 53 bits
  const unsigned long long y = (0x3feull << 52) + (m >> 11) + ((m >> 10) & 1ull);
  const double t = __longlong_as_double((long long)y) * pm;  // [1, 4]
  const int be = (int)((unsigned long long)__double_as_longlong(t) >> 52) + E - lz - 1;
  double v;
  if (be >= 1 && be <= 2046)
    v = __longlong_as_double(__double_as_longlong(t) + ((long long)(E - lz - 1) << 52));
  else
    v = scalbn(t, E - lz - 1);
  return neg ? -v : v;
}

template <bool CPLX>
__global__ void __launch_bounds__(256) k_crt_join(const uint8_t* __restrict__ R, int mp, int np, int moduli, CrtJoin cj,
                                                  int m, int n, int bits, const int* __restrict__ ea,
                                                  const int* __restrict__ eb, int lower, double* __restrict__ C,
                                                  int64_t ldc) {
  pdl_wait();
  constexpr int PR = CPLX ? 3 : 1;
  const int m4 = (m + 3) / 4;
  const int64_t total = (int64_t)m4 * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int r0 = 4 * (int)(t % m4), col = (int)(t / m4);
    if (lower && (r0 >> 8) < (col >> 8)) continue;  // tiles that were not computed
    unsigned long long acc[4][PR][3];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < PR; ++q) acc[i][q][0] = acc[i][q][1] = acc[i][q][2] = 0;
    const uint8_t* p = R + (int64_t)col * mp + r0;
    const int64_t zs = (int64_t)np * mp;
#pragma unroll 2
    for (int l = 0; l < moduli; ++l) {
      uint32_t w[PR];
#pragma unroll
      for (int q = 0; q < PR; ++q) { w[q] = __ldg(reinterpret_cast<const uint32_t*>(p)); p += zs; }
      const uint32_t c0 = cj.c[l][0], c1 = cj.c[l][1], c2 = cj.c[l][2];
#pragma unroll
      for (int q = 0; q < PR; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t b = (w[q] >> (8 * i)) & 255u;
          acc[i][q][0] += (unsigned long long)b * c0;
          acc[i][q][1] += (unsigned long long)b * c1;
          acc[i][q][2] += (unsigned long long)b * c2;
        }
    }
    const int e_col = eb[col];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r0 + i;
      if (row >= m) break;
      const int E = cj.pe + ea[row] + e_col - 2 * bits;
      long long d[PR][3];
#pragma unroll
      for (int q = 0; q < PR; ++q)
#pragma unroll
        for (int u = 0; u < 3; ++u) d[q][u] = (long long)acc[i][q][u];
      if constexpr (CPLX) {
        const double re = crt_value(d[0][0] - d[1][0], d[0][1] - d[1][1], d[0][2] - d[1][2], cj.pm, E);
        const double im = crt_value(d[2][0] - d[0][0] - d[1][0], d[2][1] - d[0][1] - d[1][1],
                                    d[2][2] - d[0][2] - d[1][2], cj.pm, E);
        reinterpret_cast<double2*>(C)[row + (int64_t)col * ldc] = make_double2(re, im);
      } else {
        const bool finite = ea[row] != CRT_NOT_FINITE && e_col != CRT_NOT_FINITE;
        C[row + (int64_t)col * ldc] = finite ? crt_value(d[0][0], d[0][1], d[0][2], cj.pm, E)
                                             : __longlong_as_double(0x7ff8000000000000ll);
      }
    }
  }
}

// constants of the reconstruction from the first L moduli
CrtJoin crt_constants(int L) {
  CrtJoin j{};
  uint32_t P[6] = {1, 0, 0, 0, 0, 0};  // product of the moduli
  for (int l = 0; l < L; ++l) {
    unsigned long long carry = 0;
    for (uint32_t& w : P) { carry += (unsigned long long)w * CRT_P[l]; w = (uint32_t)carry; carry >>= 32; }
  }
  int top = 5;
  while (P[top] == 0) --top;
  // the product's 64 leading bits
  const unsigned long long hi = ((unsigned long long)P[top] << 32) | (top > 0 ? P[top - 1] : 0u);
  const int lz = __builtin_clzll(hi);
  unsigned long long lead = hi << lz;
  if (lz && top > 1) lead |= (unsigned long long)P[top - 2] >> (32 - lz);
  j.pm = (double)(lead >> 11) / 4503599627370496.0;
  j.pe = 32 * (top + 1) - 1 - lz;
  for (int l = 0; l < L; ++l) {
    const int p = CRT_P[l];
    int r = 1;  // P / p_l mod p_l
    for (int q = 0; q < L; ++q)
      if (q != l) r = r * (CRT_P[q] % p) % p;
    int inv = 1;
    while (r * inv % p != 1) ++inv;
    // 2^96 inv / p by long division
    unsigned long long rem = (unsigned long long)inv;
    for (int w = 2; w >= 0; --w) {
      rem <<= 32;
      j.c[l][w] = (uint32_t)(rem / p);
      rem %= p;
    }
  }
  return j;
}

int rup(int a, int b) { return (a + b - 1) / b * b; }

int crt_map(CUtensorMap* tm, const void* base, int64_t Kp, int64_t rows) {
  auto enc = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tensor_map_encode_fn());
  if (!enc) { set_error_message("cuTensorMapEncodeTiled unavailable"); return ZQ_ERR_CUDA; }
  cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Kp * 2};
  cuuint32_t box[2] = {(cuuint32_t)CB_K, 128u};
  cuuint32_t es[2] = {1u, 1u};
  const CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error_message("cuTensorMapEncodeTiled failed"); return ZQ_ERR_CUDA; }
  return ZQ_OK;
}

}  // namespace

int crt_moduli(int bits, double terms) {
  int lg = 0;
  while ((double)(1ll << lg) < terms) ++lg;
  for (int l = 1; l <= CRT_MAX; ++l)
    if (CRT_LOG2[l] >= 2 * bits + lg + 1) return l;
  return 0;
}

CrtShape crt_shape(int m, int n, int K, int moduli, bool cplx) {
  CrtShape s{};
  s.mp = rup(m, CB_M); s.np = rup(n, CB_N); s.Kp = rup(K, CB_K);
  s.moduli = moduli; s.prods = cplx ? 3 : 1;
  const size_t z = (size_t)moduli * s.prods;
  s.a_bytes = z * s.mp * s.Kp * 2;
  s.b_bytes = z * s.np * s.Kp * 2;
  s.r_bytes = z * s.mp * s.np;
  return s;
}

int crt_split(const CrtSide& s, bool is_a, int count, int count_pad, int Kp, const int* exps, int bits, int moduli,
              void* out, cudaStream_t st) {
  ZQ_CUDA(launch_pdl_smem(k_crt_split<true>, dim3((unsigned)(count_pad / 32), (unsigned)(Kp / 64)), dim3(256), 0, st, s, is_a, count, count_pad, Kp, exps, bits, moduli, reinterpret_cast<__nv_bfloat16*>(out)));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int crt_multiply(const CrtShape& sh, const void* a, const void* b, void* r, bool lower, int* err, cudaStream_t st) {
  const int Z = sh.moduli * sh.prods;
  CUtensorMap ta, tb;
  if (int rc = crt_map(&ta, a, sh.Kp, (int64_t)Z * sh.mp)) return rc;
  if (int rc = crt_map(&tb, b, sh.Kp, (int64_t)Z * sh.np)) return rc;
  static std::atomic<int> sms[64];
  int dev = 0;
  ZQ_CUDA(cudaGetDevice(&dev));
  int count = sms[dev & 63].load();
  if (count == 0) {
    ZQ_CUDA(cudaFuncSetAttribute(k_crt_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, CB_SMEM));
    ZQ_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
    sms[dev & 63].store(count);
  }
  CrtMma g{};
  g.mp = sh.mp; g.np = sh.np; g.Kp = sh.Kp;
  g.tm = sh.mp / CB_M; g.tn = sh.np / CB_N;
  g.lower = lower ? 1 : 0;
  g.tiles = lower ? g.tm * (g.tm + 1) / 2 : g.tm * g.tn;
  g.prods = sh.prods;
  g.jobs = Z * g.tiles;
  g.R = reinterpret_cast<uint8_t*>(r);
  g.err = err;
  g.wait = pipeline_wait_cycles();
  const int pairs = count / 2 < g.jobs ? count / 2 : g.jobs;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(2 * pairs));
  cfg.blockDim = dim3(CB_THREADS);
  cfg.dynamicSmemBytes = CB_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  prof_add_flops(PC_OZAKI, 2.0 * g.jobs * CB_M * CB_N * (double)sh.Kp);
  prof_begin(PC_OZAKI, st);
  ZQ_CUDA(cudaLaunchKernelEx(&cfg, k_crt_mma, ta, tb, g));
  prof_end(PC_OZAKI, st);
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

int crt_join(const CrtShape& sh, const void* r, int m, int n, int bits, const int* ea, const int* eb, bool lower,
             double2* C, int64_t ldc, cudaStream_t st) {
  const int64_t blocks = ((int64_t)((m + 3) / 4) * n + 255) / 256;
  const unsigned grid = (unsigned)(blocks > 16384 ? 16384 : blocks);
  const CrtJoin cj = crt_constants(sh.moduli);
  const uint8_t* R = reinterpret_cast<const uint8_t*>(r);
  if (sh.prods == 3)
    ZQ_CUDA(launch_pdl_smem(k_crt_join<true>, dim3(grid), dim3(256), 0, st, R, sh.mp, sh.np, sh.moduli, cj, m, n, bits, ea, eb, lower ? 1 : 0, reinterpret_cast<double*>(C), ldc));
  else
    ZQ_CUDA(launch_pdl_smem(k_crt_join<false>, dim3(grid), dim3(256), 0, st, R, sh.mp, sh.np, sh.moduli, cj, m, n, bits, ea, eb, lower ? 1 : 0, reinterpret_cast<double*>(C), ldc));
  ZQ_LAUNCH_CHECK();
  return ZQ_OK;
}

// Bits of a real operand's largest entry. A double's 53 and seven more: entries below
// the largest of their row or column lose only what lies 2^-60 under it (with 55 bits
// localised eigenvectors came out up to 1.5 times less orthogonal than FP64 merges
// leave them, with 60 as orthogonal; one modulus in 16 more)
constexpr int CRT_FP64_BITS = 60;

size_t crt_dgemm_workspace(int m, int n, int k) {
  const int L = crt_moduli(CRT_FP64_BITS, k);
  const CrtShape s = crt_shape(m, n, k, L ? L : CRT_MAX, false);
  return s.a_bytes + s.b_bytes + s.r_bytes + sizeof(int) * (size_t)(s.mp + s.np) + 6 * 256;
}

int crt_dgemm(int m, int n, int k, const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
              void* ws, int* err, cudaStream_t st) {
  const int L = crt_moduli(CRT_FP64_BITS, k);
  if (L == 0) { set_error_message("crt_dgemm: inner dimension too large"); return ZQ_ERR_LIMIT; }
  const CrtShape sh = crt_shape(m, n, k, L, false);
  char* p = reinterpret_cast<char*>(ws);
  auto take = [&](size_t bytes) { char* q = p; p += (bytes + 255) & ~(size_t)255; return q; };
  void* a = take(sh.a_bytes);
  void* b = take(sh.b_bytes);
  void* r = take(sh.r_bytes);
  int* ea = reinterpret_cast<int*>(take(sizeof(int) * sh.mp));
  int* eb = ea + sh.mp;
  take(sizeof(int) * sh.np);
  ZQ_CUDA(launch_pdl_smem(k_crt_exp_init, dim3(ceil_div(sh.mp + sh.np, 256)), dim3(256), 0, st, ea, sh.mp + sh.np));
  ZQ_LAUNCH_CHECK();
  ZQ_CUDA(launch_pdl_smem(k_crt_exp_real, dim3((unsigned)ceil_div(m, 32), (unsigned)ceil_div(k, 256)), dim3(256), 0, st, A, lda, m, k, true, ea));
  ZQ_LAUNCH_CHECK();
  ZQ_CUDA(launch_pdl_smem(k_crt_exp_real, dim3((unsigned)ceil_div(n, 8)), dim3(256), 0, st, B, ldb, n, k, false, eb));
  ZQ_LAUNCH_CHECK();
  CrtSide s{};
  s.X1 = reinterpret_cast<const double2*>(A); s.ld1 = lda; s.op1 = OP_N; s.K1 = k;
  ZQ_CUDA(launch_pdl_smem(k_crt_split<false>, dim3((unsigned)(sh.mp / 32), (unsigned)(sh.Kp / 64)), dim3(256), 0, st, s, true, m, sh.mp, sh.Kp, ea, CRT_FP64_BITS, L, reinterpret_cast<__nv_bfloat16*>(a)));
  ZQ_LAUNCH_CHECK();
  s.X1 = reinterpret_cast<const double2*>(B); s.ld1 = ldb;
  ZQ_CUDA(launch_pdl_smem(k_crt_split<false>, dim3((unsigned)(sh.np / 32), (unsigned)(sh.Kp / 64)), dim3(256), 0, st, s, false, n, sh.np, sh.Kp, eb, CRT_FP64_BITS, L, reinterpret_cast<__nv_bfloat16*>(b)));
  ZQ_LAUNCH_CHECK();
  if (int rc = crt_multiply(sh, a, b, r, false, err, st)) return rc;
  return crt_join(sh, r, m, n, CRT_FP64_BITS, ea, eb, false, reinterpret_cast<double2*>(C), ldc, st);
}

}  // namespace zq
