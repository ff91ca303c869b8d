// Internal interfaces between the solver's translation units.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

#include "zq_common.cuh"

namespace zq {

// ---------------------------------------------------------------- tridiagonal
// widest panel of the blocked reduction (reflectors kept per panel)
constexpr int NBMAX = 128;

template <typename R>
struct TridiagView {
  cplx<R>* M;      // [A; B], 2n x n, column-major
  int n;
  int64_t ld;
  cplx<R>* Ya;     // panel aux vectors, n x nbmax (global row index), ld = ldy
  cplx<R>* Yb;
  int64_t ldy;
  int nbmax;
  cplx<R>* ga;     // g of the current column (n)
  cplx<R>* gb;
  cplx<R>* hpart;  // hemv tile partials: hblk x hblk x 32 x 2
  int hblk;
  cplx<R>* dpart;  // panel dot partials, one set per 128 rows: hblk x nbmax x 4 (room for 4x that)
  cplx<R>* dots;   // the summed panel dot products: 4 * nbmax
  double* npart;   // norm partials: 2 * hblk
  double* cpart;   // c partials, one per hreduce CTA: ceil(n / 8) + 1
  double* scal;    // per-column scalars (16): [0..3] x_1 of the column, [4] f, [5..8] f m (reflector head)
  unsigned* counter;  // colupd CTAs finished for the current column (the last one forms the reflector)
  double* d;       // diagonal (n)
  double* e;       // quaternion subdiagonal (4 doubles each, n)
  double* tau;     // 1 if reflector j exists else 0 (n)
  int* tc_err;     // raised when a bounded wait ran out (null: NaN in d only); FP32: tensor-core products
                   // allowed where it is set, CUDA cores only where it is null
  void* rws;       // exchange area of the resident reduction (zq_resident.cu)
  int ctas;        // CTAs it may use (0: the per-column kernels only)
};

template <typename R>
size_t tridiag_workspace_bytes(int n, int nbmax);
template <typename R>
TridiagView<R> tridiag_bind(void* ws, cplx<R>* M, int n, int64_t ld, int nbmax, double* d, double* e, double* tau);
template <typename R>
int tridiagonalize(TridiagView<R> v, int nb, cudaStream_t st);

// ---------------------------------------------------------------------- GEMM
enum { OP_N = 0, OP_T = 1, OP_C = 2, OP_R = 3 };

template <typename R>
struct ZgemmArgsT {
  int m, n, k1, k2;
  const cplx<R>* A1; int64_t lda1;
  const cplx<R>* B1; int64_t ldb1;
  const cplx<R>* A2; int64_t lda2;   // null: single segment
  const cplx<R>* B2; int64_t ldb2;
  R s2;
  cplx<R> alpha, beta;
  cplx<R>* C; int64_t ldc;
  cplx<R>* P; int64_t pcap;          // optional split-K partial buffer (complex elements)
};
using ZgemmArgs = ZgemmArgsT<double>;
template <typename R>
int zgemm(int opa1, int opb1, int opa2, int opb2, const ZgemmArgsT<R>& g, int batch, cudaStream_t st);

template <typename R>
struct DgemmDescT {
  const R* A; const R* B; R* C;
  int64_t lda, ldb, ldc;
  int64_t off_a, off_b, off_c;  // plan-time offsets (bound to pointers before upload)
  int m, n, k;
  int ta, tb;
  int tile0;
  R alpha, beta;
};
using DgemmDesc = DgemmDescT<double>;
template <typename R>
int dgemm_grouped(DgemmDescT<R>* host_descs, int count, DgemmDescT<R>* dev_descs, cudaStream_t st);
template <typename R>
void grouped_launch(const DgemmDescT<R>* dev_descs, int count, int tiles, cudaStream_t st);
int dgemm_tiles(int m, int n);

// ------------------------------------------------------------------ D&C (c)
// A node covers positions [a, b) (children [a, c) and [c, b)); position r, c of
// its matrix lie at zoff + r + c ld of the eigenvector buffers.
struct DcNode {
  int a, c, b;
  int K, ndefl, nrot;
  double rho, rho2;
  long long zoff;
  int ld, pad;
};
// one matrix of a forest: positions [p, p + n), eigenvalues at eig + eoff
struct DcMat {
  int p, n;
  long long eoff;
};
struct DcWork {
  double *sd, *sz, *nd_val, *nd_z, *df_val, *df_sval, *rot_c, *rot_s, *r_tau, *r_lam, *zhat;
  int *perm, *nd_col, *df_col, *df_scol, *rot_p, *rot_j, *r_orig;
};
struct DcPlan {
  int n = 0;           // positions (the order, or the sum of the orders of a forest)
  size_t nn = 0;       // elements of one eigenvector buffer (the sum of the squares)
  std::vector<DcMat> mats_host;
  std::vector<long long> zoff;  // per matrix: element (0, 0) of its block in the eigenvector buffers
  int max_depth = 0;
  std::vector<DcNode> nodes_host;
  std::vector<int> depth_off, depth_cnt, leaf_off, leaf_cnt;
  std::vector<int> depth_mmax;  // largest node (b - a) per depth
  std::vector<DgemmDesc> gemm_host;
  std::vector<int> gemm_off, gemm_tiles;
  // device
  double* base = nullptr;
  double* Z[2] = {nullptr, nullptr};
  double* Mb = nullptr;
  double* lam[2] = {nullptr, nullptr};
  double *dmod = nullptr, *es = nullptr, *scal = nullptr;  // scal: one scale per matrix
  DcMat* mats_dev = nullptr;
  DcWork w{};
  DcNode* nodes_dev = nullptr;
  DgemmDesc* descs_dev = nullptr;
  // single-precision views of Z and M, and their descriptors (after the double
  // ones and two spare slots in the descriptor area)
  float* Zf[2] = {nullptr, nullptr};
  float* Mbf = nullptr;
  DgemmDescT<float>* fdescs_dev = nullptr;
  double* crt_ws = nullptr;  // scratch of the residue-arithmetic merges (orders from DC_CRT_MIN)
  int* err = nullptr;        // raised when one of their pipeline waits ran out: the eigenvalues become NaN
  int* tc_err = nullptr;  // run_single: merges of large nodes on the tensor cores (timeout flag) when set

  // lean: without the scratch of the residue merges, which then run on the FP64 pipe
  static size_t workspace_doubles(int n, bool lean = false);
  size_t forest_doubles() const;  // the same for a built plan of several matrices, without their table
  int build(int n);
  // several tridiagonals at once: orders ns, eigenvalues at eoffs of the
  // array given to run_forest
  int build(const std::vector<int>& ns, const std::vector<long long>& eoffs);
  size_t num_nodes() const { return nodes_host.size(); }
  size_t num_descs() const { return gemm_host.size(); }
  int gemm_cnt(int t) const {  // descriptors of depth t
    return (t + 1 < (int)gemm_off.size() ? gemm_off[t + 1] : (int)gemm_host.size()) - gemm_off[t];
  }
  // mats: the table's place where the workspace is not the plan's alone (null: in the workspace)
  int upload(double* ws, DcNode* dnodes, DgemmDesc* ddescs, cudaStream_t st, DcMat* mats = nullptr, bool lean = false);
  // d (n), e (n-1) on device; lam_out (n) on device; z_out points into the workspace
  // flags (two ints, null: the plan's own, cleared here): raised when a wait of a residue
  // product ran out; the eigenvalues become NaN when [0] is up, which then raises [1] too
  int run(const double* d, const double* e, double* lam_out, double*& z_out, cudaStream_t st, int* flags = nullptr);
  // a forest: d, e indexed by position (e of a matrix's last position unused),
  // eigenvalues to eig + eoff of each matrix, eigenvectors in Z[0]
  // (info: one int per matrix, zeroed by the caller, counts its eigenvalues that are not finite)
  int run_forest(const double* d, const double* e, double* eig, int* info, cudaStream_t st);
  // same tree with Z and the merge products in FP32 (eigenvalues and the
  // secular equation stay FP64): the refined path's decomposition
  // the same for couplings e of either sign, Z stored at ldz: e_abs and signs are n doubles of scratch each
  int run_signed(const double* d, const double* e, double* lam_out, double* Z_out, int64_t ldz, double* e_abs,
                 double* signs, cudaStream_t st);
  int run_single(const double* d, const double* e, double* lam_out, float*& z_out, cudaStream_t st);
  // descriptor area bytes for upload(): double descriptors + 2 spare + float descriptors
  static size_t desc_bytes(size_t ndescs) {
    return sizeof(DgemmDescT<double>) * (ndescs + 2) + sizeof(DgemmDescT<float>) * ndescs;
  }
};

// ------------------------------------------------------------ back-transform
// phase reduction of the quaternion tridiagonal: e (4 doubles per entry) ->
// real off-diagonal |e_k| and unit quaternions phi_k = (alpha_k, beta_k)
int phase_reduce(const double* e, int n, double* offd, double* phi, cudaStream_t st);
// the same for each matrix of a forest (arrays indexed by position)
int phase_reduce_forest(const double* e, const DcMat* mats, int count, int nmax, double* offd, double* phi,
                        cudaStream_t st);
// X = [diag(alpha); diag(beta)] (2n x n complex, ld), then Q X by blocked reflectors
// tc_err (FP32 only, may be null): with it, the large products run on the
// tensor cores (zq_tc32.cu) and a pipeline-wait timeout raises *tc_err
template <typename R>
int form_q(const cplx<R>* M, int64_t ldm, int n, const double* phi, cplx<R>* X, int64_t ldx,
           int nbq, void* ws, cudaStream_t st, int* tc_err = nullptr, void* big = nullptr, size_t big_bytes = 0);
size_t form_q_workspace_bytes(int n, int nbq);
// out (2n x n complex, ldo) = X (2n x n complex, ldx) * Z (n x n real, ldz)
template <typename R>
int apply_z(const cplx<R>* X, int64_t ldx, const R* Z, int64_t ldz, int n, cplx<R>* out, int64_t ldo,
            DgemmDescT<R>* dev_desc, cudaStream_t st, int* tc_err = nullptr);
// FP32 products of the refined decomposition that may run on the TF32x3
// tensor-core kernel: trailing update, Q formation (the W^H X products with
// inner dimension L, and the X updates with inner dimension nbq), back-transform,
// divide-and-conquer merges
enum { TC_USE_TRAIL = 0, TC_USE_FORMQ = 1, TC_USE_APPLYZ = 2, TC_USE_DC = 3, TC_USE_FORMQ_X = 4 };
bool fp32_products_on_tensor_cores(int use);
// right half of the n2 x n2 output from the left half (U; V)
int symmetry_fill(double2* D, int64_t ld, int n, cudaStream_t st);

// ------------------------------------------------------ refined (mixed) path
struct RefineArgs {
  double2* dD; int64_t ldd; int n; double* deig;
  void* ws;                    // refine_workspace_bytes(n, nbq)
  void* ows; size_t ows_bytes; // accurate-product workspace (mode 1)
  DcPlan* dc;                  // uploaded plan for n
  DgemmDescT<float>* fdesc;    // one device descriptor slot
  int nb, nbq, mode, max_iter;
  double tol;
  double cluster_tol;          // accepted in-cluster coupling (relative to max |lambda|)
  double pair_eps;             // first-order formula only where |coupling| <= pair_eps |gap| (first step)
  double pair_eps_late;        // the same bound in the later steps
  int slices0;                 // Ozaki slices of the first step's products
  int slices_res;              // Ozaki slices of the products with the residual R = HX - X Lambda
  int values_only;             // the eigenvalues alone: no last update of X, no vectors in place
  int digits;                  // the products' workspace holds digit slices only
  int coop;                    // no other solve runs beside this one: the FP32 reduction may take every SM
  cudaStream_t st;
  cudaStream_t st2;            // second stream: Q formation overlaps the tridiagonal solve
  cudaEvent_t ev_fork, ev_join;
  int iters; double last_emax;  // outputs
  double last_cluster;         // in-cluster coupling of the last step (before rotation)
  int clusters;                // clusters resolved (-1: one too large)
  int cluster_max;             // largest cluster rotated
};
size_t refine_workspace_bytes(int n, int nbq);
int refined_solve(RefineArgs& ra);

// Ozaki-sliced FP64-accurate complex product (zq_ozaki.cu)
struct OzOpts {
  int slices;      // bf16 slices per operand (7 bits each), 2..8
  int structured;  // 0 general; +1 Hermitian / -1 antisymmetric square output (lower tiles computed)
  int reuse_a;     // 1: the A operand is the same as in the previous call (slices kept)
  int nofill;      // structured: leave the upper triangle to the caller (who fills it with structured_fill)
  int prev_slices; // reuse_a: the slices of the previous call
  int* err;        // device flag a pipeline timeout raises, cleared and read by the caller (null: here, with a wait)
  int digits;      // 1: digit slices at any accuracy (workspaces too small for residues)
};
int zgemm_ozaki(int opa1, int opb1, int opa2, int opb2, const ZgemmArgs& g, void* ws, size_t ws_bytes, cudaStream_t st,
                const OzOpts& opt);
// workspace of one product (K = the complex inner dimension of all segments)
size_t zgemm_ozaki_bytes(int m, int n, int64_t K, int slices, bool digits = false);
size_t ozaki_workspace_bytes(int n, bool digits = false);
// the current device's pool for the scratch of single calls: stream-ordered,
// keeps up to SCRATCH_KEEP bytes mapped between calls (zq_release_workspace
// returns them)
constexpr unsigned long long SCRATCH_KEEP = 4ull << 30;
int scratch_pool(cudaMemPool_t* pool);
void scratch_pool_trim();
// limit of every mbarrier wait in the tensor-core pipelines, SM clock cycles
// (<= 0: the default, about 2 s); a test hook for the timeout path
void set_pipeline_wait_cycles(long long cycles);
long long pipeline_wait_cycles();
// the driver's cuTensorMapEncodeTiled (null when unavailable)
void* tensor_map_encode_fn();
// upper triangle of a square structured matrix from its lower triangle (sym +1 Hermitian, -1 antisymmetric)
int structured_fill(double2* C, int64_t ldc, int n, int sym, cudaStream_t st);

}  // namespace zq
