// Solver context: the streams, events and device workspace one solve at a
// time runs with. The drop-in entry points share one context per device; the
// request server (zq_serve.cu) owns one per lane and binds each request's
// workspace to it from the stream-ordered pool.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <vector>

#include "zq_forest.h"
#include "zq_kernels.h"

namespace zq {

struct RefineBuffers {
  void* dev = nullptr;
  size_t bytes = 0;
  bool external = false;  // bound by the caller: never freed or grown here
  bool digits = false;    // room for the products' digit slices only
  int last_iters = 0;
  double last_emax = 0.0;
  int last_fallback = 0;
};

struct BatchBuffers {
  void* dev = nullptr;
  size_t bytes = 0;
  std::vector<char> host_tasks;
};

struct Context {
  int device = -1;
  cudaStream_t st = nullptr, st2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  void* ws = nullptr;
  size_t ws_bytes = 0;
  bool ws_external = false;  // bound by the caller: never freed or grown here
  int dc_n = -1;
  bool lean = false;         // the workspace of that plan is without the residue merges' scratch
  DcPlan dc;
  // Device flags of the FP64 path (two ints, made by the first solve), raised when a
  // device-side wait ran out: [0] in the last solve, whose eigenvalues are NaN then,
  // [1] in any since it was last cleared
  int* err = nullptr;
  bool err_set = false;  // the flags are of a solve since the caller reset this
  RefineBuffers rb;
  BatchBuffers bb;
  BatchForest forest;  // layout and scratch of the last batch's mid-size matrices, rebuilt when the layout changes
  // no other solve runs beside this context's (false for the server's lanes): the
  // resident reduction takes every SM, else a quarter of them where that is enough
  bool coop = true;
  // device copy of D for the host-memory entry points, kept between calls
  // (a 1 GB cudaMallocAsync + cudaFreeAsync per n2 = 8192 call cost ~44 ms in
  // a process whose other allocations kept the pool from reusing the memory)
  void* hbuf = nullptr;
  size_t hbuf_bytes = 0;
  std::mutex mu;
};

// Streams and events of a new context on `device` (no workspace yet).
int context_create(int device, Context** out);
// Frees what the context owns (not bound workspace); synchronises its streams.
void context_destroy(Context* c);
// Device bytes one solve of quaternion size n needs: the FP64 path's workspace
// and, for refined = true, the refinement buffers on top (with the Ozaki
// products' residues). lean: the least it runs in, without residues.
void solve_workspace_bytes(int n, size_t* fp64_bytes, size_t* refine_bytes, bool lean = false);
// Use caller-owned workspace for the next solves (nullptr/0 unbinds).
void context_bind(Context* c, void* ws, size_t ws_bytes, void* rws, size_t rws_bytes);

int ensure_ws(Context* c, size_t bytes);
int ensure_plan(Context* c, int n);
// reads one of the context's flags if a solve has set it, waiting for c->st: ZQ_ERR_TIMEOUT if it is up
int check_timeout(Context* c, int flag);
int solve_device(Context* c, double2* dD, int64_t ldd, int n, double* deig, bool vectors, cudaStream_t st);
int refined_device(Context* c, double2* dD, int64_t ldd, int n, double* deig, cudaStream_t st, int mode,
                   bool vectors = true);
// drop-in policy: 0 FP64 path, 1 refined path for quaternion size n
int path_for(int n);
// tuned panel widths (prec 0: FP64 path, 1: FP32 decomposition), 0 = not tuned
void nb_table_set(int prec, int n, int nb);
int nb_table_get(int prec, int n);

// batched kernels (zq_batched.cu, zq_small.cu)
// a task table sorted largest first: `large` tasks for a CTA each, then `small`
// ones, of order at most small_max, for a warp each
struct BatchSplit { int large = 0, small = 0, small_max = 0; };
template <typename F> BatchSplit batched_split(int count, int wmax, F&& order_of) {
  BatchSplit s;
  while (s.large < count && order_of(s.large) > wmax) ++s.large;
  s.small = count - s.large;
  s.small_max = s.small > 0 ? order_of(s.large) : 0;
  return s;
}
long long batched_ws_stride();
int batched_max_n();
int batched_launch(const void* dev_tasks, const BatchSplit& split, int* dev_counter, double2* D, double* eig, double* ws,
                   int ctas, int* dev_info, cudaStream_t st);
int batched_warp_max();
void batched_set_warp_max(int v);
size_t batched_task_bytes();
void batched_fill_task(void* dst, long long off, long long eoff, int n, int ld, int slot);
// task addressing its matrix and eigenvalues by pointer (D, eig of the launch unused for it)
void batched_fill_task_ptr(void* dst, double2* D, double* eig, int n, int ld, int slot);

}  // namespace zq
