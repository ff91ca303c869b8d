// Batches of mid-size matrices (order 33 to 256, from 16 where a batch has few small
// ones; FP64) as a few launches over all matrices at once. Reference: the steps of ts::zquatev (zquatev.cc:42-100) once
// per matrix; it has no batched entry point.
//
//   1. the reductions: a queue of matrices, largest first, each taken by a cluster
//      of CTAs that holds it in shared memory (zq_resident.cu);
//   2. the phases, one CTA per matrix (zq_backtransform.cu);
//   3. one divide and conquer over all tridiagonals: the trees of the matrices
//      form a forest whose depths are merged together (zq_stedc.cu);
//   4. the back-transform, one CTA per eigenvector column (zq_applyq.cu).
//
// Why: one CTA per matrix (zq_batched.cu) left an order-256 matrix on one SM,
// where the FP64 pipe (2 FMA per clock) alone needs 76 ms and the serial QL
// iteration as much again: 340 ms, whatever the batch. Here every step spreads
// over the GPU, bound by the FP64 pipe: 40 matrices each of orders 256, 215,
// 214, 140, 47, 34, 23 and 13 take 120 ms instead of 338 (reductions 58 ms,
// 27 ms of FP64 pipe time; divide and conquer 12 ms; back-transform 50 ms, 40 ms
// of pipe time; the small ones 3 ms).
#include "zq_common.cuh"
#include "zq_forest.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "zq_applyq.h"
#include "zq_context.h"
#include "zq_resident.h"

namespace zq {

// Elements of one eigenvector buffer of a chunk: positions and tile counts of its
// divide and conquer stay within 32 bits, and the scratch of the chunks, which run one
// after another in the same memory, within 6.5 GB (ZQ_FOREST_CHUNK: smaller chunks)
constexpr size_t FOREST_CHUNK = (size_t)1 << 28;
static size_t forest_chunk() {
  const char* s = getenv("ZQ_FOREST_CHUNK");
  const long long v = s ? atoll(s) : 0;
  return v > 0 && (size_t)v < FOREST_CHUNK ? (size_t)v : FOREST_CHUNK;
}

// A part of the batch with its own tables (batches beyond 2 GiB of eigenvectors have
// several) and the scratch that all parts share.
struct BatchForest::Chunk {
  DcPlan dc;
  int count = 0, N = 0;
  struct TriClass { int first, count, m_max, G; void* ws; int* queue; };
  std::vector<TriClass> tri;
  struct ApplyClass { int col0, cols, nmax, block0, blocks; };
  std::vector<ApplyClass> apply;
  // device
  TriTask<double>* tri_tasks = nullptr;
  ApplyQTask* apply_tasks = nullptr;
  int* task_of = nullptr;
  bool warp_columns = false;
  std::vector<int2> blocks_host;
  int2* blocks = nullptr;
  double *d = nullptr, *e = nullptr, *tau = nullptr, *offd = nullptr, *phi = nullptr;
  size_t tri_ws_bytes = 0;
  double* dcws = nullptr;
  DcNode* nodes = nullptr;
  DgemmDesc* descs = nullptr;
  DcMat* mats = nullptr;
};

BatchForest::~BatchForest() { release(); }

void BatchForest::release() {
  for (Chunk* c : chunks_) delete c;
  chunks_.clear();
  drop();
  items_.clear();
}

void BatchForest::drop() {
  if (dev_ && pooled_) cudaFreeAsync(dev_, st_);
  else if (dev_) cudaFree(dev_);
  dev_ = nullptr;
  bytes_ = 0;
}

int BatchForest::reserve(size_t bytes, cudaStream_t st) {
  if (bytes_ >= bytes) return ZQ_OK;
  drop();
  st_ = st;
  const cudaError_t e = pooled_ ? cudaMallocAsync(&dev_, bytes, st) : cudaMalloc(&dev_, bytes);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    dev_ = nullptr;
    release();
    set_error_message("batch: device allocation failed");
    return ZQ_ERR_NOMEM;
  }
  bytes_ = bytes;
  return ZQ_OK;
}

int BatchForest::build(const std::vector<ForestItem>& items, cudaStream_t st) {
  if (dev_) ZQ_CUDA(cudaStreamSynchronize(st));  // the memory is reused
  for (Chunk* c : chunks_) delete c;
  chunks_.clear();
  items_.clear();
  if (items.empty()) return ZQ_OK;
  int dev = 0, sms = 0;
  ZQ_CUDA(cudaGetDevice(&dev));
  ZQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  size_t tables = up(sizeof(int) * items.size()), scratch = 0;
  const size_t limit = forest_chunk();
  for (size_t i0 = 0; i0 < items.size();) {
    Chunk* c = new Chunk();
    chunks_.push_back(c);
    std::vector<int> ns;
    std::vector<long long> eo;
    size_t nn = 0, i1 = i0;
    while (i1 < items.size() && (i1 == i0 || nn + (size_t)items[i1].n * items[i1].n <= limit)) {
      nn += (size_t)items[i1].n * items[i1].n;
      ns.push_back(items[i1].n);
      eo.push_back(items[i1].eoff);
      ++i1;
    }
    c->count = (int)ns.size();
    c->dc.build(ns, eo);
    c->N = c->dc.n;
    // Reductions: one queue for all matrices or one per range of orders (up to
    // 96, 160, 224, 256), each with the cluster size that finishes it soonest,
    // whichever is less in all: large clusters suit few large matrices, small ones
    // waste fewer SMs in the phases between the sweeps (the batch above: 71.5 ms
    // at 8 CTAs for every order).
    double one = 0.0, split = 0.0;
    const int G1 = tri_queue_cluster(ns.data(), c->count, &one);
    if (G1 == 0) { set_error_message("batch: no cluster holds the largest matrix"); return ZQ_ERR_LIMIT; }
    std::vector<Chunk::TriClass> parts;
    for (int q = 0; q < c->count;) {
      const int lim = ns[q] > 224 ? 224 : (ns[q] > 160 ? 160 : (ns[q] > 96 ? 96 : 0));
      int q1 = q;
      while (q1 < c->count && ns[q1] > lim) ++q1;
      double t = 0.0;
      const int G = tri_queue_cluster(ns.data() + q, q1 - q, &t);
      split += t;
      parts.push_back({q, q1 - q, ns[q], G, nullptr, nullptr});
      q = q1;
    }
    if (one <= split) parts.assign(1, Chunk::TriClass{0, c->count, ns[0], G1, nullptr, nullptr});
    c->tri = parts;
    for (const Chunk::TriClass& t : c->tri) c->tri_ws_bytes = std::max(c->tri_ws_bytes, tri_queue_bytes(t.G, t.m_max, t.count));
    c->tri_ws_bytes = up(c->tri_ws_bytes) + 256;  // and the queue's counter
    // Back-transform: one launch per register class (largest order first). With
    // more columns than the GPU has quadrants several times over, a warp takes a
    // column (less FP64 work per reflector); with fewer, a CTA does.
    c->warp_columns = c->N >= 4 * 4 * sms;
    static const int wide[] = {256, 224, 192, 160, 128, 96, 64}, narrow[] = {256, 192, 128, 96, 64};
    int col = 0;
    for (int q = 0; q < c->count;) {
      int lim = 0;
      if (c->warp_columns) { for (int k : wide) if (ns[q] > k) { lim = k; break; } }
      else { for (int k : narrow) if (ns[q] > k) { lim = k; break; } }
      int q1 = q, cols = 0;
      const int b0 = (int)c->blocks_host.size();
      for (; q1 < c->count && ns[q1] > lim; ++q1) {
        cols += ns[q1];
        for (int f = 0; f < ns[q1] && c->warp_columns; f += APPLYQ_WARP_COLUMNS) c->blocks_host.push_back(make_int2(q1, f));
      }
      c->apply.push_back({col, cols, ns[q], b0, (int)c->blocks_host.size() - b0});
      col += cols;
      q = q1;
    }
    const size_t N = (size_t)c->N;
    tables += up(sizeof(TriTask<double>) * c->count) + up(sizeof(ApplyQTask) * c->count) + up(sizeof(int) * N) +
              up(sizeof(int2) * (c->blocks_host.size() + 1)) + up(sizeof(DcNode) * (c->dc.num_nodes() + 1)) +
              up(DcPlan::desc_bytes(c->dc.num_descs())) + up(sizeof(DcMat) * c->count);
    scratch = std::max(scratch, up(sizeof(double) * 11 * N) + c->tri_ws_bytes + up(sizeof(double) * c->dc.forest_doubles()));
    i0 = i1;
  }
  if (int rc = reserve(tables + scratch, st)) return rc;
  char* p = reinterpret_cast<char*>(dev_);
  auto take = [&](size_t b) { char* q = p; p += up(b); return q; };
  info_ = reinterpret_cast<int*>(take(sizeof(int) * items.size()));
  size_t base = 0;
  for (Chunk* c : chunks_) {
    const size_t N = (size_t)c->N;
    c->tri_tasks = reinterpret_cast<TriTask<double>*>(take(sizeof(TriTask<double>) * c->count));
    c->apply_tasks = reinterpret_cast<ApplyQTask*>(take(sizeof(ApplyQTask) * c->count));
    c->task_of = reinterpret_cast<int*>(take(sizeof(int) * N));
    c->blocks = reinterpret_cast<int2*>(take(sizeof(int2) * (c->blocks_host.size() + 1)));
    c->nodes = reinterpret_cast<DcNode*>(take(sizeof(DcNode) * (c->dc.num_nodes() + 1)));
    c->descs = reinterpret_cast<DgemmDesc*>(take(DcPlan::desc_bytes(c->dc.num_descs())));
    c->mats = reinterpret_cast<DcMat*>(take(sizeof(DcMat) * c->count));
    char* const next = p;
    p = reinterpret_cast<char*>(dev_) + tables;  // the chunks' common scratch
    double* v = reinterpret_cast<double*>(take(sizeof(double) * 11 * N));
    c->d = v; c->e = v + N; c->tau = v + 5 * N; c->offd = v + 6 * N; c->phi = v + 7 * N;
    int* queue = reinterpret_cast<int*>(take(256));
    void* tri_ws = take(c->tri_ws_bytes - 256);
    for (Chunk::TriClass& t : c->tri) { t.queue = queue; t.ws = tri_ws; }
    c->dcws = reinterpret_cast<double*>(take(sizeof(double) * c->dc.forest_doubles()));
    p = next;
    if (int rc = c->dc.upload(c->dcws, c->nodes, c->descs, st, c->mats)) return rc;
    std::vector<TriTask<double>> tt(c->count);
    std::vector<ApplyQTask> at(c->count);
    std::vector<int> of(N);
    for (int q = 0; q < c->count; ++q) {
      const ForestItem& it = items[base + q];
      const int P = c->dc.mats_host[q].p;
      tt[q] = TriTask<double>{nullptr, it.n, 0, it.ld, c->d + P, c->e + 4 * (size_t)P, c->tau + P, it.off};
      at[q] = ApplyQTask{nullptr, c->phi + 4 * (size_t)P, c->dc.Z[0] + c->dc.zoff[q], it.ld, it.n, it.n, P, it.off};
      for (int i = 0; i < it.n; ++i) of[P + i] = q;
    }
    base += c->count;
    ZQ_CUDA(cudaMemcpyAsync(c->tri_tasks, tt.data(), sizeof(tt[0]) * tt.size(), cudaMemcpyHostToDevice, st));
    ZQ_CUDA(cudaMemcpyAsync(c->apply_tasks, at.data(), sizeof(at[0]) * at.size(), cudaMemcpyHostToDevice, st));
    ZQ_CUDA(cudaMemcpyAsync(c->task_of, of.data(), sizeof(int) * of.size(), cudaMemcpyHostToDevice, st));
    if (!c->blocks_host.empty())
      ZQ_CUDA(cudaMemcpyAsync(c->blocks, c->blocks_host.data(), sizeof(int2) * c->blocks_host.size(),
                              cudaMemcpyHostToDevice, st));
    ZQ_CUDA(cudaStreamSynchronize(st));  // the host arrays go out of scope
  }
  items_ = items;
  return ZQ_OK;
}

int BatchForest::run(double2* D, double* eig, cudaStream_t st) {
  if (items_.empty()) return ZQ_OK;
  ZQ_CUDA(cudaMemsetAsync(info_, 0, sizeof(int) * items_.size(), st));
  int* info = info_;
  for (Chunk* c : chunks_) {
    for (const Chunk::TriClass& t : c->tri)
      if (int rc = tri_queue(c->tri_tasks + t.first, t.count, D, t.m_max, t.G, t.ws, t.queue, st)) return rc;
    if (int rc = phase_reduce_forest(c->e, c->dc.mats_dev, c->count, items_.front().n, c->offd, c->phi, st)) return rc;
    if (int rc = c->dc.run_forest(c->d, c->offd, eig, info, st)) return rc;
    info += c->count;
    ApplyQTask base{};
    base.D = D;
    for (const Chunk::ApplyClass& a : c->apply) {
      if (c->warp_columns) {
        if (int rc = apply_q_warp(c->apply_tasks, c->blocks + a.block0, a.blocks, D, a.nmax, st)) return rc;
      } else {
        if (int rc = apply_q(c->apply_tasks, c->task_of, base, a.col0, a.cols, a.nmax, st)) return rc;
      }
    }
    if (c->warp_columns)
      if (int rc = apply_q_finish(c->apply_tasks, c->task_of, base, 0, c->N, items_.front().n, st)) return rc;
  }
  return ZQ_OK;
}

}  // namespace zq
