// Definitions of the opaque C-ABI handles (internal to the engine library).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <tuple>
#include <vector>

#include "kernels.h"
#include "params.h"
#include "xpir_b200.h"

struct xpir_b200_db;
struct BatchPlan;  // batch.cu

// Tile-shape choices made by xpir_b200_autotune, keyed by level shape (P, n_i, groups).
typedef std::map<std::tuple<uint64_t, uint64_t, uint64_t>, int> TuneTable;

struct xpir_b200_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  // Host queries of recursive replies: the later levels' ciphertexts are copied on this
  // stream while the first level replies; the event marks the end of that copy.
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t query_copied = nullptr;
  xpir::ParamSet ps;           // b is set per database
  uint64_t *d_tables = nullptr;  // also holds zero_poly and stop_flags
  std::mutex mu;
  std::atomic<uint64_t> launches{0};  // engine kernels launched (also counted off the lock)
  std::atomic<int> servers{0};         // servers with a lane on this context
  cudaError_t last_error = cudaSuccess;  // the last CUDA error of a batch on this context
  // grow-only workspaces (device)
  void *ws_query = nullptr;
  size_t ws_query_bytes = 0;
  void *ws_a = nullptr;  // level replies
  size_t ws_a_bytes = 0;
  void *ws_b = nullptr;  // re-imported level databases
  size_t ws_b_bytes = 0;
  void *tasks_dev = nullptr;   // task table of uncaptured batches (device copy)
  void *tasks_host = nullptr;  // and its pinned staging copy
  size_t tasks_cap = 0;        // entries of both
  // Stream-ordered pool of the client-side entry points' per-call buffers (query
  // generation, extraction): it keeps freed memory for the next call (release threshold
  // UINT64_MAX), so that a call after the first maps no new device memory.
  cudaMemPool_t pool = nullptr;
  // mapped pinned memory: [0] kernel status, kRedoFlags redo flags (SumLevelArgs), then
  // kZeroHints ints that databases hold one of each (xpir_b200_db::hint)
  int *status_host = nullptr;
  int *status_dev = nullptr;
  uint64_t *zero_poly = nullptr;  // [m][N]: import of a zero bit stream
  int *stop_flags = nullptr;      // SumLevelArgs::stop, kRedoFlags ints
  uint64_t *ws_part = nullptr;    // residues of runs (SumLevelArgs::part), kPartWords words
  std::vector<int> free_hints;   // indexes of status_host that no database holds
  std::set<xpir_b200_db *> dbs;  // databases imported through this context
  TuneTable tuned;
  uint64_t tune_epoch = 0;  // bumped by every autotune (invalidates captured batches)
  xpir::WaitTest wait_test;  // test support of the bounded waits (xpir_b200_ctx_set_wait_test)
  // Kernel timing (xpir_b200_ctx_set_kernel_timing): an event pair around each level's
  // reply launch and each re-import of xpir_b200_reply, summed after the call's sync.
  bool timing = false;
  cudaEvent_t timing_ev[2 * XPIR_B200_MAX_LEVELS][2] = {};
  double reply_ms[XPIR_B200_MAX_LEVELS] = {}, import_ms = 0;
  uint64_t reply_timed[XPIR_B200_MAX_LEVELS] = {}, import_timed = 0;
  std::vector<std::shared_ptr<BatchPlan>> plans;  // captured batches (batch.cu)
};

constexpr int kZeroHints = 1022;
constexpr int kFirstHint = 1 + (int)xpir::kRedoFlags;  // in status_host
constexpr size_t kSpareBytes = 1ull << 30;

// Workspace of the residue sums' runs: 3.8 MiB per context (of a slab of 32 MB, which a
// program's first context allocates and seven more share), taken with it, so that no reply
// allocates it (a level takes as many runs as fit; the 100,000 x 4 KB level's 27 take 221,184
// words).
constexpr uint64_t kPartWords = 500000;

// Tile shape for a level shape: the autotuned one if any, else -1 (default).
inline int tuned_tile(const xpir_b200_ctx *ctx, uint64_t P, uint64_t n_i, uint64_t groups) {
  auto it = ctx->tuned.find(std::make_tuple(P, n_i, groups));
  return it == ctx->tuned.end() ? -1 : it->second;
}

struct xpir_b200_db {
  xpir_b200_ctx *ctx = nullptr;
  uint64_t id = 0;  // unique per import in this process (never reused, unlike the address)
  uint64_t *d_polys = nullptr;
  size_t alloc_bytes = 0;  // of d_polys
  uint64_t n_agg = 0;
  uint64_t P = 0;
  uint32_t b = 0;
  uint32_t alpha = 1;
  uint64_t element_bytes = 0;
  // Index in status_host of this database's zero hint (AggSource), 0: none.  Long stretches of
  // words 0 and p, the import of zero bits, keep the residue sums from deciding a chain, so
  // replies from a database with kZeroPolys all-zero polys anywhere run slot by slot at once.
  // Only a hint: it may be set late (imports from device memory are asynchronous), and the sums
  // notice by themselves.  Such a first reply may run twice; 100,000 x 4 KB, import and first
  // reply: no zeros 6.70 ms, the last tenth zero 8.16 (slot by slot alone 7.31).
  int hint = 0;
  bool zero_polys() const { return hint && ((volatile int *)ctx->status_host)[hint] != 0; }
};

// Whether a level takes the residue-sum path: no pinned or tuned tile shape.
inline bool sum_level(const xpir_b200_ctx *ctx, const xpir::ParamSet &ps, uint64_t n_real, uint64_t n_live, uint64_t P,
                      uint64_t n_i, uint64_t groups, uint64_t ntasks) {
  return tuned_tile(ctx, P, n_i, groups) < 0 && xpir::sum_level_supported(ps, n_real, n_live, P, n_i, groups, ntasks);
}

inline xpir::SumLevelArgs sum_args(const xpir_b200_ctx *ctx, uint64_t n_real, uint64_t n_live, uint64_t P,
                                   uint64_t n_groups, uint64_t n_i, bool write_idle, uint32_t first = 0) {
  return {n_real,     n_live, P, n_groups, n_i, write_idle, ctx->zero_poly, ctx->ws_part, kPartWords,
          ctx->status_dev, ctx->stop_flags, first, {}};
}

// Clears the kernel status and the redo flags of a call's queries.
inline void clear_status(xpir_b200_ctx *ctx, uint64_t queries = 1) {
  memset(ctx->status_host, 0, (1 + std::min<uint64_t>(queries, xpir::kRedoFlags)) * sizeof(int));
}
// Whether query i of the call that ended has to be repeated slot by slot.
inline bool asked_again(const xpir_b200_ctx *ctx, uint64_t i = 0) {
  return ((volatile int *)ctx->status_host)[1 + std::min<uint64_t>(i, xpir::kRedoFlags - 1)] != 0;
}
// Lets every CTA work again, before such a repeat.
inline cudaError_t clear_stop(xpir_b200_ctx *ctx) {
  return cudaMemsetAsync(ctx->stop_flags, 0, xpir::kRedoFlags * sizeof(int), ctx->stream);
}

struct xpir_b200_request;

namespace xpir {
// Spare memory: the polys of databases freed last, at most kSpareBytes per device and one block
// by each context, for the next import of any context there (mapping and unmapping 655 MB
// costs more than importing them).  Given back when the context that freed it is destroyed,
// and by allocate and pool_allocate when an allocation on the device fails.  Nothing queued
// anywhere uses a spare block.  Callable from any thread.
bool take_spare(const xpir_b200_ctx *ctx, size_t bytes, void **ptr, size_t *have);
void keep_spare(const xpir_b200_ctx *ctx, void *ptr, size_t bytes);  // or frees it
void drop_spare(const xpir_b200_ctx *ctx);
// cudaMalloc on `device` (the current one), and cudaMallocFromPoolAsync.
cudaError_t allocate(int device, void **buf, size_t bytes);
cudaError_t pool_allocate(int device, void **buf, size_t bytes, cudaMemPool_t pool, cudaStream_t stream);
inline cudaError_t allocate(const xpir_b200_ctx *ctx, void **buf, size_t bytes) {
  return allocate(ctx->device, buf, bytes);
}
inline cudaError_t pool_allocate(const xpir_b200_ctx *ctx, void **buf, size_t bytes) {
  return pool_allocate(ctx->device, buf, bytes, ctx->pool, ctx->stream);
}

// Whether two address ranges share a byte.
inline bool overlap(const void *a, uint64_t a_bytes, const void *b, uint64_t b_bytes) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + b_bytes && y < x + a_bytes;
}

// Records a CUDA error as the calling thread's xpir_b200_last_cuda_error().
void note_cuda_error(cudaError_t e);
}  // namespace xpir

namespace xpir {

// A fresh database id (1, 2, ...): captured batches are keyed by it, so a database
// imported at the address of a freed one never replays the freed one's graph.
inline uint64_t next_db_id() {
  static std::atomic<uint64_t> counter{0};
  return ++counter;
}

// Drops the captured batches that read database `db_id` (batch.cu).  The caller holds
// ctx->mu and has synchronised the context's stream.
void drop_plans_of(xpir_b200_ctx *ctx, uint64_t db_id);

// Supplies the workspace of an uncaptured batch: device buffers of at least `a` bytes
// (level replies) and `b` bytes (re-imported level databases), valid in stream order on
// the context's stream until the batch call returns.
typedef std::function<cudaError_t(size_t a, size_t b, void **pa, void **pb)> WorkspaceFn;

// xpir_b200_reply_batch with an optional workspace supplier (null: the context's own
// cached workspaces).  Used by the serving loop to draw workspaces from its budgeted pool.
int reply_batch_impl(xpir_b200_ctx *ctx, xpir_b200_request *reqs, uint32_t count, int use_graph,
                     const WorkspaceFn *workspace);

}  // namespace xpir
