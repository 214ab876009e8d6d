// Reply generation for one recursion level by residue sums and an exact tail
// (residue_sum.cuh): the same replies as the slot-by-slot kernel of reply.cu, bit for bit,
// without its per-slot chain, Shoup factors and Shoup products on all but the last slots.
//
// The columns of a level are its (group, poly) pairs: column j = g*P + cp reads database
// words ((g*n_i + slot)*P + cp)*m*N + ..., and all columns share the query's rows.  One CTA
// owns W coefficients of one modulus, C columns and a run of slots:
//
//   warp 0      TMA producer: per tile of E slots one box per column and one of the query's
//               a/b rows, into an NS-stage ring (slots past the last live element come back
//               as zeros, XPIR's zero padding).
//   the others  one coefficient each, both ciphertext halves of the C columns in registers.
//
// With one run per column the same threads go on with the exact tail and write the reply.
// With several (levels too small to fill the GPU otherwise, or very long ones) each run
// writes its residue, and reply_finish_kernel adds them and runs the tail.
//
// What bounds it: at one column (the 100,000 x 4 KB level: 24 bytes of database and query per
// word) HBM, 1.50 ms against 2.26 slot by slot and a copy of the same bytes 1.505; at several
// columns the multiplier.  On B200 a 32x32+64-bit multiply-add takes four issue cycles of a
// warp scheduler and the additions around it hardly overlap with it: a word and half cost
// four of those and about twelve other instructions (32 cycles), where the slot-by-slot
// kernel spends 56 on a Shoup factor and a Shoup product alone.  1,048,576 x 256 B in 16s:
// level 1 2.47 -> 1.57 ms.  Up to four columns per CTA share the query words' preparation.
//
// What the sums cannot decide sets the query's redo flag, and the caller repeats that query
// slot by slot.  A CTA that finds such a word stops at once, and the query's other CTAs that
// see it, so a query of unreduced words costs one tile.  The other queries go on.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "kernels.h"
#include "modarith.cuh"
#include "residue_sum.cuh"
#include "sm100.cuh"

namespace xpir {
namespace {

constexpr uint32_t kAllTiles = ~0u;
constexpr uint32_t kTopOfP = 0x1fffffffu;  // p >> 32 of every modulus

// A kernel parameter: kept small (16 bytes more took the 1,000 x 12 KB reply from 38.7 to 39.2 us).
struct SumShape {
  uint64_t P, n_i;
  uint64_t cols;      // groups with live elements * P
  uint64_t n_live;    // elements of db; slots past them read as zeros
  uint32_t N, m;
  uint32_t slices;    // m*N / W
  uint32_t col_blocks, ntasks, runs;
  uint32_t n_eff;     // slots with live elements (of a full group)
  uint32_t prefix;    // slots summed; the exact tail takes the rest
  uint32_t idle, pad;  // slots after n_eff: constant import of a zero bit stream, zero words
  const uint64_t *zero_poly;  // [m][N] that constant
  uint64_t *part;     // [task][column][half][run][m][N]
  int *status;        // the redo flags follow it
  int *stop;          // device copies of those: a query's CTAs that see its flag set do no more work
  uint32_t first;     // task 0's place among the flags
  uint32_t spin_limit;    // polls of a wait (read with TEST only, as the next)
  uint32_t issued_tiles;  // tiles the producer issues at most (kAllTiles: all)
};

__host__ __device__ __forceinline__ uint32_t flag_of(uint32_t first, uint32_t task) {
  return first + task < kRedoFlags ? first + task : kRedoFlags - 1;
}

// What a CTA rarely needs, in shared memory instead of registers: the products of four
// columns leave none over.
struct alignas(16) CtaState {
  int quit;       // set: the CTA has given up
  uint32_t flag;  // its query's place among the flags
};

template <int W, int C, int E, int NS>
struct SumCfg {
  static constexpr int kThreads = W + 32;
  static constexpr int kX = C * E * W, kQ = E * 2 * W;  // words per stage
  static constexpr size_t kBytes = (size_t)NS * (kX + kQ) * 8 + 2 * NS * 8 + sizeof(CtaState);
  static_assert(E % 4 == 0 && W % 32 == 0 && W <= 256, "tile shape");
};

// Waits for a phase; false after `limit` polls or when the CTA has given up.
__device__ __forceinline__ bool wait_or_quit(uint64_t *bar, uint32_t parity, volatile CtaState *state, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (state->quit) return false;
  }
  return false;
}

// One chain whose candidates did not meet in the tail: from kBackSlots before it (or from
// the first slot).  residue: of the prefix.  False when they do not meet there either.
__device__ __noinline__ bool chain_again(const ReplyTask &task, const SumShape &sh, uint64_t j, uint32_t h, uint32_t c,
                                         uint64_t at, uint64_t residue, uint64_t p, uint64_t np, uint32_t delta,
                                         uint64_t *rop) {
  const uint64_t mN = (uint64_t)sh.m * sh.N, g = j / sh.P, cp = j - g * sh.P;
  const uint32_t from = sh.prefix > kBackSlots ? sh.prefix - kBackSlots : 0;
  auto term = [&](uint32_t e) -> uint64_t {
    if (g * sh.n_i + e >= sh.n_live) return 0;
    const uint64_t x = task.db[((g * sh.n_i + e) * sh.P + cp) * mN + at], y = task.query[(2ull * e + h) * mN + at];
    return shoup_lazy_np(x, y, shoup_factor8_np(y, p, np, delta), np);
  };
  ExactTail s{0, 0, 0};
  if (from) {
    s = ExactTail{residue, kMaxAbove, 0};
    for (uint32_t e = from; e < sh.prefix; e++) s.rop = residue_before(s.rop, term(e), p);
  }
  for (uint32_t e = from; e < sh.n_eff; e++) tail_step(s, term(e), p);
  *rop = s.rop;
  return s.above == 0 && (!from || tail_in_range(s, kMaxAbove));
}

// TEST: with the wait test's limit and withheld tile (xpir_b200_ctx_set_wait_test), in kernels of
// their own: as variables of the one kernel they cost it up to 1.6 % (a batch of three queries,
// 131 x 139 slots, 17,862 x 717 B: 699 us, without them 688; 65,536 x 8 KB, 256 x 256 slots from
// host memory: 1,023 and 1,016).
template <int W, int C, int E, int NS, bool ONE, bool TEST>
__device__ __forceinline__ void sum_tile(const ReplyTask &task, const uint32_t task_id, const uint32_t slice,
                                         const uint32_t cb, const uint32_t run, const SumShape &sh,
                                         const DevModuli &dm) {
  using S = SumCfg<W, C, E, NS>;
  extern __shared__ __align__(128) uint64_t sm[];
  uint64_t *xs = sm;                 // [NS][C][E][W]
  uint64_t *qs = xs + NS * S::kX;    // [NS][E][2][W]
  uint64_t *full = qs + NS * S::kQ, *empty = full + NS;
  volatile CtaState *state = (volatile CtaState *)(empty + NS);

  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t per_mod = sh.N / W;
  const uint32_t c = slice / per_mod, k0 = (slice - c * per_mod) * W;
  // The prefix's tiles in `runs` equal parts.
  const uint32_t sum_all = sh.prefix / E;
  const uint32_t s0 = (uint32_t)((uint64_t)sum_all * run / sh.runs) * E;
  const uint32_t sum_end = (uint32_t)((uint64_t)sum_all * (run + 1) / sh.runs) * E;
  const uint32_t end = ONE ? sh.n_eff : sum_end;
  const uint32_t tiles = (end - s0 + E - 1) / E;

  const uint32_t limit = TEST ? sh.spin_limit : kSpinLimit;
  if constexpr (!ONE) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (threadIdx.x == 0) {
    state->quit = 0;
    state->flag = flag_of(sh.first, task_id);
    for (int s = 0; s < NS; s++) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, W / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&task.tm_db);
      tma_prefetch_desc(&task.tm_q);
      int row[C], poly[C];
#pragma unroll
      for (int i = 0; i < C; i++) {
        const uint64_t j = min((uint64_t)cb * C + i, sh.cols - 1);
        const uint64_t g = j / sh.P;
        row[i] = (int)(g * sh.n_i);
        poly[i] = (int)(j - g * sh.P);
      }
      uint32_t t = 0, st = 0, phase = 1;
      for (; t < tiles; ++t) {
        if (state->quit) break;
        if (TEST && t == sh.issued_tiles) break;
        if (t % 64 == (uint32_t)NS && *(volatile int *)(sh.stop + state->flag)) {
          state->quit = 1;
          *(volatile int *)(sh.status + 1 + state->flag) = 1;  // also after a call that failed before it cleared the flag
          __threadfence_system();
          break;
        }
        if (t >= (uint32_t)NS && !wait_or_quit(empty + st, phase, state, limit)) break;
        mbar_arrive_expect_tx(full + st, (uint32_t)((S::kX + S::kQ) * 8));
        const int slot = (int)(s0 + t * E);
#pragma unroll
        for (int i = 0; i < C; i++)
          tma_load_4d(xs + st * S::kX + i * E * W, &task.tm_db, (int)k0, (int)c, poly[i], row[i] + slot, full + st);
        tma_load_4d(qs + st * S::kQ, &task.tm_q, (int)k0, (int)c, 0, slot, full + st);
        if (++st == NS) {
          st = 0;
          phase ^= 1;
        }
      }
      // Every issued copy must have landed before the CTA exits.
      const uint32_t first = t > (uint32_t)NS ? t - NS : 0;
      for (uint32_t u = first; u < t; ++u) mbar_wait(full + (u % NS), (u / NS) & 1);
    }
    return;
  }

  const uint32_t k = threadIdx.x - 32;
  const uint64_t p = dm.p[c], np = opaque(0 - p);
  const uint32_t delta = (uint32_t)dm.shoup_delta[c], d64 = delta * 8;
  SumAcc acc[2][C];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int i = 0; i < C; i++) sum_clear(acc[h][i], ONE ? 0 : kBoundStart);
  bool bad = false, late = false;
  const uint32_t sum_tiles = (sum_end - s0) / E;
  uint32_t t = 0, st = 0, phase = 0;
  // Waits for tile t; false (in the whole warp) when it must stop.
  auto tile_ready = [&]() -> bool {
    const bool ok = mbar_try_wait(full + st, phase) || wait_or_quit(full + st, phase, state, limit);
    if (!__any_sync(~0u, bad || !ok)) return true;
    late = !__all_sync(~0u, ok);
    bad = __any_sync(~0u, bad);
    return false;
  };
  auto tile_done = [&] {
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + st);
    if (++st == NS) {
      st = 0;
      phase ^= 1;
    }
  };
  for (; t < sum_tiles && tile_ready(); ++t) {
    const uint64_t *xst = xs + st * S::kX + k, *qst = qs + st * S::kQ + k;
    int32_t peak = 0;
#pragma unroll
    for (int e = 0; e < E; e += 4) {
      uint64_t x[C][4];
      int32_t step[C];
#pragma unroll
      for (int i = 0; i < C; i++) {
        uint32_t x1 = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
          x[i][r] = xst[(i * E + e + r) * W];
          x1 += (uint32_t)(x[i][r] >> 32);
        }
        step[i] = sum_block(x1);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint64_t y[4];
        SumWord w[4];
        uint32_t top = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
          y[r] = qst[((e + r) * 2 + h) * W];
          w[r] = sum_word(y[r], d64);
          top = max(top, (uint32_t)(y[r] >> 32));
        }
        if (top >= kTopOfP)  // rarely reached by a word below p
          bad |= y[0] >= p || y[1] >= p || y[2] >= p || y[3] >= p;
#pragma unroll
        for (int i = 0; i < C; i++) {
          uint32_t v[4];
#pragma unroll
          for (int r = 0; r < 4; r++) v[r] = sum_slot(acc[h][i], x[i][r], w[r]);
          acc[h][i].bound = sum_bound(acc[h][i].bound + step[i], v);
          peak = max(peak, acc[h][i].bound);
        }
      }
    }
    bad |= peak > kBoundMax;
    tile_done();
  }
  const uint64_t mN = (uint64_t)sh.m * sh.N;
  const uint64_t at = (uint64_t)c * sh.N + k0 + k;
  if (!bad && !late && sum_tiles > 0) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < C; i++) bad |= acc[h][i].bound > kBoundStart;
  }
  if constexpr (ONE) {
    ExactTail tail[2][C];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < C; i++)
        tail[h][i] = sum_tiles ? ExactTail{sum_residue(acc[h][i], p, np, delta), sum_above(acc[h][i].bound), 0}
                               : ExactTail{0, 0, 0};
    for (; t < tiles && !late && tile_ready(); ++t) {
      const uint64_t *xst = xs + st * S::kX + k, *qst = qs + st * S::kQ + k;
      const uint32_t left = min((uint32_t)E, end - (s0 + t * E));
      for (uint32_t e = 0; e < left; e++) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint64_t y = qst[(e * 2 + h) * W];
          if (sum_tiles) bad |= y >= p;
          const uint64_t ys = shoup_factor8_np(y, p, np, delta);
#pragma unroll
          for (int i = 0; i < C; i++) tail_step(tail[h][i], shoup_lazy_np(xst[(i * E + e) * W], y, ys, np), p);
        }
      }
      tile_done();
    }
    if (!bad && !late) {
      const bool zero_p = sh.idle && sh.zero_poly[at] != 0;
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < C; i++) {
          const uint64_t j = (uint64_t)cb * C + i;
          if (j >= sh.cols) continue;
          uint64_t rop = tail[h][i].rop;
          if (sum_tiles) {
            bad |= !tail_in_range(tail[h][i], kRunAbove);
            if (tail[h][i].above)
              bad |= !chain_again(task, sh, j, h, c, at, sum_residue(acc[h][i], p, np, delta), p, np, delta, &rop);
          }
          task.out[(j * 2 + h) * mN + at] = zero_steps(rop, (uint64_t)(zero_p ? 0 : sh.idle) + sh.pad, p);
        }
    }
  } else if (!bad && !late) {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < C; i++) {
        const uint64_t j = (uint64_t)cb * C + i;
        if (j < sh.cols)
          sh.part[((((uint64_t)task_id * sh.cols + j) * 2 + h) * sh.runs + run) * mN + at] =
              sum_residue(acc[h][i], p, np, delta) | (uint64_t)sum_above(acc[h][i].bound) << 61;
      }
  }
  if (bad) {
    state->quit = 1;
    *(volatile int *)(sh.stop + state->flag) = 1;
    *(volatile int *)(sh.status + 1 + state->flag) = 1;
  }
  if (late && !state->quit) *(volatile int *)sh.status = kStatusWaitTimeout;
  if (bad || late) __threadfence_system();
}

// Block order: the column blocks of a slice run side by side (they read the same query rows),
// then the tasks (the same database rows), then the slices.  With the slices first the query
// came from HBM once per few column blocks: 1,048,576 x 256 B 1904 us, so 1814; a batch of
// eight 5.26 and 5.06 ms.
__device__ __forceinline__ void decode_block(const SumShape &sh, uint32_t *slice, uint32_t *task, uint32_t *cb,
                                             uint32_t *run) {
  uint32_t id = blockIdx.x;
  *cb = id % sh.col_blocks;
  id /= sh.col_blocks;
  *task = id % sh.ntasks;
  id /= sh.ntasks;
  *slice = id % sh.slices;
  *run = id / sh.slices;
}

// One query: its task by value (tasks null).  Several: a table in global memory.
template <int W, int C, int E, int NS, bool ONE, int MINB, bool TEST>
__global__ void __launch_bounds__(SumCfg<W, C, E, NS>::kThreads, MINB)
    reply_sum_kernel(const __grid_constant__ ReplyTask one, const ReplyTask *__restrict__ tasks, const SumShape sh,
                     const DevModuli dm) {
  uint32_t slice, tk, cb, run;
  decode_block(sh, &slice, &tk, &cb, &run);
  sum_tile<W, C, E, NS, ONE, TEST>(tasks ? tasks[tk] : one, tk, slice, cb, run, sh, dm);
}

// Adds the runs' residues of one column's kFinishCoefs coefficients and runs the exact
// tail: all threads compute the tail's terms, then one thread per (half, coefficient) steps
// through them.  Grid: x = coefficient slice, y = column, z = task.
constexpr int kFinishCoefs = 32, kFinishThreads = 256, kMaxTail = 24;

__device__ __forceinline__ void finish_tile(const ReplyTask &task, const SumShape &sh, const DevModuli &dm) {
  __shared__ uint64_t terms[kMaxTail][2][kFinishCoefs];
  __shared__ uint64_t sums[kFinishThreads / (2 * kFinishCoefs)][2][kFinishCoefs];
  __shared__ uint32_t above[2][kFinishCoefs];
  const uint64_t mN = (uint64_t)sh.m * sh.N, j = blockIdx.y;
  const uint64_t at0 = (uint64_t)blockIdx.x * kFinishCoefs;
  const uint32_t c = (uint32_t)(at0 / sh.N);
  const uint64_t p = dm.p[c], np = opaque(0 - p);
  const uint32_t delta = (uint32_t)dm.shoup_delta[c];
  const uint32_t k = threadIdx.x % kFinishCoefs, w = threadIdx.x / kFinishCoefs;
  const uint32_t tail = sh.n_eff - sh.prefix;
  const uint64_t g = j / sh.P, cp = j - g * sh.P;
  const uint64_t *x = task.db + ((g * sh.n_i + sh.prefix) * sh.P + cp) * mN + at0 + k;
  const uint64_t *q = task.query + (uint64_t)sh.prefix * 2 * mN + at0 + k;
  bool bad = false;
  // The terms do not depend on the runs: they are computed while the last of them finish.
  for (uint32_t e = w; e < tail; e += kFinishThreads / kFinishCoefs) {
    const uint64_t ya = q[(2ull * e) * mN], yb = q[(2ull * e + 1) * mN];
    const uint64_t xv = g * sh.n_i + sh.prefix + e < sh.n_live ? x[(uint64_t)e * sh.P * mN] : 0;
    bad |= ya >= p || yb >= p;
    terms[e][0][k] = shoup_lazy_np(xv, ya, shoup_factor8_np(ya, p, np, delta), np);
    terms[e][1][k] = shoup_lazy_np(xv, yb, shoup_factor8_np(yb, p, np, delta), np);
  }
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  {
    const uint32_t h = w & 1;
    const uint64_t *part = sh.part + (((uint64_t)blockIdx.z * sh.cols + j) * 2 + h) * sh.runs * mN + at0 + k;
    uint64_t r = 0;
    for (uint32_t u = w / 2; u < sh.runs; u += kFinishThreads / (2 * kFinishCoefs)) {
      const uint64_t v = part[(uint64_t)u * mN];
      if (u + 1 == sh.runs) above[h][k] = (uint32_t)(v >> 61);
      r += v & ((1ull << 61) - 1);
      r = r >= p ? r - p : r;
    }
    sums[w / 2][h][k] = r;
  }
  __syncthreads();
  if (w < 2) {
    uint64_t r = 0;
#pragma unroll
    for (int u = 0; u < kFinishThreads / (2 * kFinishCoefs); u++) {
      r += sums[u][w][k];
      r = r >= p ? r - p : r;
    }
    ExactTail s{r, above[w][k], 0};
    for (uint32_t e = 0; e < tail; e++) tail_step(s, terms[e][w][k], p);
    bad |= !tail_in_range(s, kRunAbove);
    if (s.above) bad |= !chain_again(task, sh, j, w, c, at0 + k, r, p, np, delta, &s.rop);
    const bool zero_p = sh.idle && sh.zero_poly[at0 + k] != 0;
    task.out[(j * 2 + w) * mN + at0 + k] = zero_steps(s.rop, (uint64_t)(zero_p ? 0 : sh.idle) + sh.pad, p);
  }
  if (bad) {
    *(volatile int *)(sh.status + 1 + flag_of(sh.first, blockIdx.z)) = 1;
    __threadfence_system();
  }
}

__global__ void __launch_bounds__(kFinishThreads)
    reply_finish_kernel(const __grid_constant__ ReplyTask one, const ReplyTask *__restrict__ tasks, const SumShape sh,
                        const DevModuli dm) {
  finish_tile(tasks ? tasks[blockIdx.z] : one, sh, dm);
}

// Query words of slots that meet a constant import must lie in [1, p): then a constant p
// leaves the chain as it is.  words: slots * 2*m*N, a multiple of 2.
__global__ void __launch_bounds__(256) query_range_kernel(const ulonglong2 *__restrict__ q, uint64_t pairs, uint32_t N,
                                                          uint32_t m, const DevModuli dm, int *redo) {
  bool bad = false;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
#pragma unroll 4
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += stride) {
    const ulonglong2 v = q[i];
    const uint64_t p1 = dm.p[(uint32_t)((2 * i / N) % m)] - 1;
    bad |= v.x - 1 >= p1 || v.y - 1 >= p1;
  }
  if (bad) {
    *(volatile int *)redo = 1;
    __threadfence_system();
  }
}

typedef cudaError_t (*SumFn)(const ReplyTask &, const ReplyTask *, const SumShape &, const DevModuli &, cudaStream_t);
struct SumEntry {
  int W, C, E, NS, ctas;  // ctas: resident per SM
  SumFn one, runs;
  const void *kernels[2];
  size_t bytes;  // their dynamic shared memory
};

template <int W, int C, int E, int NS, bool ONE, int MINB>
cudaError_t launch_sum(const ReplyTask &one, const ReplyTask *dev, const SumShape &sh, const DevModuli &dm,
                       cudaStream_t stream) {
  using S = SumCfg<W, C, E, NS>;
  const uint64_t blocks = (uint64_t)sh.slices * sh.ntasks * sh.col_blocks * sh.runs;
  if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
  auto kern = reply_sum_kernel<W, C, E, NS, ONE, MINB, false>;
  if (sh.spin_limit != kSpinLimit || sh.issued_tiles != kAllTiles) {  // loaded when first asked for
    kern = reply_sum_kernel<W, C, E, NS, ONE, MINB, true>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kBytes);
    if (e != cudaSuccess) return e;
  }
  kern<<<(unsigned)blocks, S::kThreads, S::kBytes, stream>>>(one, dev, sh, dm);
  return cudaGetLastError();
}

#define XPIR_SUM(W, C, E, NS, MINB)                                                                 \
  {                                                                                                 \
    W, C, E, NS, MINB, &launch_sum<W, C, E, NS, true, MINB>, &launch_sum<W, C, E, NS, false, MINB>, \
    {                                                                                               \
      (const void *)reply_sum_kernel<W, C, E, NS, true, MINB, false>,                               \
          (const void *)reply_sum_kernel<W, C, E, NS, false, MINB, false>                           \
    }, SumCfg<W, C, E, NS>::kBytes                                                                  \
  }

constexpr uint32_t kMaxRuns = 64;
constexpr uint64_t kLongSlots = 128;

// By column count.  Three CTAs of four warps per SM hide the TMA's latency with one and two
// columns; their rings (72 and 64 KB) and registers fill an SM.  Three and four columns take
// 80 and 96 KB and 168 registers: two CTAs.
const SumEntry kSums[] = {
    XPIR_SUM(128, 1, 8, 3, 3),
    XPIR_SUM(128, 2, 8, 2, 3),
    XPIR_SUM(128, 3, 8, 2, 2),
    XPIR_SUM(128, 4, 8, 2, 2),
};

// Columns per CTA.  Four share the query words' preparation best, but leave too few CTAs and a
// longer tail on small or short levels (us with two / four: 1,024 slots of 64 groups, N=4096
// 2085 / 1903; 61 slots of 110 columns 161 / 174; 1,000 slots of 7 polys, N=1024 39 / 43).
const SumEntry &sum_entry(uint32_t mN, uint64_t cols, uint64_t n_eff, uint64_t ntasks) {
  if (cols == 3 && n_eff >= kLongSlots) return kSums[2];
  const uint64_t ctas4 = mN / 128 * ((cols + 3) / 4) * ntasks;
  if (cols >= 4 && n_eff >= kLongSlots && ctas4 >= 592) return kSums[3];
  return kSums[cols == 1 ? 0 : 1];
}


int sum_sm_count() {
  static int cache[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}

bool encode_sum_task(int W, int E, const uint64_t *db, const uint64_t *query, uint64_t n_live, uint64_t P, uint64_t n_i,
                     const ParamSet &ps, uint64_t *out, ReplyTask *t) {
  const uint64_t N = ps.N, m = ps.m;
  const uint64_t db_dims[4] = {N, m, P, n_live}, db_strides[3] = {N * 8, m * N * 8, P * m * N * 8};
  const uint32_t db_box[4] = {(uint32_t)W, 1, 1, (uint32_t)E};
  const uint64_t q_dims[4] = {N, m, 2, n_i}, q_strides[3] = {N * 8, m * N * 8, 2 * m * N * 8};
  const uint32_t q_box[4] = {(uint32_t)W, 1, 2, (uint32_t)E};
  t->out = out;
  t->db = db;
  t->query = query;
  return encode_tensor_map_u64_4d(&t->tm_db, db, db_dims, db_strides, db_box) &&
         encode_tensor_map_u64_4d(&t->tm_q, query, q_dims, q_strides, q_box);
}

}  // namespace

// Where the residue sums are the faster way.  Both kernels timed on B200 (us slot by slot /
// here, event pairs):  chains long enough to be cut into runs (1,000 slots of one poly, N=1024
// 23.8 / 18.8, N=2048 32.7 / 25.9; 500 slots 17.4 / 18.7), and shorter ones where one run per
// column already fills the GPU: with several polys per element from 250 CTAs (N=4096, 3
// moduli, 6 polys, 16 slots 22.9 / 14.7), with one poly, where the slot-by-slot kernel shares
// its factors among groups, from 500 (N=2048, 20 slots of 40 groups 30.2 / 27.5, of 20 groups
// 20.3 / 22.2) or from 250 with 96 slots (100 slots of 30 groups 61.1 / 51.1); one group of
// 100 slots 16.4 / 25.3.  And any level whose elements are mostly idle, which the
// slot-by-slot kernel multiplies and this one skips.
bool sum_level_supported(const ParamSet &ps, uint64_t n_real, uint64_t n_live, uint64_t P, uint64_t n_i,
                         uint64_t groups, uint64_t ntasks) {
  const uint64_t live_groups = active_groups(n_live, n_i, groups);
  const uint64_t n_eff = std::min(n_i, n_live);
  if (live_groups == 0 || ps.N % 128 != 0 || n_eff >= (1u << 30) || live_groups * P >= (1u << 30) ||
      !reply_level_supported(ps, n_live, n_i, live_groups) || ntasks > 65535 || live_groups * P > 65535)
    return false;
  const uint64_t cols = live_groups * P;  // in CTAs of 128 coefficients and two columns
  const uint64_t ctas = (uint64_t)ps.m * ps.N / 128 * ((cols + 1) / 2) * ntasks;
  if (n_live * 2 < n_real) return true;
  return n_eff >= 600 || (n_eff >= kTailSlots && ctas >= (P > 1 ? 250u : 500u)) || (n_eff >= 96 && ctas >= 250);
}

cudaError_t launch_sum_level(const SumLevelArgs &a, const uint64_t *const *db, const uint64_t *const *query,
                             uint64_t *const *out, uint32_t ntasks, const ParamSet &ps, const DevModuli &dm,
                             ReplyTask *host_tasks, ReplyTask *dev_tasks, cudaStream_t stream, uint32_t *launches) {
  const uint64_t live_groups = active_groups(a.n_live, a.n_i, a.n_groups);
  const uint64_t mN = (uint64_t)ps.m * ps.N, ct_words = 2 * mN;
  if (live_groups < a.n_groups && a.write_idle)
    for (uint32_t t = 0; t < ntasks; t++) {
      cudaError_t e = cudaMemsetAsync(out[t] + live_groups * a.P * ct_words, 0,
                                      (a.n_groups - live_groups) * a.P * ct_words * 8, stream);
      if (e != cudaSuccess) return e;
    }
  SumShape sh{};
  sh.P = a.P;
  sh.n_i = a.n_i;
  sh.N = ps.N;
  sh.m = ps.m;
  sh.ntasks = ntasks;
  sh.zero_poly = a.zero_poly;
  sh.part = a.part;
  sh.status = a.status;
  sh.stop = a.stop;
  sh.first = a.first;
  sh.spin_limit = a.wait_test.spin_limit ? a.wait_test.spin_limit : kSpinLimit;
  sh.issued_tiles = a.wait_test.withhold_tile < 0 ? kAllTiles : (uint32_t)a.wait_test.withhold_tile;
  // Elements past n_live (idle): the group that holds the first of them is a launch of its
  // own when there are others, since its chain ends at another slot.
  const bool idle = a.n_live < a.n_real;
  const uint64_t whole = idle && live_groups > 1 && a.n_live % a.n_i != 0 ? live_groups - 1 : live_groups;
  if (idle) {
    // Query rows that idle slots read: all of them when a whole group is idle.
    const uint64_t real_groups = active_groups(a.n_real, a.n_i, a.n_groups);
    const uint64_t from = real_groups > live_groups || a.n_live % a.n_i == 0 ? 0 : a.n_live % a.n_i;
    const uint64_t to = real_groups > live_groups ? a.n_i : std::min(a.n_i, a.n_real - (live_groups - 1) * a.n_i);
    const uint64_t pairs = (to - from) * mN;
    for (uint32_t t = 0; t < ntasks && pairs; t++) {
      const unsigned blocks = (unsigned)std::min<uint64_t>((pairs + 1023) / 1024, 8ull * sum_sm_count());
      query_range_kernel<<<blocks, 256, 0, stream>>>((const ulonglong2 *)(query[t] + from * ct_words), pairs, ps.N,
                                                     ps.m, dm, a.status + 1 + flag_of(a.first, t));
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      if (launches) (*launches)++;
    }
  }
  for (uint64_t g0 = 0; g0 < live_groups; g0 += whole) {
    const uint64_t groups = g0 == 0 ? whole : 1;
    const uint64_t live = a.n_live - g0 * a.n_i;  // of this launch's groups and those after
    const uint64_t real = a.n_real - g0 * a.n_i;
    sh.cols = groups * a.P;
    sh.n_live = live;
    sh.n_eff = (uint32_t)std::min(a.n_i, live);
    const uint64_t last_real = groups == 1 ? std::min(a.n_i, real) : a.n_i;
    sh.idle = (uint32_t)(last_real - sh.n_eff);  // n_i < 2^31 (reply_level_supported)
    sh.pad = (uint32_t)(a.n_i - last_real);
    const SumEntry &entry = sum_entry((uint32_t)mN, sh.cols, sh.n_eff, ntasks);
    sh.slices = (uint32_t)(mN / entry.W);
    sh.col_blocks = (uint32_t)((sh.cols + entry.C - 1) / entry.C);
    sh.prefix = sh.n_eff > kTailSlots ? (sh.n_eff - kTailSlots) / entry.E * entry.E : 0;
    // Runs: enough CTAs for every SM, in whole waves where the level is long enough.
    const uint64_t base = (uint64_t)sh.slices * sh.col_blocks * ntasks, room = (uint64_t)sum_sm_count() * entry.ctas;
    const uint64_t part_runs = a.part_words / (std::max<uint64_t>(1, ntasks * sh.cols) * ct_words);
    const uint64_t max_runs = std::min<uint64_t>({kMaxRuns, sh.prefix / (kMinRunSlots + entry.E), part_runs});
    uint64_t runs = 1;
    if (base < 4 * room && max_runs > 1) {
      double best = 0;
      for (uint64_t r = 1; r <= max_runs; r++) {
        const uint64_t waves = (base * r + room - 1) / room;
        if (waves > 8 && r > 1) break;
        const double use = (double)(base * r) / (double)(waves * room);
        if (use > best * 1.02) {
          best = use;
          runs = r;
        }
      }
    }
    sh.runs = (uint32_t)runs;
    // The second launch has table entries of its own: the first one's copy may be in flight.
    ReplyTask *ht = host_tasks + (g0 ? ntasks : 0), *dt = ntasks > 1 ? dev_tasks + (g0 ? ntasks : 0) : nullptr;
    for (uint32_t t = 0; t < ntasks; t++)
      if (!encode_sum_task(entry.W, entry.E, db[t] + g0 * a.n_i * a.P * mN, query[t], live, a.P, a.n_i, ps,
                           out[t] + g0 * a.P * ct_words, ht + t))
        return cudaErrorInvalidValue;
    cudaError_t e;
    if (dt) {
      e = cudaMemcpyAsync(dt, ht, ntasks * sizeof(ReplyTask), cudaMemcpyHostToDevice, stream);
      if (e != cudaSuccess) return e;
    }
    e = (runs > 1 ? entry.runs : entry.one)(*ht, dt, sh, dm, stream);
    if (e != cudaSuccess) return e;
    if (runs > 1) {
      cudaLaunchAttribute early{};  // may start before the runs end, and waits for them itself
      early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      early.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)(mN / kFinishCoefs), (unsigned)sh.cols, ntasks);
      cfg.blockDim = dim3(kFinishThreads);
      cfg.stream = stream;
      cfg.attrs = &early;
      cfg.numAttrs = 1;
      e = cudaLaunchKernelEx(&cfg, reply_finish_kernel, *ht, (const ReplyTask *)dt, sh, dm);
      if (e != cudaSuccess) return e;
    }
    if (launches) *launches += runs > 1 ? 2 : 1;
    if (groups == live_groups || g0 > 0) break;
  }
  return cudaSuccess;
}

cudaError_t preload_sum_kernels() {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, reply_finish_kernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, query_range_kernel);
  for (const SumEntry &s : kSums)
    for (const void *k : s.kernels)
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.bytes);
  return e;
}

}  // namespace xpir
