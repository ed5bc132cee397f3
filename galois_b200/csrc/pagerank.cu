// PageRank: pull-topological, pull-residual and residual-push.
//
// Reference semantics (lonestar/analytics/cpu/pagerank):
//   pull-topological  PageRank-pull.cpp:196-251 over the TRANSPOSED graph:
//                     value = 1/n; nout = in-degree of the stored graph
//                     (computeOutDeg :90-122); per iteration
//                     value[v] = alpha * sum_{u in edges(v)} value[u]/nout[u]
//                                + (1-alpha)/n,
//                     stop when sum |delta| <= tol or at maxIterations.
//                     The CPU code updates in place (schedule-dependent); the
//                     device runs the Jacobi form, which the FP64 oracle
//                     restates.
//   pull-residual     PageRank-pull.cpp:132-190 (delta/residual rounds).
//   residual push     PageRank-push.cpp:103-188 (Sync): value 0, residual
//                     1-alpha; active vertices over tol absorb their residual
//                     and push residual*alpha/outdeg along out-edges; a
//                     vertex is activated when its residual crosses tol.
//                     PageRank-push.cpp:68-101 (Async, the app's default):
//                     the same operator over a worklist with no rounds -- a
//                     vertex is processed when it is taken, absorbing the
//                     residual accumulated until then (exchange with 0), and
//                     pushed again when an add lifts its residual from below
//                     tol to tol or above.
//
// B200 design: one cooperative persistent launch per solve.  Pull iterations
// use the cached all-vertex sweep schedule (sweep.cuh): 32 consecutive
// vertices per warp, eight lanes to a row (chunk_row_sums), heavy vertices as
// tiles whose partial sums meet in an accumulator, a contribution array
// c[u] = value[u]/nout[u] (SoA, double-buffered) so each arc costs one 4-byte
// column read and one 4-byte gather, and the L1 change reduced in fp64.  In
// file order the columns of a power-law graph are renamed by falling in-degree
// (ensure_hot).  On a degree-ordered graph both pull variants run over a
// binned layout instead (pr_pull_binned, below).  Residual push (Sync) reuses
// the frontier queues (frontier.cuh); Async runs over the device worklist
// (gb_worklist.cuh): a warp keeps working on the vertices it activated itself,
// surplus goes to the ring, and the launch ends when the worklist's work count
// reaches zero.

#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "device_common.cuh"
#include "device_graph.cuh"
#include "frontier.cuh"
#include "gb_worklist.cuh"
#include "sweep.cuh"

#include <cstring>

// The binned layout of a degree-ordered graph's arcs for the PageRank pull
// (pr_pull_binned), cached in the graph handle.
struct PrBins {
  void* mem = nullptr;       // the arrays but rdst
  uint16_t* src = nullptr;
  uint8_t* flag = nullptr;
  uint32_t* crun = nullptr;
  uint32_t* rdst = nullptr;  // per run: its destination
  uint4* tasks = nullptr;
  uint32_t ntasks = 0;
};

// The row sweeps' renamed columns of a graph in file order (ensure_hot), cached
// in the graph handle.
struct PrHot {
  uint32_t* col = nullptr;   // [m] the columns as slots, then rank (nullptr: not renamed)
  uint32_t* rank = nullptr;  // [n] vertex -> slot of its contribution
};

namespace gb {

void free_pr_hot(gb_graph* g) {
  if (!g->prh) return;
  cudaFree(g->prh->col);
  delete g->prh;
  g->prh = nullptr;
}

void free_pr_bins(gb_graph* g) {
  if (!g->prb) return;
  cudaFree(g->prb->mem);
  cudaFree(g->prb->rdst);
  delete g->prb;
  g->prb = nullptr;
}

namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kL1Slots = 32;  // the per-iteration L1 sum is spread over this many words

struct PrCtl {
  GridBar bar;
  int err;
  uint32_t iters;
  double l1[3][kL1Slots];  // per-iteration L1 change, one slot per (CTA % kL1Slots)
  uint32_t linf[3];        // max |delta| as float bits (non-negative floats order as uints)
  uint32_t active[3];
  uint32_t pad;
  FrontierCounters fc[3];
  unsigned long long pushes;
  unsigned long long absorbs;  // Async push: residuals taken
  uint32_t task_next[2];       // binned pull: next gather task (iteration parity)
};

struct PrArgs {
  const uint64_t* __restrict__ offs;
  const uint32_t* __restrict__ col;
  const uint32_t* __restrict__ nout;
  uint32_t n;
  float alpha;
  float base;
  float tol;
  uint32_t max_iter;
  float init;  // initial rank (1/n for the lonestar app)
  int linf;    // 1: stop on max |delta| (python/galois/_pagerank.pyx:114-139)
  float* value;
  float* c[2];
  float* acc;   // per-row partial sums of heavy rows (and flat-swept light rows)
  float* acc2;  // the alternate accumulator (pull kernels): iteration it adds into
                // (it & 1 ? acc2 : acc) and zeroes the other; a plain store to a
                // word the same iteration's atomics just updated stalled (~0.4 ms
                // for 9 M words at RMAT-24), one iteration later it does not
  SweepSched sched;
  PrCtl* ctl;
  // residual variants
  float* residual;
  float* delta;
  uint32_t* active[2];
  uint32_t* stamp;
  FrontierQueues fq;
  uint32_t heavy, tile;
  worklists::Ring ring;  // Async push: the worklist ring
  uint32_t zero_from;  // first vertex of the no-in-arc suffix (degree-ordered graphs), else n
  // flat sweep of the light rows (degree-ordered graphs): arcs [lr_arc0,
  // lr_arc1) in runs of kLightRun; an arc's row is lr_runrow[run] +
  // lr_rowd[arc - lr_arc0] (a run spans at most kLightRun rows, so the
  // offset fits a byte: a quarter of the bytes of a row id per arc)
  const uint32_t* __restrict__ lr_runrow;
  const uint8_t* __restrict__ lr_rowd;
  uint64_t lr_arc0, lr_arc1;
  // binned pull (degree-ordered graphs, pr_pull_binned)
  const uint16_t* __restrict__ b_src;   // per padded arc: source - block base (kBinPart: padding)
  const uint8_t* __restrict__ b_flag;   // per 8 arcs: which of them start a run
  const uint32_t* __restrict__ b_crun;  // per 256-arc chunk: its first run; then the number of runs
  const uint32_t* __restrict__ b_rdst;  // per run: its destination
  double* hacc;       // binned: sums of the top rows (ids below b_nheavy), [2][b_nheavy], in acc's place
  uint32_t b_nheavy;  // (0: not binned)
  const uint4* __restrict__ b_tasks;    // (block base, sources, chunk begin, chunk end)
  uint32_t b_ntasks;
  const uint32_t* __restrict__ rank;  // row sweeps: slot of a vertex's contribution (nullptr: its id)
};

constexpr int kLightRun = 256;  // arcs per light-row run of pr_pull_flat (32 lanes x 8)

__global__ void count_nout(const uint32_t* __restrict__ col, uint64_t m, uint32_t* nout) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = tid; e < m; e += stride) atomicAdd(&nout[col[e]], 1u);
}

__global__ void pr_pull_init(PrArgs a) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const float init = a.init;  // 1/n: PageRank-pull.cpp:62
  for (uint64_t v = tid; v < a.n; v += stride) {
    a.value[v] = init;
    const uint32_t k = a.nout[v];
    a.c[0][a.rank ? a.rank[v] : v] = k ? init / (float)k : 0.f;
    a.acc[v] = 0.f;
    a.acc2[v] = 0.f;
  }
}

// Segmented (by owner lane) warp reduction of x; returns true on the lane
// that heads its segment, which then holds the segment's sum.
__device__ __forceinline__ bool seg_reduce(bool valid, uint32_t owner, float& x) {
  const uint32_t lane = lane_id();
  const uint32_t key = valid ? owner : 0xFFFFFFFFu;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float y = __shfl_down_sync(kFull, x, off);
    const uint32_t k2 = __shfl_down_sync(kFull, key, off);
    if (lane + off < 32 && k2 == key) x += y;
  }
  const uint32_t kprev = __shfl_up_sync(kFull, key, 1);
  return valid && (lane == 0 || kprev != key);
}

// Sums over the rows of a 32-row chunk whose lanes hold (first arc, arc
// count): four rows at a time, eight lanes each, four columns per lane loaded
// ahead of the four gathers, the next four rows' columns loading meanwhile.
// Returns the lane's own row's sum.  Walking the chunk's arcs 32 at a time
// (owner search and segmented sum, about 80 instructions per 32 arcs) was
// bound by instruction issue; this takes about 20.  Pull-residual, RMAT-21
// directed in file order (32 M arcs): 204 -> 174 us a round, 189 G arcs/s,
// now about the rate of 4-byte gathers from L2.
// gather(u) takes 0xFFFFFFFF for no arc and returns 0 for it.  A chunk of rows
// of at most eight arcs takes a lane per row.
template <class Gather>
__device__ __forceinline__ float chunk_row_sums(const uint32_t* __restrict__ col, uint64_t b, uint32_t d,
                                                Gather&& gather) {
  const uint32_t lane = lane_id(), sub = lane & 7u, grp = lane >> 3;
  if (__reduce_max_sync(kFull, d) <= 8) {
    float x[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) x[j] = gather(j < d ? ldg(col + b + j) : 0xFFFFFFFFu);
    return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  }
  auto load = [&](uint64_t rb, uint32_t rd, uint32_t k, uint32_t (&u)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = k + 8 * j < rd ? ldg(col + rb + k + 8 * j) : 0xFFFFFFFFu;
  };
  auto sum4 = [&](const uint32_t (&u)[4]) {
    float x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = gather(u[j]);
    return (x[0] + x[1]) + (x[2] + x[3]);
  };
  float mine = 0.f;
  uint64_t rb = __shfl_sync(kFull, b, grp);
  uint32_t rd = __shfl_sync(kFull, d, grp);
  uint32_t u[4];
  load(rb, rd, sub, u);
#pragma unroll 1
  for (uint32_t q = 0; q < 8; ++q) {
    const uint64_t nb = __shfl_sync(kFull, b, (4 * q + 4 + grp) & 31);
    uint32_t nd = __shfl_sync(kFull, d, (4 * q + 4 + grp) & 31);
    if (q == 7) nd = 0;
    uint32_t un[4];
    load(nb, nd, sub, un);
    float sum = sum4(u);
    for (uint32_t k = sub + 32; k < rd; k += 32) {
      load(rb, rd, k, u);
      sum += sum4(u);
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    const float got = __shfl_sync(kFull, sum, (lane & 3u) * 8);
    if ((lane >> 2) == q) mine = got;
    rb = nb, rd = nd;
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = un[j];
  }
  return mine;
}

// The sum over one tile [b, e) of a heavy row, by a warp (in every lane):
// 8 column loads per lane per round, the next round's loads issued before
// this round's gathers are summed.
template <class Gather>
__device__ __forceinline__ float tile_row_sum(const uint32_t* __restrict__ col, uint64_t b, uint64_t e,
                                              Gather&& gather) {
  const uint32_t lane = lane_id();
  constexpr int UT = 8;
  uint32_t u[UT];
#pragma unroll
  for (int k = 0; k < UT; ++k) {
    const uint64_t i = b + lane + 32 * k;
    u[k] = i < e ? ldg(col + i) : 0xFFFFFFFFu;
  }
  float sum = 0.f;
  for (uint64_t i0 = b; i0 < e; i0 += 32 * UT) {
    uint32_t un[UT];
#pragma unroll
    for (int k = 0; k < UT; ++k) {
      const uint64_t i = i0 + 32 * UT + lane + 32 * k;
      un[k] = i < e ? ldg(col + i) : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int k = 0; k < UT; ++k) sum += gather(u[k]);
#pragma unroll
    for (int k = 0; k < UT; ++k) u[k] = un[k];
  }
  return warp_sum(sum);
}

// Publish this thread's share of the iteration's L1 / max change: summed per
// CTA in shared memory, then one atomic per CTA into one of kL1Slots words
// (an atomic per warp on one word serialised ~7 K atomics per iteration), the
// max with a read before the atomic.  All threads of the CTA call.
__device__ __forceinline__ void publish_change(PrCtl* ctl, uint32_t slot_set, double my_l1, float my_max,
                                               double* s_l1, uint32_t* s_max) {
  my_l1 = warp_sum(my_l1);
  const uint32_t mbits = __reduce_max_sync(kFull, __float_as_uint(my_max));
  if (lane_id() == 0) {
    if (my_l1 != 0.0) atomicAdd(s_l1, my_l1);
    if (mbits != 0u) atomicMax(s_max, mbits);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*s_l1 != 0.0) atomicAdd(&ctl->l1[slot_set][blockIdx.x % kL1Slots], *s_l1);
    if (*s_max > *reinterpret_cast<volatile uint32_t*>(&ctl->linf[slot_set])) atomicMax(&ctl->linf[slot_set], *s_max);
    *s_l1 = 0.0;
    *s_max = 0u;
  }
}

// The iteration's change after the barrier that follows publish_change: one
// thread per CTA reads the slots and shares the total through shared memory
// (every thread reading them would hammer the same L2 lines).  All threads
// of the CTA call.
__device__ __forceinline__ double read_change(const PrCtl* ctl, uint32_t slot_set, int linf, double* s_total) {
  if (threadIdx.x == 0) {
    double v = 0.0;
    if (linf) {
      v = (double)__uint_as_float(*reinterpret_cast<const volatile uint32_t*>(&ctl->linf[slot_set]));
    } else {
      for (int k = 0; k < kL1Slots; ++k) v += *reinterpret_cast<const volatile double*>(&ctl->l1[slot_set][k]);
    }
    *s_total = v;
  }
  __syncthreads();
  const double v = *s_total;
  __syncthreads();  // s_total is rewritten next iteration
  return v;
}

// Zero the slots of iteration it+1 (by one thread, before that iteration's barrier).
__device__ __forceinline__ void clear_change(PrCtl* ctl, uint32_t slot_set) {
  for (int k = 0; k < kL1Slots; ++k) ctl->l1[slot_set][k] = 0.0;
  ctl->linf[slot_set] = 0u;
}

// Jacobi pull iterations, one cooperative persistent launch.  Shared memory
// holds only the change's totals, so the SM's unified L1/shared array serves as
// L1 for the gathers: the hot contributions sit on few lines (degree order, or
// renamed columns) and stay there.  On a degree-ordered graph the vertices from
// zero_from on have no in-arcs, so after two iterations their rank and
// contribution are constants and their chunks are skipped.
template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) pr_pull_persistent(PrArgs a) {
  __shared__ double s_l1, s_total;
  __shared__ uint32_t s_max;
  if (threadIdx.x == 0) {
    s_l1 = 0.0;
    s_max = 0u;
  }
  __syncthreads();
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)BLOCK + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * BLOCK;
  const uint64_t gwarp = gtid >> 5, nwarps = gthreads >> 5;
  const uint32_t lane = lane_id();
  for (uint32_t it = 0;; ++it) {
    const float* __restrict__ c_in = a.c[it & 1];
    float* __restrict__ c_out = a.c[(it + 1) & 1];
    float* const acc_cur = (it & 1) ? a.acc2 : a.acc;
    float* const acc_nxt = (it & 1) ? a.acc : a.acc2;
    if (gtid == 0) clear_change(ctl, (it + 1) % 3);
    auto gather = [&](uint32_t u) -> float { return u != 0xFFFFFFFFu ? c_in[u] : 0.f; };
    double my_l1 = 0.0;
    float my_max = 0.f;
    auto finish = [&](uint32_t v, float sum) {
      const float value = sum * a.alpha + a.base;  // PageRank-pull.cpp:222
      const float old = a.value[v];
      a.value[v] = value;
      const uint32_t k = a.nout[v];
      c_out[a.rank ? a.rank[v] : v] = k ? value / (float)k : 0.f;
      my_l1 += (double)fabsf(value - old);
      my_max = fmaxf(my_max, fabsf(value - old));
    };
    // Tasks: 32-vertex chunks (a chunk without arcs only finishes its
    // vertices), then heavy-vertex tiles (sweep.cuh's decomposition).
    const uint64_t nchunks = ((uint64_t)(it >= 2 ? a.zero_from : a.n) + 31) >> 5;  // constant tail skipped
    const uint64_t total = nchunks + a.sched.ntiles;
    for (uint64_t t = gwarp; t < total; t += nwarps) {
      if (t < nchunks) {
        const uint64_t v = (t << 5) + lane;
        uint64_t b = 0;
        uint32_t d = 0;
        bool heavy = false;
        if (v < a.n) {
          b = ldg(a.offs + v);
          const uint64_t dd = ldg(a.offs + v + 1) - b;
          heavy = dd > a.sched.heavy;
          d = heavy ? 0u : (uint32_t)dd;
        }
        const float sum = __any_sync(kFull, d != 0) ? chunk_row_sums(a.col, b, d, gather) : 0.f;
        if (v < a.n && !heavy) finish((uint32_t)v, sum);
      } else {
        const uint2 tv = a.sched.tiles[t - nchunks];
        const uint64_t vb = ldg(a.offs + tv.x), ve = ldg(a.offs + tv.x + 1);
        const uint64_t b = vb + (uint64_t)tv.y * a.sched.tile;
        const float sum = tile_row_sum(a.col, b, min(ve, b + a.sched.tile), gather);
        if (lane == 0) atomicAdd(&acc_cur[tv.x], sum);
      }
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    for (uint64_t i = gtid; i < a.sched.nheavy; i += gthreads) {
      const uint32_t v = a.sched.heavy_list[i];
      const float sum = acc_cur[v];
      acc_nxt[v] = 0.f;
      finish(v, sum);
    }
    publish_change(ctl, it % 3, my_l1, my_max, &s_l1, &s_max);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    const double l1 = read_change(ctl, it % 3, a.linf, &s_total);
    if (gtid == 0) ctl->iters = it + 1;
    if (l1 <= (double)a.tol || it + 1 >= a.max_iter) break;  // PageRank-pull.cpp:238-243
  }
}

// Jacobi pull iterations for a degree-ordered graph.  Its heavy rows are the
// ids [0, nheavy) and its light rows follow with falling degree, so the light
// rows' arcs form one contiguous range.  That range is swept flat, like a
// tile: 256 arcs per warp task, 8 column ids and 8 row ids per lane loaded
// together, 8 gathers in flight, a segmented warp sum per 32 arcs and one
// atomicAdd per row segment into acc.  Heavy rows keep their tiles.  A
// coalesced pass over the vertices then finishes every row from acc (rows
// from zero_from on have no in-arcs: constant after two iterations, skipped).
template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) pr_pull_flat(PrArgs a) {
  __shared__ double s_l1, s_total;
  __shared__ uint32_t s_max;
  if (threadIdx.x == 0) {
    s_l1 = 0.0;
    s_max = 0u;
  }
  __syncthreads();
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)BLOCK + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * BLOCK;
  const uint64_t gwarp = gtid >> 5, nwarps = gthreads >> 5;
  const uint32_t lane = lane_id();
  constexpr int UT = 8;
  const uint64_t nruns = (a.lr_arc1 - a.lr_arc0 + 32 * UT - 1) / (32 * UT);
  const uint64_t total = (uint64_t)a.sched.ntiles + nruns;
  for (uint32_t it = 0;; ++it) {
    const float* __restrict__ c_in = a.c[it & 1];
    float* __restrict__ c_out = a.c[(it + 1) & 1];
    float* const acc_cur = (it & 1) ? a.acc2 : a.acc;
    float* const acc_nxt = (it & 1) ? a.acc : a.acc2;
    if (gtid == 0) clear_change(ctl, (it + 1) % 3);
    for (uint64_t t = gwarp; t < total; t += nwarps) {
      if (t < a.sched.ntiles) {
        const uint2 tv = a.sched.tiles[t];
        const uint64_t vb = ldg(a.offs + tv.x), ve = ldg(a.offs + tv.x + 1);
        const uint64_t b = vb + (uint64_t)tv.y * a.sched.tile;
        const float sum = tile_row_sum(a.col, b, min(ve, b + a.sched.tile), [&](uint32_t u) { return u != 0xFFFFFFFFu ? c_in[u] : 0.f; });
        if (lane == 0) atomicAdd(&acc_cur[tv.x], sum);
      } else {
        // one run of 256 arcs of the light rows
        static_assert(32 * UT == kLightRun, "a light run is one warp step of UT arcs per lane");
        const uint64_t run = t - a.sched.ntiles;
        const uint64_t r0 = a.lr_arc0 + run * kLightRun;
        const uint32_t row0 = ldg(a.lr_runrow + run);
        uint32_t u[UT], row[UT];
#pragma unroll
        for (int k = 0; k < UT; ++k) {
          const uint64_t i = r0 + lane + 32 * k;
          const bool ok = i < a.lr_arc1;
          u[k] = ok ? ldg(a.col + i) : 0u;
          row[k] = ok ? row0 + (uint32_t)__ldg(a.lr_rowd + (i - a.lr_arc0)) : 0xFFFFFFFFu;
        }
        float x[UT];
#pragma unroll
        for (int k = 0; k < UT; ++k) x[k] = row[k] != 0xFFFFFFFFu ? c_in[u[k]] : 0.f;
#pragma unroll
        for (int k = 0; k < UT; ++k) {
          if (seg_reduce(row[k] != 0xFFFFFFFFu, row[k], x[k])) atomicAdd(&acc_cur[row[k]], x[k]);
        }
      }
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    double my_l1 = 0.0;
    float my_max = 0.f;
    const uint32_t vend = it >= 2 ? a.zero_from : a.n;  // constant tail skipped
    for (uint64_t v = gtid; v < vend; v += gthreads) {
      const float sum = acc_cur[v];
      acc_nxt[v] = 0.f;
      const float value = sum * a.alpha + a.base;  // PageRank-pull.cpp:222
      const float old = a.value[v];
      a.value[v] = value;
      const uint32_t k = a.nout[v];
      c_out[v] = k ? value / (float)k : 0.f;
      my_l1 += (double)fabsf(value - old);
      my_max = fmaxf(my_max, fabsf(value - old));
    }
    publish_change(ctl, it % 3, my_l1, my_max, &s_l1, &s_max);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    const double l1 = read_change(ctl, it % 3, a.linf, &s_total);
    if (gtid == 0) ctl->iters = it + 1;
    if (l1 <= (double)a.tol || it + 1 >= a.max_iter) break;  // PageRank-pull.cpp:238-243
  }
}

// ---- binned pull (degree-ordered graphs) --------------------------------------
// The sources are cut into blocks of kBinPart consecutive ids whose
// contributions fit in shared memory.  The in-arcs of a block are ordered by
// destination, so the arcs into one destination form a run; they are stored in
// 256-arc chunks (per arc a 2-byte local source, per 8 arcs a byte that says
// which start a run; every chunk starts one), and per run its destination.
// Per iteration
//   gather: a CTA takes a task (a range of chunks of one block), loads the
//     block's contributions into shared memory, streams the chunks, sums each
//     run (8 arcs per lane, runs that span lanes by a segmented warp sum) and
//     adds the runs' sums to their destinations with reductions that return
//     nothing (32 consecutive runs at a time: ascending destinations);
//   finish: per vertex the new rank and its contribution (coalesced).
// An arc costs 2.1 streamed bytes and one shared-memory read, a run 4 bytes
// and one reduction in L2 (0.16 runs per arc on RMAT graphs in degree order at
// 4 M vertices).  The reverse, destinations cut into blocks with their sums in
// shared memory and one contribution gathered per run, adds every arc with a
// shared-memory atomic: RMAT-23 symmetric (15 iterations) 10.6 ms, 10.0 with
// each chunk's contributions staged in shared memory, against 8.1 here (0.54 ms
// an iteration, 470 G arcs/s; RMAT-21 of edge factor 8 3.2 -> 1.8), and the
// sort by block of sources alone builds the layout in 18 ms instead of 65.
// Bound by instruction issue and the shared-memory reads of the gather (about
// four fifths) and by the vertex pass.

constexpr uint32_t kBinPart = 32768;  // sources per block (a local id fits 16 bits, with kBinPart for padding)
constexpr uint32_t kBinChunk = 256;   // arcs per chunk
constexpr int kBinBlock = 1024;
// A row gets one addition per block of sources and chunk.  In 32 bits the
// largest ranks' rounding put the result 3.6e-7 of its norm off at RMAT-23
// (2.7e-7 with the sums built in shared memory), so the kBinHubs largest rows
// are added up in 64 bits: 6e-8; 4096 rows 1.4e-7.  All heavy rows: 4e-8, but
// the conversions of every run's sum cost 0.2 ms an iteration.
constexpr uint32_t kBinHubs = 16384;
// Shared memory of the gather: the block's contributions, a zero for padding,
// then per warp a chunk's run sums.
constexpr size_t kBinSmem = sizeof(float) * (kBinPart + 32 + kBinBlock / 32 * kBinChunk);

// A lane's 8 arcs of chunk c and their run flags (nothing past the task's end).
__device__ __forceinline__ void bin_load_chunk(const PrArgs& a, uint64_t c, uint64_t cend, uint32_t lane, uint4& u,
                                               uint32_t& f) {
  u = make_uint4(0u, 0u, 0u, 0u);
  f = 0u;
  if (c < cend) {
    u = ldg(reinterpret_cast<const uint4*>(a.b_src + c * kBinChunk) + lane);
    f = ldg(a.b_flag + c * (kBinChunk / 8) + lane);
  }
}

// The runs of chunk c: the first and their number.
__device__ __forceinline__ uint2 bin_runs(const PrArgs& a, uint64_t c, uint64_t cend) {
  if (c >= cend) return make_uint2(0u, 0u);
  const uint32_t r = ldg(a.b_crun + c);
  return make_uint2(r, ldg(a.b_crun + c + 1) - r);
}

// The destinations of a chunk's first 64 runs, two per lane.
__device__ __forceinline__ uint2 bin_dests(const PrArgs& a, uint2 runs, uint32_t lane) {
  return make_uint2(lane < runs.y ? ldg(a.b_rdst + runs.x + lane) : 0u,
                    lane + 32 < runs.y ? ldg(a.b_rdst + runs.x + lane + 32) : 0u);
}

// The sums of a chunk's runs into s_run.  All lanes call.
__device__ __forceinline__ void bin_run_sums(const float* s_c, uint4 u, uint32_t f, uint32_t lane, float* s_run) {
  uint32_t upto = __popc(f);  // runs that start in this lane or before it
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, upto, o);
    if (lane >= (uint32_t)o) upto += y;
  }
  float x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t w = k < 2 ? u.x : k < 4 ? u.y : k < 6 ? u.z : u.w;
    x[k] = s_c[(w >> (16 * (k & 1))) & 0xFFFFu];
  }
  // runs that start and end here are stored; the arcs before the lane's first
  // start belong to a run of the lanes before, the ones from its last start on
  // to one that may go on in the next lanes
  uint32_t r = upto - __popc(f);  // the next run to start here
  float sum = x[0], head = 0.f;
  bool started = f & 1u;
  r += started;
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    if ((f >> k) & 1u) {
      if (started) s_run[r - 1] = sum;
      else head = sum;
      started = true;
      ++r;
      sum = x[k];
    } else {
      sum += x[k];
    }
  }
  const float next = __shfl_down_sync(kFull, head, 1);
  if (lane < 31) sum += next;
  // a lane without a start only continues the run of the lanes before it
  if (__any_sync(kFull, f == 0)) seg_reduce(true, upto, sum);
  if (f) s_run[upto - 1] = sum;
}

// The gather phase of a binned iteration: the CTA takes tasks until none is
// left and adds to acc_cur (zero before) the sums of c_in over the in-arcs.
// All threads of the CTA call.
template <int BLOCK>
__device__ __forceinline__ void bin_gather(const PrArgs& a, const float* c_in, float* acc_cur, double* hacc_cur,
                                           uint32_t it, float* s_c, uint32_t* s_task) {
  const uint32_t tid = threadIdx.x, lane = lane_id(), wib = tid >> 5;
  constexpr uint32_t kW = BLOCK / 32;
  static_assert(BLOCK == 1024, "a lane per warp adds up the warps' chunks of one run");
  __shared__ uint32_t s_hub[kW];
  __shared__ double s_hsum[kW];
  auto add = [&](uint32_t v, float x) {
    if (x == 0.f) return;
    if (v < a.b_nheavy) atomicAdd(&hacc_cur[v], (double)x);
    else atomicAdd(&acc_cur[v], x);
  };
  auto add_hub = [&](uint32_t v, double x) {
    if (x == 0.0) return;
    if (v < a.b_nheavy) atomicAdd(&hacc_cur[v], x);
    else atomicAdd(&acc_cur[v], (float)x);
  };
  float* s_run = s_c + kBinPart + 32 + wib * kBinChunk;
  if (tid == 0) s_c[kBinPart] = 0.f;
  for (;;) {
    if (tid == 0) *s_task = atomicAdd(&a.ctl->task_next[it & 1], 1u);
    __syncthreads();
    const uint32_t t = *s_task;
    if (t >= a.b_ntasks) break;  // uniform
    const uint4 tk = ldg(a.b_tasks + t);
    // written by the finish pass: plain loads, not ldg
    const float4* c4 = reinterpret_cast<const float4*>(c_in + tk.x);  // a multiple of kBinPart
#pragma unroll 4
    for (uint32_t d = tid; d < tk.y / 4; d += BLOCK) reinterpret_cast<float4*>(s_c)[d] = c4[d];
    for (uint32_t d = (tk.y & ~3u) + tid; d < tk.y; d += BLOCK) s_c[d] = c_in[tk.x + d];
    __syncthreads();
    // loaded ahead: a chunk's runs two chunks before it is summed, its arcs and
    // the runs' destinations one
    uint64_t c = tk.z + wib;
    const uint64_t cend = tk.w;
    uint4 u;
    uint32_t f;
    bin_load_chunk(a, c, cend, lane, u, f);
    uint2 r0 = bin_runs(a, c, cend), r1 = bin_runs(a, c + kW, cend);
    uint2 d0 = bin_dests(a, r0, lane);
    // whole chunks of one destination are summed over the task before they are
    // added: a hub's sum takes one addition per task, not one per chunk
    uint32_t hub = 0xFFFFFFFFu;
    double hsum = 0.0;
    for (; c < cend; c += kW) {
      uint4 un;
      uint32_t fn;
      bin_load_chunk(a, c + kW, cend, lane, un, fn);
      const uint2 d1 = bin_dests(a, r1, lane), r2 = bin_runs(a, c + 2 * kW, cend);
      bin_run_sums(s_c, u, f, lane, s_run);
      __syncwarp();
      if (r0.y == 1) {
        const uint32_t v = __shfl_sync(kFull, d0.x, 0);
        if (v != hub) {
          if (lane == 0) add_hub(hub, hsum);  // nothing the first time
          hub = v;
          hsum = 0.0;
        }
        hsum += s_run[0];
        r0.y = 0;
      }
      if (lane < r0.y) add(d0.x, s_run[lane]);
      if (lane + 32 < r0.y) add(d0.y, s_run[lane + 32]);
#pragma unroll 2
      for (uint32_t k = 64 + lane; k < r0.y; k += 32) {
        add(ldg(a.b_rdst + r0.x + k), s_run[k]);
      }
      __syncwarp();  // s_run is rewritten by the next chunk
      u = un, f = fn;
      r0 = r1, r1 = r2, d0 = d1;
    }
    if (lane == 0) {
      s_hub[wib] = hub;
      s_hsum[wib] = hsum;
    }
    __syncthreads();  // s_c and s_task are reused by the next task
    if (wib == 0) {
      const uint32_t v = s_hub[lane];
      const double x = s_hsum[lane];
      for (unsigned left = __ballot_sync(kFull, v != 0xFFFFFFFFu); left;) {
        const uint32_t w = __shfl_sync(kFull, v, __ffs(left) - 1);
        const double sum = warp_sum(v == w ? x : 0.0);
        if (lane == 0) add_hub(w, sum);
        left &= ~__ballot_sync(kFull, v == w);
      }
    }
  }
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1) pr_pull_binned(PrArgs a) {
  extern __shared__ __align__(16) float s_c[];  // kBinSmem bytes
  __shared__ double s_l1, s_total;
  __shared__ uint32_t s_max, s_task;
  if (threadIdx.x == 0) {
    s_l1 = 0.0;
    s_max = 0u;
  }
  __syncthreads();
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)BLOCK + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * BLOCK;
  float* const c_io = a.c[0];  // gathered, then rewritten after the barrier
  for (uint32_t it = 0;; ++it) {
    float* const acc_cur = (it & 1) ? a.acc2 : a.acc;
    float* const acc_nxt = (it & 1) ? a.acc : a.acc2;
    double* const hacc_cur = a.hacc + (it & 1) * a.b_nheavy;
    double* const hacc_nxt = a.hacc + ((it + 1) & 1) * a.b_nheavy;
    if (gtid == 0) {
      clear_change(ctl, (it + 1) % 3);
      ctl->task_next[(it + 1) & 1] = 0u;  // the counter iteration it + 1 takes (it - 1's is done)
    }
    bin_gather<BLOCK>(a, c_io, acc_cur, hacc_cur, it, s_c, &s_task);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    // ---- finish: ranks and contributions for the next gather
    double my_l1 = 0.0;
    float my_max = 0.f;
    const uint32_t vend = it >= 2 ? a.zero_from : a.n;  // constant tail skipped (its values stay)
    auto finish = [&](uint64_t v, float sum, float old, uint32_t k) {
      const float value = sum * a.alpha + a.base;  // PageRank-pull.cpp:222
      a.value[v] = value;
      c_io[v] = k ? value / (float)k : 0.f;
      my_l1 += (double)fabsf(value - old);
      my_max = fmaxf(my_max, fabsf(value - old));
    };
    const uint32_t nh = min(a.b_nheavy, vend);
    for (uint64_t v = gtid; v < nh; v += gthreads) {
      const double sum = hacc_cur[v];
      hacc_nxt[v] = 0.0;
      finish(v, (float)sum, a.value[v], a.nout[v]);
    }
    // four vertices' loads together, as no load may pass the stores (one
    // vertex at a time: 0.77 ms an iteration of RMAT-23, not 0.54)
    for (uint64_t v0 = nh + gtid; v0 < vend; v0 += 4 * gthreads) {
      float sum[4], old[4];
      uint32_t k[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t v = v0 + j * gthreads;
        if (v < vend) sum[j] = acc_cur[v], old[j] = a.value[v], k[j] = a.nout[v];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t v = v0 + j * gthreads;
        if (v >= vend) break;
        acc_nxt[v] = 0.f;
        finish(v, sum[j], old[j], k[j]);
      }
    }
    publish_change(ctl, it % 3, my_l1, my_max, &s_l1, &s_max);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    const double l1 = read_change(ctl, it % 3, a.linf, &s_total);
    if (gtid == 0) ctl->iters = it + 1;
    if (l1 <= (double)a.tol || it + 1 >= a.max_iter) break;  // PageRank-pull.cpp:238-243
  }
}

// Layout build, once per graph: arcs per block of sources, then per arc its
// block (the sort key) and destination << 16 | local source.
__global__ void bin_count_kernel(const uint32_t* __restrict__ nout, uint32_t n, unsigned long long* __restrict__ count) {
  const uint64_t v0 = (uint64_t)blockIdx.x * kBinPart, v1 = min(v0 + kBinPart, (uint64_t)n);
  unsigned long long mine = 0;
  for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) mine += nout[v];
  mine = warp_sum(mine);
  if (lane_id() == 0 && mine) atomicAdd(&count[blockIdx.x], mine);
}

__global__ void bin_keys_kernel(const uint64_t* __restrict__ offs, const uint32_t* __restrict__ col, uint32_t n,
                                uint16_t* __restrict__ key, uint64_t* __restrict__ val) {
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t v = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
    for (uint64_t j = offs[v] + lane; j < offs[v + 1]; j += 32) {
      const uint32_t u = col[j];
      key[j] = (uint16_t)(u / kBinPart);
      val[j] = v << 16 | u % kBinPart;
    }
  }
}

// A warp's chunk of the sorted arcs (arcs first[p] .. of block p fill the
// chunks from pad[p] / kBinChunk on): its lane's 8 destinations and local
// sources (kBinPart past the block's end) and the byte of run starts.
__device__ __forceinline__ uint32_t bin_chunk_arcs(const uint64_t* __restrict__ val, const uint64_t* __restrict__ first,
                                                   const uint64_t* __restrict__ pad, uint32_t P, uint64_t c,
                                                   uint32_t (&dst)[8], uint32_t (&src)[8]) {
  uint32_t lo = 0, hi = P;  // the last block that starts at or before the chunk and is not empty
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (pad[mid] <= c * kBinChunk) lo = mid;
    else hi = mid;
  }
  const uint32_t lane = lane_id();
  const uint64_t i = first[lo] + (c * kBinChunk - pad[lo]) + lane * 8;
  const uint64_t e = first[lo + 1];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const bool ok = i + k < e;
    const uint64_t x = ok ? val[i + k] : 0ull;
    dst[k] = (uint32_t)(x >> 16);
    src[k] = ok ? (uint32_t)x & 0xFFFFu : kBinPart;
  }
  const uint32_t before = __shfl_up_sync(kFull, dst[7], 1);
  uint32_t f = (lane == 0 || (i < e && dst[0] != before)) ? 1u : 0u;
#pragma unroll
  for (int k = 1; k < 8; ++k)
    if (i + k < e && dst[k] != dst[k - 1]) f |= 1u << k;
  return f;
}

__global__ void bin_place_kernel(const uint64_t* __restrict__ val, const uint64_t* __restrict__ first,
                                 const uint64_t* __restrict__ pad, uint32_t P, uint64_t nchunks, uint16_t* __restrict__ src,
                                 uint8_t* __restrict__ flag, uint32_t* __restrict__ count) {
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t c = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; c < nchunks; c += nw) {
    uint32_t d[8], u[8];
    const uint32_t f = bin_chunk_arcs(val, first, pad, P, c, d, u);
    reinterpret_cast<uint4*>(src + c * kBinChunk)[lane] =
        make_uint4(u[0] | u[1] << 16, u[2] | u[3] << 16, u[4] | u[5] << 16, u[6] | u[7] << 16);
    flag[c * (kBinChunk / 8) + lane] = (uint8_t)f;
    const uint32_t runs = __reduce_add_sync(kFull, __popc(f));
    if (lane == 0) count[c] = runs;
  }
}

__global__ void bin_runs_kernel(const uint64_t* __restrict__ val, const uint64_t* __restrict__ first,
                                const uint64_t* __restrict__ pad, uint32_t P, uint64_t nchunks,
                                const uint32_t* __restrict__ crun, uint32_t* __restrict__ rdst) {
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t c = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; c < nchunks; c += nw) {
    uint32_t d[8], u[8];
    const uint32_t f = bin_chunk_arcs(val, first, pad, P, c, d, u);
    uint32_t upto = __popc(f);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, upto, o);
      if (lane >= (uint32_t)o) upto += y;
    }
    uint32_t r = crun[c] + upto - __popc(f);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if ((f >> k) & 1u) rdst[r++] = d[k];
  }
}

// The light rows' run table, in two passes: the row holding each run's first
// arc, then every arc's offset from it.
__global__ void light_runrow_kernel(const uint64_t* __restrict__ offs, uint32_t row0, uint32_t row1, uint64_t arc0,
                                    uint32_t* __restrict__ runrow) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = row0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < row1; v += stride) {
    const uint64_t b = offs[v] - arc0, e = offs[v + 1] - arc0;
    // the runs whose first arc lies in [b, e)
    for (uint64_t r = (b + kLightRun - 1) / kLightRun; r * kLightRun < e; ++r) runrow[r] = (uint32_t)v;
  }
}

__global__ void light_rowd_kernel(const uint64_t* __restrict__ offs, uint32_t row0, uint32_t row1, uint64_t arc0,
                                  const uint32_t* __restrict__ runrow, uint8_t* __restrict__ rowd) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = row0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < row1; v += stride)
    for (uint64_t e = offs[v] - arc0; e < offs[v + 1] - arc0; ++e)
      rowd[e] = (uint8_t)((uint32_t)v - runrow[e / kLightRun]);
}

// ---- pull-residual (PageRank-pull.cpp:132-190) ------------------------------
__global__ void pr_resid_init(PrArgs a) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = tid; v < a.n; v += stride) {
    a.value[v] = 0.f;
    a.delta[v] = 0.f;
    a.residual[v] = 1.0f - a.alpha;  // INIT_RESIDUAL, PageRank-constants.h:33
  }
}

// The vertex pass of pull-residual round it: closes round it - 1 (a positive
// sum becomes the residual), then takes the residuals above tol (value +=
// residual, delta = residual * alpha / outdeg) and counts those with out-arcs.
__device__ __forceinline__ void resid_vertex_pass(const PrArgs& a, uint32_t it, const float* acc_prev, float* acc_cur,
                                                  uint64_t gtid, uint64_t gthreads) {
  uint32_t my_accum = 0;
  for (uint64_t v = gtid; v < a.n; v += gthreads) {
    float r = a.residual[v];
    // the sums of round it - 2, read by round it - 1: zeroed for this
    // round's gather (zeroing the slots the last gather's atomics just
    // updated stalls)
    float sum;
    if (v < a.b_nheavy) {
      sum = (float)a.hacc[((it + 1) & 1) * a.b_nheavy + v];
      a.hacc[(it & 1) * a.b_nheavy + v] = 0.0;
    } else {
      sum = acc_prev[v];
      acc_cur[v] = 0.f;
    }
    if (it > 0 && sum > 0.f) r = sum;
    float d = 0.f;
    if (r > a.tol) {
      a.value[v] += r;
      const uint32_t k = a.nout[v];
      if (k > 0) {
        d = r * a.alpha / (float)k;
        ++my_accum;
      }
      r = 0.f;
    }
    a.residual[v] = r;
    a.delta[a.rank ? a.rank[v] : v] = d;
  }
  my_accum = __reduce_add_sync(kFull, my_accum);
  if (lane_id() == 0 && my_accum) atomicAdd(&a.ctl->active[it % 3], my_accum);
}

// Pull-residual rounds over the rows as stored: the vertex pass, then every
// row's sum of deltas (light rows stored, heavy rows' tiles added), two grid
// barriers a round.  RMAT-21 directed (32 M arcs): see chunk_row_sums.
__global__ void __launch_bounds__(kBlock, 6) pr_pull_residual_persistent(PrArgs a) {
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)kBlock + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * kBlock;
  const uint64_t gwarp = gtid >> 5, nwarps = gthreads >> 5;
  const uint32_t lane = lane_id();
  const uint64_t nchunks = ((uint64_t)a.n + 31) >> 5;
  for (uint32_t it = 0;; ++it) {
    float* const acc_prev = (it & 1) ? a.acc : a.acc2;
    float* const acc_cur = (it & 1) ? a.acc2 : a.acc;
    if (gtid == 0) ctl->active[(it + 1) % 3] = 0;
    resid_vertex_pass(a, it, acc_prev, acc_cur, gtid, gthreads);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    auto gather = [&](uint32_t u) {
      const float d = u != 0xFFFFFFFFu ? a.delta[u] : 0.f;
      return d > 0.f ? d : 0.f;
    };
    for (uint64_t t = gwarp; t < nchunks + a.sched.ntiles; t += nwarps) {
      if (t < nchunks) {
        const uint64_t v = (t << 5) + lane;
        uint64_t b = 0;
        uint32_t d = 0;
        if (v < a.n) {
          b = ldg(a.offs + v);
          const uint64_t dd = ldg(a.offs + v + 1) - b;
          d = dd > a.sched.heavy ? 0u : (uint32_t)dd;
        }
        if (!__any_sync(kFull, d != 0)) continue;
        const float sum = chunk_row_sums(a.col, b, d, gather);
        if (sum > 0.f) acc_cur[v] = sum;
      } else {
        const uint2 tv = a.sched.tiles[t - nchunks];
        const uint64_t vb = ldg(a.offs + tv.x), ve = ldg(a.offs + tv.x + 1);
        const uint64_t b = vb + (uint64_t)tv.y * a.sched.tile;
        const float sum = tile_row_sum(a.col, b, min(ve, b + a.sched.tile), gather);
        if (lane == 0 && sum > 0.f) atomicAdd(&acc_cur[tv.x], sum);
      }
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    const uint32_t accum = *reinterpret_cast<volatile uint32_t*>(&ctl->active[it % 3]);
    if (gtid == 0) ctl->iters = it + 1;
    if (it + 1 >= a.max_iter || accum == 0) break;
  }
}

// The same rounds over the binned layout (degree-ordered graphs).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1) pr_resid_binned(PrArgs a) {
  extern __shared__ __align__(16) float s_c[];  // kBinSmem bytes
  __shared__ uint32_t s_task;
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)BLOCK + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * BLOCK;
  for (uint32_t it = 0;; ++it) {
    float* const acc_prev = (it & 1) ? a.acc : a.acc2;  // round it - 1's sums
    float* const acc_cur = (it & 1) ? a.acc2 : a.acc;
    if (gtid == 0) {
      ctl->active[(it + 1) % 3] = 0;
      ctl->task_next[(it + 1) & 1] = 0u;
    }
    resid_vertex_pass(a, it, acc_prev, acc_cur, gtid, gthreads);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    bin_gather<BLOCK>(a, a.delta, acc_cur, a.hacc + (it & 1) * a.b_nheavy, it, s_c, &s_task);
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    const uint32_t accum = *reinterpret_cast<volatile uint32_t*>(&ctl->active[it % 3]);
    if (gtid == 0) ctl->iters = it + 1;
    if (it + 1 >= a.max_iter || accum == 0) break;
  }
}

// ---- residual push, Sync (PageRank-push.cpp:103-188) ------------------------
__global__ void pr_push_init(PrArgs a) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = tid; v < a.n; v += stride) {
    a.value[v] = 0.f;
    a.residual[v] = 1.0f - a.alpha;
    a.active[0][v] = (uint32_t)v;
    a.stamp[v] = 0xFFFFFFFFu;
  }
  if (tid == 0) a.ctl->active[0] = a.n;
}

__global__ void __launch_bounds__(kBlock) pr_push_persistent(PrArgs a) {
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)kBlock + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * kBlock;
  const uint32_t lane = lane_id();
  unsigned long long my_push = 0;
  for (uint32_t it = 0;; ++it) {
    const uint32_t na = min(ctl->active[it % 3], a.n);
    if (na == 0 || it >= a.max_iter) break;
    const int fset = it % 3;
    if (gtid == 0) {
      ctl->active[(it + 2) % 3] = 0;
      ctl->fc[(it + 1) % 3] = FrontierCounters{};
    }
    FrontierCounters& fc = ctl->fc[fset];
    const uint32_t* act = a.active[it & 1];
    uint32_t* act_next = a.active[(it + 1) & 1];
    // phase A: absorb residual, compute delta, queue vertices with out-arcs
    for (uint64_t base = gtid - lane; base < na; base += gthreads) {
      const uint64_t i = base + lane;
      bool q = false;
      uint32_t v = 0;
      if (i < na) {
        v = act[i];
        const float r = a.residual[v];
        if (r > a.tol) {
          const float old = atomicExch(&a.residual[v], 0.f);
          if (old > 0.f) {
            a.value[v] += old;
            const uint64_t deg = ldg(a.offs + v + 1) - ldg(a.offs + v);
            if (deg > 0) {
              a.delta[v] = old * a.alpha / (float)deg;
              q = true;
            }
          }
        }
      }
      push_discovered(a.fq, it & 1, fc, q, v, a.offs, a.heavy, a.tile, &ctl->err);
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    // phase B: push deltas along out-arcs, activate on crossing tol
    const uint32_t q_light = min(fc.light, a.fq.light_cap), q_tiles = min(fc.tiles, a.fq.tile_cap);
    auto apply = [&](bool valid, uint32_t u, float d) {
      bool act_u = false;
      if (valid) {
        const float old = atomicAdd(&a.residual[u], d);
        ++my_push;
        if (old <= a.tol && old + d >= a.tol) {
          if (a.stamp[u] != it) act_u = atomicExch(&a.stamp[u], it) != it;
        }
      }
      warp_push(act_u, u, act_next, &ctl->active[(it + 1) % 3], a.n, &ctl->err);
    };
    const uint32_t* qin = a.fq.light[it & 1];
    const uint2* tin = a.fq.tiles[it & 1];
    for (;;) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&fc.light_work, 32u);
      base = __shfl_sync(kFull, base, 0);
      if (base >= q_light) break;
      const uint32_t idx = base + lane;
      uint64_t b = 0;
      uint32_t d = 0;
      float dl = 0.f;
      if (idx < q_light) {
        const uint32_t v = qin[idx];
        b = ldg(a.offs + v);
        d = (uint32_t)(ldg(a.offs + v + 1) - b);
        dl = a.delta[v];
      }
      warp_expand(b, d, __float_as_uint(dl), [&](bool valid, uint64_t e, uint32_t, uint32_t pl) {
        apply(valid, valid ? ldg(a.col + e) : 0u, __uint_as_float(pl));
      });
    }
    for (;;) {
      uint32_t t = 0;
      if (lane == 0) t = atomicAdd(&fc.tile_work, 1u);
      t = __shfl_sync(kFull, t, 0);
      if (t >= q_tiles) break;
      const uint2 tv = tin[t];
      const uint64_t vb = ldg(a.offs + tv.x), ve = ldg(a.offs + tv.x + 1);
      const uint64_t b = vb + (uint64_t)tv.y * a.tile;
      const uint64_t e_end = min(ve, b + a.tile);
      const float dl = a.delta[tv.x];
      for (uint64_t e0 = b; e0 < e_end; e0 += 32) {
        const uint64_t e = e0 + lane;
        apply(e < e_end, e < e_end ? ldg(a.col + e) : 0u, dl);
      }
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    if (gtid == 0) ctl->iters = it + 1;
  }
  my_push = warp_sum(my_push);
  if (lane == 0 && my_push) atomicAdd(&ctl->pushes, my_push);
}

// ---- residual push, Async (PageRank-push.cpp:68-101) -------------------------
// Worklist entries: (v, kAbsorb, 0, 0) "take v's residual if it is above
// tol" -- every vertex once at the start (the reference iterates the whole
// graph), then each vertex whose residual an add lifts across tol -- and
// (v, k, delta bits, 0): "add delta along the k-th tile of v's arcs", made
// when a heavy vertex is absorbed.
constexpr uint32_t kAbsorb = 0xFFFFFFFFu;
constexpr int kPushLQ = 64;

__global__ void pr_push_async_init(PrArgs a, uint32_t nchunks) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = tid; v < a.n; v += stride) {
    a.value[v] = 0.f;
    a.residual[v] = 1.0f - a.alpha;  // INIT_RESIDUAL, PageRank-constants.h:33
  }
  // the initial worklist: every vertex, 32 per chunk, published
  for (uint64_t i = tid; i <= a.ring.mask; i += stride) {
    if (i < nchunks) {
      const uint32_t first = (uint32_t)(i * 32);
      const uint32_t cnt = min(32u, a.n - first);
      for (uint32_t j = 0; j < cnt; ++j) a.ring.ent[i * 32 + j] = make_uint4(first + j, kAbsorb, 0u, 0u);
      a.ring.cnt[i] = cnt;
      a.ring.seq[i] = i + 1;
    } else {
      a.ring.seq[i] = i;
    }
  }
  if (tid == 0) {
    a.ring.rc->tail = nchunks;
    a.ring.rc->work = (int)nchunks;
  }
}

__global__ void __launch_bounds__(kBlock, 1) pr_push_async(PrArgs a) {
  __shared__ uint4 s_lq[kWarps][kPushLQ];
  PrCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint32_t lane = lane_id();
  unsigned long long my_push = 0, my_absorb = 0;
  worklists::WarpQueue<kPushLQ> q(s_lq[threadIdx.x >> 5], a.ring, &ctl->err, deadline);
  const float tol = a.tol;
  // add d to u's residual; activate u when the add lifts it across tol
  // (old < tol <= old + d, PageRank-push.cpp:92-94)
  auto add = [&](bool valid, uint32_t u, float d) {
    bool act = false;
    if (valid && d > 0.f) {
      const float old = atomicAdd(&a.residual[u], d);
      ++my_push;
      act = old < tol && old + d >= tol;
    }
    q.push(act, make_uint4(u, kAbsorb, 0u, 0u));
  };
  for (;;) {
    uint4 ent;
    bool has;
    const int got = q.next(ent, has);
    if (got <= 0) break;
    // tiles of heavy vertices: the whole warp adds along each in turn
    unsigned tm = __ballot_sync(kFull, has && ent.y != kAbsorb);
    while (tm) {
      const int j = __ffs(tm) - 1;
      tm &= tm - 1u;
      const uint32_t v = __shfl_sync(kFull, ent.x, j);
      const uint32_t k = __shfl_sync(kFull, ent.y, j);
      const float d = __uint_as_float(__shfl_sync(kFull, ent.z, j));
      const uint64_t vb = ldg(a.offs + v), ve = ldg(a.offs + v + 1);
      const uint64_t b = vb + (uint64_t)k * a.tile, e_end = min(ve, b + a.tile);
      for (uint64_t e0 = b; e0 < e_end; e0 += 32) {
        const uint64_t e = e0 + lane;
        add(e < e_end, e < e_end ? ldg(a.col + e) : 0u, d);
      }
    }
    // absorb: exchange the residual with 0 if it is above tol
    const bool absorb = has && ent.y == kAbsorb;
    uint64_t b = 0, deg = 0;
    float delta = 0.f;
    if (absorb && __ldcg(a.residual + ent.x) > tol) {
      const float old = atomicExch(&a.residual[ent.x], 0.f);
      atomicAdd(&a.value[ent.x], old);  // a vertex may be queued twice when tol >= 1 - alpha
      ++my_absorb;
      b = ldg(a.offs + ent.x);
      deg = ldg(a.offs + ent.x + 1) - b;
      if (deg > 0) delta = old * a.alpha / (float)deg;
    }
    const bool light = deg > 0 && deg <= a.heavy;
    // light rows: their arcs spread over the warp
    warp_expand(b, light ? (uint32_t)deg : 0u, __float_as_uint(delta), [&](bool valid, uint64_t e, uint32_t, uint32_t pl) {
      add(valid, valid ? ldg(a.col + e) : 0u, __uint_as_float(pl));
    });
    // heavy rows: one worklist entry per tile
    unsigned hm = __ballot_sync(kFull, deg > a.heavy && delta > 0.f);
    while (hm) {
      const int j = __ffs(hm) - 1;
      hm &= hm - 1u;
      const uint32_t v = __shfl_sync(kFull, ent.x, j);
      const uint32_t nt = (uint32_t)((__shfl_sync(kFull, deg, j) + a.tile - 1) / a.tile);
      const uint32_t dbits = __shfl_sync(kFull, __float_as_uint(delta), j);
      for (uint32_t t0 = 0; t0 < nt; t0 += 32) q.push(t0 + lane < nt, make_uint4(v, t0 + lane, dbits, 0u));
    }
    q.share();
  }
  my_push = warp_sum(my_push);
  my_absorb = warp_sum(my_absorb);
  if (lane == 0) {
    if (my_push) atomicAdd(&ctl->pushes, my_push);
    if (my_absorb) atomicAdd(&ctl->absorbs, my_absorb);
  }
}

int ensure_nout(gb_graph* g, cudaStream_t s) {
  if (g->outdeg_of_stored) return GB_OK;
  GB_CUDA(cudaMalloc(&g->outdeg_of_stored, sizeof(uint32_t) * g->n));
  GB_CUDA(cudaMemsetAsync(g->outdeg_of_stored, 0, sizeof(uint32_t) * g->n, s));
  if (g->m) count_nout<<<g->sm_count * 8, 256, 0, s>>>(g->col, g->m, g->outdeg_of_stored);
  GB_CUDA(cudaGetLastError());
  return GB_OK;
}

enum class PrKind { Pull, PullResidual, Push, PushAsync };

// arcs[0] += the counts behind the first `cnt` sorted keys (~count).
__global__ void hot_share_kernel(const uint32_t* __restrict__ key, uint32_t cnt, unsigned long long* arcs) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long mine = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt; i += stride)
    mine += ~key[i];
  mine = warp_sum(mine);
  if (lane_id() == 0 && mine) atomicAdd(arcs, mine);
}

__global__ void hot_keys_kernel(const uint32_t* __restrict__ count, uint32_t n, uint32_t* __restrict__ key,
                                uint32_t* __restrict__ id) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += stride) {
    key[v] = ~count[v];  // ascending order of the inverted count: most gathered first
    id[v] = (uint32_t)v;
  }
}

__global__ void hot_rank_kernel(const uint32_t* __restrict__ id, uint32_t n, uint32_t* __restrict__ rank) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) rank[id[i]] = (uint32_t)i;
}

__global__ void hot_col_kernel(const uint32_t* __restrict__ col, uint64_t m, const uint32_t* __restrict__ rank,
                               uint32_t* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += stride) out[e] = rank[col[e]];
}

// The row sweeps are bound by the rate of their 4-byte gathers (an L2 sector
// each).  In file order the few vertices that most arcs of a power-law graph
// point at are spread over all cache lines; with the contributions stored by
// falling in-degree they share the lines that L1 keeps.  The columns are
// copied once with the vertices renamed so (4 bytes per arc of memory, about
// the time of one iteration), the rows and results stay in file order.
// Where it pays: the contributions do not fit L1 anyway (n > kHotSlots), and
// the kHotSlots most gathered vertices (192 KB) take a quarter of the arcs
// (RMAT-21 directed: 67 %; a uniform graph or a grid: kHotSlots / n).
// A graph that does not qualify keeps its columns; so does one whose copy
// would take more than a quarter of the free memory, and one whose first call
// is being captured into a graph (the choice waits for a count).
// Pull-residual: RMAT-21 directed (34 rounds) 5.98 -> 5.39 ms,
// RMAT-22 symmetric 23.7 -> 16.9 ms (first call 25.2 -> 20.0); pull-topological
// on the latter 12.4 -> 10.6 ms (13.8 -> 13.6).
constexpr uint32_t kHotSlots = 49152;
constexpr double kHotShare = 0.25;

// Workspace of ensure_hot, which runs before the solve carves its own from the
// same block (0: nothing to do).
int hot_scratch(gb_graph* g, cudaStream_t s, size_t* bytes, size_t* sort_bytes) {
  *bytes = 0;
  if (g->prh || g->m == 0 || g->n <= kHotSlots) return GB_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GB_CUDA(cudaStreamIsCapturing(s, &cap));
  if (cap != cudaStreamCaptureStatusNone) return GB_OK;
  cub::DoubleBuffer<uint32_t> key(nullptr, nullptr), id(nullptr, nullptr);
  GB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, *sort_bytes, key, id, (int64_t)g->n, 0, 32, s));
  *bytes = carve_size<unsigned long long>(1) + 4 * carve_size<uint32_t>(g->n) + carve_size<char>(*sort_bytes);
  return GB_OK;
}

int ensure_hot(gb_graph* g, size_t sort_bytes, cudaStream_t s) {
  const uint32_t n = g->n;
  const uint64_t m = g->m;
  PrHot* h = new (std::nothrow) PrHot;
  if (!h) GB_FAIL(GB_ERR_OOM, "pagerank: host allocation failed");
  g->prh = h;
  Carver cv(g->ws);
  unsigned long long* arcs = cv.take<unsigned long long>(1);
  unsigned long long* harcs = static_cast<unsigned long long*>(g->pinned);
  cub::DoubleBuffer<uint32_t> key(nullptr, nullptr), id(nullptr, nullptr);
  for (int k = 0; k < 2; ++k) {
    key.d_buffers[k] = cv.take<uint32_t>(n);
    id.d_buffers[k] = cv.take<uint32_t>(n);
  }
  void* tmp = cv.take<char>(sort_bytes);
  const int grid = g->sm_count * 8;
  GB_CUDA(cudaMemsetAsync(arcs, 0, sizeof(*arcs), s));
  hot_keys_kernel<<<grid, 256, 0, s>>>(g->outdeg_of_stored, n, key.Current(), id.Current());
  GB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, sort_bytes, key, id, (int64_t)n, 0, 32, s));
  hot_share_kernel<<<64, 256, 0, s>>>(key.Current(), kHotSlots, arcs);
  GB_CUDA(cudaMemcpyAsync(harcs, arcs, sizeof(*arcs), cudaMemcpyDeviceToHost, s));
  GB_CUDA(cudaStreamSynchronize(s));
  if ((double)*harcs < kHotShare * (double)m) return GB_OK;
  // asked here, once per graph that qualifies: the question alone takes up to
  // 10 ms on a device whose memory is nearly all in use
  size_t free_bytes = 0, total_bytes = 0;
  GB_CUDA(cudaMemGetInfo(&free_bytes, &total_bytes));
  if (sizeof(uint32_t) * (m + n) > free_bytes / 4) return GB_OK;
  uint32_t* cols = nullptr;
  if (cudaMalloc(&cols, sizeof(uint32_t) * (m + n)) != cudaSuccess) {
    cudaGetLastError();
    return GB_OK;
  }
  uint32_t* const rank = cols + m;
  hot_rank_kernel<<<grid, 256, 0, s>>>(id.Current(), n, rank);
  hot_col_kernel<<<grid, 256, 0, s>>>(g->col, m, rank, cols);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {  // the handle must not be left with columns that nothing wrote
    cudaFree(cols);
    return cuda_fail(e, "pagerank: renamed columns");
  }
  h->col = cols;
  h->rank = rank;
  return GB_OK;
}

// Build (once) the binned layout of the stored arcs for pr_pull_binned.
// GB_ERR_UNSUPPORTED when it does not apply (no arcs, 2^32 arcs or more);
// on any failure nothing is cached and the caller keeps the row sweep.
int ensure_pr_bins(gb_graph* g, cudaStream_t s) {
  if (g->prb) return GB_OK;
  const uint32_t n = g->n;
  const uint64_t m = g->m;
  const uint32_t P = (uint32_t)(((uint64_t)n + kBinPart - 1) / kBinPart);
  if (m == 0 || m >= 0xFFFFFFF0ull || P > 65536) return GB_ERR_UNSUPPORTED;  // run ids are 32-bit, block ids 16-bit
  uint16_t *key0 = nullptr, *key1 = nullptr;
  uint64_t *val0 = nullptr, *val1 = nullptr, *dfirst = nullptr;
  void* tmp = nullptr;
  PrBins* b = new PrBins;
  auto cleanup = [&](bool keep) {
    cudaFree(key0);
    cudaFree(key1);
    cudaFree(val0);
    cudaFree(val1);
    cudaFree(dfirst);
    cudaFree(tmp);
    if (!keep) {
      cudaFree(b->mem);
      cudaFree(b->rdst);
      delete b;
    }
  };
#define GB_BTRY(call)                       \
  do {                                      \
    cudaError_t _e = (call);                \
    if (_e != cudaSuccess) {                \
      const int _st = cuda_fail(_e, #call); \
      cleanup(false);                       \
      return _st;                           \
    }                                       \
  } while (0)
  GB_BTRY(cudaMalloc(&dfirst, sizeof(uint64_t) * 2 * ((size_t)P + 1)));
  uint64_t* dpad = dfirst + P + 1;
  std::vector<uint64_t> first((size_t)P + 1), pad((size_t)P + 1);
  GB_BTRY(cudaMemsetAsync(dpad, 0, sizeof(uint64_t) * P, s));
  bin_count_kernel<<<P, 256, 0, s>>>(g->outdeg_of_stored, n, reinterpret_cast<unsigned long long*>(dpad));
  GB_BTRY(cudaGetLastError());
  GB_BTRY(cudaMemcpyAsync(pad.data(), dpad, sizeof(uint64_t) * P, cudaMemcpyDeviceToHost, s));
  GB_BTRY(cudaStreamSynchronize(s));
  // blocks: their arcs, padded to whole chunks; tasks of about
  // m / (6 per SM) arcs, the largest first
  uint64_t at = 0, mpad = 0;
  for (uint32_t p = 0; p < P; ++p) {
    const uint64_t cnt = pad[p];
    first[p] = at;
    pad[p] = mpad;
    at += cnt;
    mpad += (cnt + kBinChunk - 1) / kBinChunk * kBinChunk;
  }
  first[P] = at;
  pad[P] = mpad;
  const uint64_t nchunks = mpad / kBinChunk;
  if (at != m || nchunks >= 0xFFFFFFFEull) {  // chunk ids are 32-bit in the tasks
    cleanup(false);
    return GB_ERR_UNSUPPORTED;
  }
  const uint64_t target_chunks = std::max<uint64_t>(64, m / ((uint64_t)g->sm_count * 6 * kBinChunk));
  std::vector<uint4> tasks;
  for (uint32_t p = 0; p < P; ++p) {
    const uint64_t c0 = pad[p] / kBinChunk, c1 = pad[p + 1] / kBinChunk;
    if (c0 == c1) continue;  // sources without out-arcs
    const uint64_t nt = (c1 - c0 + target_chunks - 1) / target_chunks;
    const uint64_t per = (c1 - c0 + nt - 1) / nt;
    const uint32_t v0 = p * kBinPart;
    const uint32_t nv = (uint32_t)std::min<uint64_t>(kBinPart, (uint64_t)n - v0);
    for (uint64_t c = c0; c < c1; c += per)
      tasks.push_back(make_uint4(v0, nv, (uint32_t)c, (uint32_t)std::min(c1, c + per)));
  }
  std::stable_sort(tasks.begin(), tasks.end(), [](const uint4& x, const uint4& y) { return x.w - x.z > y.w - y.z; });

  GB_BTRY(cudaMalloc(&key0, sizeof(uint16_t) * m));
  GB_BTRY(cudaMalloc(&key1, sizeof(uint16_t) * m));
  GB_BTRY(cudaMalloc(&val0, sizeof(uint64_t) * m));
  GB_BTRY(cudaMalloc(&val1, sizeof(uint64_t) * m));
  GB_BTRY(cudaMemcpyAsync(dfirst, first.data(), sizeof(uint64_t) * ((size_t)P + 1), cudaMemcpyHostToDevice, s));
  GB_BTRY(cudaMemcpyAsync(dpad, pad.data(), sizeof(uint64_t) * ((size_t)P + 1), cudaMemcpyHostToDevice, s));
  const int grid = g->sm_count * 8;
  bin_keys_kernel<<<grid, 256, 0, s>>>(g->offs, g->col, n, key0, val0);
  GB_BTRY(cudaGetLastError());
  // stable: the rows' order (by destination) stays inside a block
  int end_bit = 1;
  while ((1u << end_bit) < P) ++end_bit;
  cub::DoubleBuffer<uint16_t> dk(key0, key1);
  cub::DoubleBuffer<uint64_t> dv(val0, val1);
  // the cached layout but the runs' destinations, one allocation (parts 256-byte aligned)
  auto part = [](uint64_t bytes) { return (bytes + 255) & ~uint64_t(255); };
  const uint64_t sz_src = part(2 * mpad), sz_flag = part(mpad / 8), sz_crun = part(4 * (nchunks + 1)),
                 sz_tasks = part(16 * tasks.size());
  GB_BTRY(cudaMalloc(&b->mem, sz_src + sz_flag + sz_crun + sz_tasks));
  char* q = static_cast<char*>(b->mem);
  b->src = reinterpret_cast<uint16_t*>(q);
  q += sz_src;
  b->flag = reinterpret_cast<uint8_t*>(q);
  q += sz_flag;
  b->crun = reinterpret_cast<uint32_t*>(q);
  q += sz_crun;
  b->tasks = reinterpret_cast<uint4*>(q);
  b->ntasks = (uint32_t)tasks.size();
  size_t tmp_bytes = 0, scan_bytes = 0;
  GB_BTRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, dk, dv, (int64_t)m, 0, end_bit, s));
  GB_BTRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, b->crun, b->crun, (int64_t)(nchunks + 1), s));
  tmp_bytes = std::max(tmp_bytes, scan_bytes);
  GB_BTRY(cudaMalloc(&tmp, std::max<size_t>(tmp_bytes, 16)));
  GB_BTRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, dk, dv, (int64_t)m, 0, end_bit, s));
  GB_BTRY(cudaMemcpyAsync(b->tasks, tasks.data(), 16 * tasks.size(), cudaMemcpyHostToDevice, s));
  GB_BTRY(cudaMemsetAsync(b->crun + nchunks, 0, sizeof(uint32_t), s));
  bin_place_kernel<<<grid, 256, 0, s>>>(dv.Current(), dfirst, dpad, P, nchunks, b->src, b->flag, b->crun);
  GB_BTRY(cudaGetLastError());
  GB_BTRY(cub::DeviceScan::ExclusiveSum(tmp, scan_bytes, b->crun, b->crun, (int64_t)(nchunks + 1), s));
  uint32_t runs = 0;
  GB_BTRY(cudaMemcpyAsync(&runs, b->crun + nchunks, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GB_BTRY(cudaStreamSynchronize(s));
  GB_BTRY(cudaMalloc(&b->rdst, sizeof(uint32_t) * std::max<uint32_t>(runs, 1)));
  bin_runs_kernel<<<grid, 256, 0, s>>>(dv.Current(), dfirst, dpad, P, nchunks, b->crun, b->rdst);
  GB_BTRY(cudaGetLastError());
  GB_BTRY(cudaStreamSynchronize(s));
#undef GB_BTRY
  cleanup(true);
  g->prb = b;
  return GB_OK;
}


inline float bits_to_float(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}

// The flat sweeps' run table of a degree-ordered graph (its heavy rows are
// [0, nheavy), the light rows' arcs one contiguous range): built once per
// heavy threshold and cached in the handle, then wired into `a`.
int light_run_table(gb_graph* g, const SweepSched& sched, PrArgs* a, cudaStream_t s) {
  if (!g->lr_rowid || g->lr_heavy != sched.heavy) {
    cudaFree(g->lr_rowid);
    g->lr_rowid = nullptr;
    uint64_t ends[2] = {0, 0};
    GB_CUDA(cudaMemcpyAsync(&ends[0], g->offs + sched.nheavy, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaMemcpyAsync(&ends[1], g->offs + g->zero_from, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaStreamSynchronize(s));
    if (ends[1] < ends[0]) GB_FAIL(GB_ERR_CUDA, "pagerank: light rows out of order");
    // one allocation: the run rows (uint32 per run), then a byte per arc
    const uint64_t narcs = ends[1] - ends[0];
    const uint64_t nruns = (narcs + kLightRun - 1) / kLightRun;
    GB_CUDA(cudaMalloc(&g->lr_rowid, sizeof(uint32_t) * std::max<uint64_t>(nruns, 1) + narcs + 16));
    if (g->zero_from > sched.nheavy) {
      uint32_t* runrow = g->lr_rowid;
      uint8_t* rowd = reinterpret_cast<uint8_t*>(g->lr_rowid + std::max<uint64_t>(nruns, 1));
      light_runrow_kernel<<<g->sm_count * 8, 256, 0, s>>>(g->offs, sched.nheavy, g->zero_from, ends[0], runrow);
      light_rowd_kernel<<<g->sm_count * 8, 256, 0, s>>>(g->offs, sched.nheavy, g->zero_from, ends[0], runrow, rowd);
    }
    GB_CUDA(cudaGetLastError());
    g->lr_row0 = sched.nheavy;
    g->lr_heavy = sched.heavy;
    g->lr_arc0 = ends[0];
    g->lr_arc1 = ends[1];
  }
  a->lr_runrow = g->lr_rowid;
  a->lr_rowd = reinterpret_cast<const uint8_t*>(
      g->lr_rowid + std::max<uint64_t>((g->lr_arc1 - g->lr_arc0 + kLightRun - 1) / kLightRun, 1));
  a->lr_arc0 = g->lr_arc0;
  a->lr_arc1 = g->lr_arc1;
  return GB_OK;
}

int run_pagerank(gb_graph* g, PrKind kind, float alpha, float tol, uint32_t max_iter, float* rank_out,
                 uint32_t* iters_out, gb_stats* stats, cudaStream_t s, float init = -1.f, float base = -1.f,
                 int linf = 0) {
  static_assert(sizeof(PrCtl) <= 4096, "PrCtl must fit the pinned readback area");
  if (!(alpha > 0.f && alpha < 1.f)) GB_FAIL(GB_ERR_ARG, "pagerank: alpha must be in (0,1)");
  if (!(tol >= 0.f)) GB_FAIL(GB_ERR_ARG, "pagerank: tolerance must be >= 0");
  if (max_iter == 0) GB_FAIL(GB_ERR_ARG, "pagerank: max_iter must be > 0");
  const gb_tuning t = effective_tuning(g);
  const uint32_t n = g->n;
  const bool out_dev = is_device_ptr(rank_out);
  int st = GB_OK;
  SweepSched sched{};
  if (kind == PrKind::Pull || kind == PrKind::PullResidual) {
    st = ensure_sweep_schedule(g, t.heavy_degree, t.tile_edges, s, &sched);
    if (st != GB_OK) return st;
    st = ensure_nout(g, s);
    if (st != GB_OK) return st;
  }
  FrontierLayout fl = frontier_layout(n, g->m, t.heavy_degree, t.tile_edges);
  // Async: the initial worklist (every vertex, 32 per chunk) plus room for
  // as many chunks again and the tiles of the heavy vertices
  const uint32_t nchunks = (uint32_t)(((uint64_t)n + 31) / 32);
  const unsigned long long cap = worklists::ring_capacity(2ull * nchunks + g->m / ((uint64_t)t.tile_edges * 32) + 8192);
  size_t need = carve_size<PrCtl>(1) + 5 * carve_size<float>(n) + (out_dev ? 0 : carve_size<float>(n));
  if (kind != PrKind::Pull) need += 2 * carve_size<float>(n);
  const uint32_t nheavy = g->perm ? std::min(sched.nheavy, kBinHubs) : 0;  // degree order: the first ids
  need += 2 * carve_size<double>(nheavy);
  if (kind == PrKind::Push) need += 3 * carve_size<uint32_t>(n) + fl.bytes;
  if (kind == PrKind::PushAsync) need += carve_size<char>(worklists::ring_bytes(cap));
  const bool rows = (kind == PrKind::Pull || kind == PrKind::PullResidual) && !g->perm;  // row sweeps in file order
  size_t hot = 0, sort_bytes = 0;
  if (rows) {
    st = hot_scratch(g, s, &hot, &sort_bytes);
    if (st != GB_OK) return st;
  }
  st = ws_reserve(g, std::max(need, hot), s);
  if (st != GB_OK && hot > need) {
    clear_error();
    hot = 0;
    g->prh = new (std::nothrow) PrHot;  // the columns stay: not tried again on every call
    st = ws_reserve(g, need, s);
  }
  if (st != GB_OK) return st;
  if (hot) {
    st = ensure_hot(g, sort_bytes, s);
    if (st != GB_OK) return st;
  }
  Carver cv(g->ws);
  PrArgs a{};
  a.ctl = cv.take<PrCtl>(1);
  a.c[0] = cv.take<float>(n);
  a.c[1] = cv.take<float>(n);
  a.acc = cv.take<float>(n);
  a.acc2 = cv.take<float>(n);
  a.hacc = cv.take<double>(2 * (size_t)nheavy);
  if (kind != PrKind::Pull) {
    a.residual = cv.take<float>(n);
    a.delta = cv.take<float>(n);
  }
  if (kind == PrKind::Push) {
    a.active[0] = cv.take<uint32_t>(n);
    a.active[1] = cv.take<uint32_t>(n);
    a.stamp = cv.take<uint32_t>(n);
    a.fq = carve_frontier(cv, fl);
  }
  if (kind == PrKind::PushAsync) a.ring = worklists::ring_layout(cv.take<char>(worklists::ring_bytes(cap)), cap);
  a.value = out_dev ? rank_out : cv.take<float>(n);
  a.offs = g->offs;
  a.col = g->col;
  a.nout = g->outdeg_of_stored;
  a.n = n;
  a.alpha = alpha;
  a.base = base >= 0.f ? base : (1.0f - alpha) / (float)n;  // PageRank-pull.cpp:200
  a.init = init >= 0.f ? init : 1.0f / (float)n;
  a.linf = linf;
  a.tol = tol;
  a.max_iter = max_iter;
  a.sched = sched;
  a.heavy = t.heavy_degree;
  a.tile = t.tile_edges;
  if (rows && g->prh && g->prh->col) {
    a.rank = g->prh->rank;
    a.col = g->prh->col;
  }
  GB_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(PrCtl), s));
  const void* kfn = nullptr;
  int block = kBlock;
  size_t smem = 0;
  if (kind == PrKind::Pull) {
    pr_pull_init<<<g->sm_count * 4, 256, 0, s>>>(a);
    a.zero_from = g->perm ? g->zero_from : n;
    kfn = reinterpret_cast<const void*>(&pr_pull_persistent<kBlock, 6>);
    // the flat sweep needs the degree order: heavy rows first, the light rows' arcs one range
    if (g->perm && (g->order == GB_ORDER_DEGREE || g->order == GB_ORDER_DEGREE_UNSORTED)) {
      // degree-ordered: the binned layout (sequential streams, few
      // (block, destination) runs per arc); where it cannot be built, the
      // flat sweep (heavy rows are [0, nheavy), the light rows' arcs one
      // contiguous range)
      if (ensure_pr_bins(g, s) == GB_OK) {
        const PrBins* b = g->prb;
        a.b_src = b->src;
        a.b_flag = b->flag;
        a.b_crun = b->crun;
        a.b_rdst = b->rdst;
        a.b_nheavy = nheavy;
        GB_CUDA(cudaMemsetAsync(a.hacc, 0, sizeof(double) * 2 * nheavy, s));
        a.b_tasks = b->tasks;
        a.b_ntasks = b->ntasks;
        kfn = reinterpret_cast<const void*>(&pr_pull_binned<kBinBlock>);
        block = kBinBlock;
        smem = kBinSmem;
        GB_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      } else {
        clear_error();
        st = light_run_table(g, sched, &a, s);
        if (st != GB_OK) return st;
        kfn = reinterpret_cast<const void*>(&pr_pull_flat<kBlock, 6>);
      }
    }
  } else if (kind == PrKind::PullResidual) {
    pr_resid_init<<<g->sm_count * 4, 256, 0, s>>>(a);
    GB_CUDA(cudaMemsetAsync(a.acc, 0, sizeof(float) * n, s));
    GB_CUDA(cudaMemsetAsync(a.acc2, 0, sizeof(float) * n, s));
    kfn = reinterpret_cast<const void*>(&pr_pull_residual_persistent);
    if (g->perm && (g->order == GB_ORDER_DEGREE || g->order == GB_ORDER_DEGREE_UNSORTED)) {
      if (ensure_pr_bins(g, s) == GB_OK) {  // else the row sweep
        const PrBins* b = g->prb;
        a.b_src = b->src;
        a.b_flag = b->flag;
        a.b_crun = b->crun;
        a.b_rdst = b->rdst;
        a.b_nheavy = nheavy;
        GB_CUDA(cudaMemsetAsync(a.hacc, 0, sizeof(double) * 2 * nheavy, s));
        a.b_tasks = b->tasks;
        a.b_ntasks = b->ntasks;
        kfn = reinterpret_cast<const void*>(&pr_resid_binned<kBinBlock>);
        block = kBinBlock;
        smem = kBinSmem;
        GB_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      } else {
        clear_error();
      }
    }
  } else if (kind == PrKind::Push) {
    pr_push_init<<<g->sm_count * 4, 256, 0, s>>>(a);
    kfn = reinterpret_cast<const void*>(&pr_push_persistent);
  } else {
    GB_CUDA(cudaMemsetAsync(a.ring.rc, 0, sizeof(worklists::RingCtl), s));
    pr_push_async_init<<<g->sm_count * 4, 256, 0, s>>>(a, nchunks);
    kfn = reinterpret_cast<const void*>(&pr_push_async);
  }
  GB_CUDA(cudaGetLastError());
  const int grid = coop_grid(g, kfn, block, smem, t.blocks_per_sm);
  if (grid <= 0) GB_FAIL(GB_ERR_CUDA, "pagerank: cannot size cooperative grid");
  void* args[] = {&a};
  KernelTimer kt(stats != nullptr, s);
  GB_CUDA(cudaLaunchCooperativeKernel(kfn, grid, block, args, smem, s));
  kt.stop(s);
  PrCtl* hc = reinterpret_cast<PrCtl*>(static_cast<char*>(g->pinned) + 4096);  // PrCtl is ~1 KB
  GB_CUDA(cudaMemcpyAsync(hc, a.ctl, sizeof(PrCtl), cudaMemcpyDeviceToHost, s));
  if (!out_dev) {
    st = copy_out(rank_out, a.value, sizeof(float) * n, s);
    if (st != GB_OK) return st;
  }
  if (stats || iters_out || !out_dev) {
    GB_CUDA(cudaStreamSynchronize(s));
    if (hc->err) return dev_err_status(hc->err, "pagerank");
    // Async has no rounds: one pass over the worklist
    if (kind == PrKind::PushAsync) hc->iters = 1;
    if (iters_out) *iters_out = hc->iters;
    if (stats) {
      *stats = gb_stats{};
      stats->vertices_reached = n;
      stats->edges_reached = g->m;
      stats->rounds = hc->iters;
      stats->relaxations = hc->pushes;
      if (kind == PrKind::PushAsync) stats->vertices_reached = hc->absorbs;  // residuals taken
      stats->launches = 2;
      stats->kernel_ms = kt.ms();
      double l1sum = 0.0;
      for (int k = 0; k < kL1Slots; ++k) l1sum += hc->l1[(hc->iters + 2) % 3][k];
      stats->residual = kind == PrKind::Pull ? (linf ? (double)bits_to_float(hc->linf[(hc->iters + 2) % 3]) : l1sum)
                                             : 0.0;
    }
    if (kind != PrKind::Push && kind != PrKind::PushAsync && hc->iters >= max_iter) {
      // the ranks are set; the status tells the caller the cap was hit
      gb::set_error("pagerank: failed to converge in %u iterations", hc->iters);
      return GB_ERR_NOT_CONVERGED;
    }
  }
  return GB_OK;
}

}  // namespace

// Entry wrapper: on a relabelled graph the ranks are computed in internal ids
// and mapped back (also when the iteration cap was hit: the ranks are set).
int pagerank_entry(gb_graph* g, PrKind kind, float alpha, float tol, uint32_t max_iter, float* rank_out,
                   uint32_t* iters_out, gb_stats* stats, cudaStream_t s, float init = -1.f, float base = -1.f,
                   int linf = 0) {
  if (!g->perm) return run_pagerank(g, kind, alpha, tol, max_iter, rank_out, iters_out, stats, s, init, base, linf);
  gb_stats local{};
  float* res = reinterpret_cast<float*>(result_buf(g, 0));
  int st = run_pagerank(g, kind, alpha, tol, max_iter, res, iters_out,
                        stats ? stats : (is_device_ptr(rank_out) ? nullptr : &local), s, init, base, linf);
  if (st != GB_OK && st != GB_ERR_NOT_CONVERGED) return st;
  if (stats) stats->launches += 1;  // the mapping gather
  const int fs = finish_f32(g, res, rank_out, s);
  return fs != GB_OK ? fs : st;
}

}  // namespace gb

extern "C" {

int gb_pagerank_pull(gb_graph* g, float alpha, float tol, uint32_t max_iter, float* rank_out,
                     uint32_t* iters_out, gb_stats* stats, void* stream) {
  gb::clear_error();
  if (!g || !rank_out) GB_FAIL(GB_ERR_ARG, "gb_pagerank_pull: null argument");
  GB_CUDA(cudaSetDevice(g->device));
  return gb::pagerank_entry(g, gb::PrKind::Pull, alpha, tol, max_iter, rank_out, iters_out, stats,
                            static_cast<cudaStream_t>(stream));
}

int gb_pagerank_pull_ex(gb_graph* g, float alpha, float tol, uint32_t max_iter, float init, float base,
                        int norm_linf, float* rank_out, uint32_t* iters_out, gb_stats* stats, void* stream) {
  gb::clear_error();
  if (!g || !rank_out) GB_FAIL(GB_ERR_ARG, "gb_pagerank_pull_ex: null argument");
  if (!(init >= 0.f) || !(base >= 0.f)) GB_FAIL(GB_ERR_ARG, "gb_pagerank_pull_ex: init and base must be >= 0");
  GB_CUDA(cudaSetDevice(g->device));
  return gb::pagerank_entry(g, gb::PrKind::Pull, alpha, tol, max_iter, rank_out, iters_out, stats,
                            static_cast<cudaStream_t>(stream), init, base, norm_linf ? 1 : 0);
}

int gb_pagerank_pull_residual(gb_graph* g, float alpha, float tol, uint32_t max_iter, float* rank_out,
                              uint32_t* iters_out, gb_stats* stats, void* stream) {
  gb::clear_error();
  if (!g || !rank_out) GB_FAIL(GB_ERR_ARG, "gb_pagerank_pull_residual: null argument");
  GB_CUDA(cudaSetDevice(g->device));
  return gb::pagerank_entry(g, gb::PrKind::PullResidual, alpha, tol, max_iter, rank_out, iters_out, stats,
                            static_cast<cudaStream_t>(stream));
}

int gb_pagerank_push(gb_graph* g, float alpha, float tol, uint32_t max_iter, float* rank_out,
                     uint32_t* iters_out, gb_stats* stats, void* stream) {
  gb::clear_error();
  if (!g || !rank_out) GB_FAIL(GB_ERR_ARG, "gb_pagerank_push: null argument");
  GB_CUDA(cudaSetDevice(g->device));
  return gb::pagerank_entry(g, gb::PrKind::Push, alpha, tol, max_iter, rank_out, iters_out, stats,
                            static_cast<cudaStream_t>(stream));
}

int gb_pagerank_push_ex(gb_graph* g, int algo, float alpha, float tol, uint32_t max_iter, float* rank_out,
                        uint32_t* iters_out, gb_stats* stats, void* stream) {
  gb::clear_error();
  if (!g || !rank_out) GB_FAIL(GB_ERR_ARG, "gb_pagerank_push_ex: null argument");
  if (algo != GB_PR_PUSH_ASYNC && algo != GB_PR_PUSH_SYNC) GB_FAIL(GB_ERR_ARG, "gb_pagerank_push_ex: unknown algo %d", algo);
  GB_CUDA(cudaSetDevice(g->device));
  return gb::pagerank_entry(g, algo == GB_PR_PUSH_ASYNC ? gb::PrKind::PushAsync : gb::PrKind::Push, alpha, tol,
                            max_iter, rank_out, iters_out, stats, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
