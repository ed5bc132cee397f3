// Batched personalised PageRank and its adjoint (differentiable PPR).
//
// No reference counterpart: an addition beside the PageRank kernels
// (lonestar/analytics/cpu/pagerank/PageRank-pull.cpp:196-251 is the
// un-personalised, unweighted pull iteration it generalises).
//
//   forward  x = (1-a) T + a W~ x,      W~_ij = w_ji / s_j,  s_j = sum_i w_ji
//   adjoint  lam = gx + a W~^T lam
//   grads    dL/dT = (1-a) lam
//            dL/dw_ji = a/s_j * sum_b x_j^b (lam_i^b - mu_j^b),
//            mu_j = (W~^T lam)_j = (lam_j - gx_j) / a
//
// B200 design: B right-hand sides stored vertex-major [n][B] so that, for
// B = 128, one arc's gather is a single coalesced 512-byte row (a float4 per
// lane) and the graph (column id + normalised weight, 8 bytes per arc) is
// read once per iteration for all B columns.  With fewer columns a row takes
// fewer lanes (B / 4, rounded up to a power of two) and the warp takes that
// many more arcs at once.  A warp takes the rows of a task one after another,
// the next row's column ids and weights already loaded, four 512-byte rows in
// flight; rows above the tile size are split into tiles whose partial rows
// are stored and then summed in arc order (the same result every time).  The forward pulls over the in-arcs of
// the device transpose, the adjoint over the out-arcs of the CSR; a row
// without arcs keeps its starting value and is not visited.  Each solve is
// one cooperative persistent launch; per-column L1 changes are reduced per
// block in shared memory and across blocks with fp64 atomics.  B = 1 (the
// plain single-vector solve) uses lanes over arcs instead of columns.
// RMAT-20, B = 128 (82 forward and 91 adjoint iterations): with tasks of up to
// 1024 arcs, four rows in flight and no loads ahead of the row, forward plus
// adjoint took 270 ms (a third of the warps' time waiting at the barriers);
// the walk above 187 ms, with more CTAs and fewer rows in flight each 173 ms,
// 1.0 ms an iteration or 8.2 TB/s of gathered rows (iterate_kernel below).
// 512-byte rows taken as 128- or 256-byte slices, a pass over the rows for
// each, hit L1 more often and still took 295 and 208 ms: the work per row is
// paid once for each slice.

#include <algorithm>
#include <vector>

#include "device_common.cuh"
#include "device_graph.cuh"

namespace gb {

int build_row_schedule(const uint64_t* offs, uint32_t n, uint64_t m, uint32_t heavy, uint32_t tile, int sm_count,
                       void* pinned, cudaStream_t s, uint2** tiles, uint32_t** heavy_list, uint32_t* ntiles,
                       uint32_t* nheavy);

namespace {

constexpr int kPprBlock = 256;
constexpr int kPprWarps = kPprBlock / 32;

// Arcs per tile, and per row above which a row is tiled: a sixteenth to an
// eighth of a warp's share of the arcs, so that the longest task ends with the
// others, from 32 (a small graph's iteration lasts as long as its longest
// task: 4 steps of gathers) to 512 (the partial rows stay under 1 byte per
// arc and column).
uint32_t ppr_tile(const gb_graph* g) {
  const uint64_t share = g->m / ((uint64_t)g->sm_count * 32);
  uint32_t t = 32;
  while (t < 512 && 16ull * t <= share) t *= 2;
  return t;
}

// Tiles whose partial rows one warp adds up, one after another.  A longer row
// is added up in two passes, span by span and then the spans' sums, with a grid
// barrier between; graphs without such a row do neither.  Forward + adjoint of a
// star of 500 K vertices, B = 4 / 128, ms: 135 / 315 with one warp for all 15 625
// tiles, 29 / 50 so; eight hubs of 62 K arcs 34 / 75, 22 / 43.  Spans of 128
// tiles took 20 / 41 there, but their pass and barrier cost RMAT-18, whose
// longest row has some 400, 3 to 6 %.
constexpr uint32_t kPprSpan = 512;

struct RowSched {
  uint2* tiles = nullptr;
  uint32_t ntiles = 0;
  uint32_t tile = 0;  // arcs per tile; a row of more is heavy
  bool spans = false;  // some row has more than kPprSpan tiles
};

struct PprState {
  RowSched fwd, bwd;      // over the transpose (in-arcs) and the CSR (out-arcs)
  float* s = nullptr;     // [n] out-weight sums
  float* wn = nullptr;    // [m] w / s_src, CSR order
  float* wn_t = nullptr;  // [m] the same, transpose order
  uint32_t* flags = nullptr;  // [n/32] rows with a non-zero source term
  double* l1 = nullptr;       // [3][128] per-column L1 change ring, then [128] ppr_seed's non-finite columns
  double* colnorm = nullptr;  // [128] per-column L1 norm of the adjoint's source term
  float* part = nullptr;      // [max(ntiles)][128] partial rows of the heavy rows' tiles
};

void free_state(gb_graph* g) {
  PprState* st = static_cast<PprState*>(g->ppr_state);
  if (!st) return;
  for (RowSched* r : {&st->fwd, &st->bwd}) cudaFree(r->tiles);
  cudaFree(st->s);
  cudaFree(st->wn);
  cudaFree(st->wn_t);
  cudaFree(st->flags);
  cudaFree(st->l1);
  cudaFree(st->colnorm);
  cudaFree(st->part);
  delete st;
  g->ppr_state = nullptr;
  g->ppr_free = nullptr;
}

// s_j = sum of out-arc weights; wn[e] = w[e] / s_j (one warp per row j)
__global__ void ppr_normalise(const uint64_t* __restrict__ offs, const float* __restrict__ w, uint32_t n,
                              float* __restrict__ s, float* __restrict__ wn) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t j = gw; j < n; j += nw) {
    const uint64_t b = offs[j], e = offs[j + 1];
    float acc = 0.f;
    for (uint64_t k = b + lane; k < e; k += 32) acc += w[k];
    acc = warp_sum(acc);
    if (lane == 0) s[j] = acc;
    const float inv = acc > 0.f ? 1.0f / acc : 0.f;
    for (uint64_t k = b + lane; k < e; k += 32) wn[k] = w[k] * inv;
  }
}

__global__ void ppr_permute(const float* __restrict__ wn, const uint64_t* __restrict__ emap, uint64_t m,
                            float* __restrict__ wn_t) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t e = tid; e < m; e += stride) wn_t[e] = wn[emap[e]];
}

// flags[r] = 1 if row r of src has a non-zero entry; both iterates start as
// scale * src (rows without arcs stay so).  A column with a value that is not
// finite never converges, wherever its row: bad[column] becomes NaN.
__global__ void ppr_seed(const float* __restrict__ src, float scale, uint32_t n, uint32_t B, uint32_t* flags,
                         float* __restrict__ dst, float* __restrict__ dst2, double* bad) {
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = lane_id();
  for (uint64_t r = gw; r < n; r += nw) {
    bool nz = false;
    for (uint32_t b = lane; b < B; b += 32) {
      const float v = src[r * B + b];
      nz |= v != 0.f;
      dst[r * B + b] = dst2[r * B + b] = scale * v;
      if (!isfinite(v)) bad[b] = nan("");
    }
    nz = __any_sync(kFull, nz);
    if (lane == 0 && nz) atomicOr(&flags[r >> 5], 1u << (r & 31));
  }
}

struct IterCtl {
  GridBar bar;
  int err;
  uint32_t iters;
};

struct IterArgs {
  const uint64_t* __restrict__ offs;  // rows: in-arcs (forward) or out-arcs (adjoint)
  const uint32_t* __restrict__ col;
  const float* __restrict__ wn;       // normalised weight per arc
  uint32_t n, B;
  const float* __restrict__ src;      // source term, [n][B]
  float src_scale;
  const uint32_t* __restrict__ flags;  // rows with a source term (nullptr: every row)
  float* buf[2];                       // buf[0] holds x0
  float alpha, tol;
  uint32_t max_iter;
  RowSched sched;
  float* part;  // [ntiles][B]
  double* l1;   // [3][128], then [128]: NaN for a column whose source term has a non-finite value
  const double* col_scale;  // per-column stopping scale (nullptr: 1)
  IterCtl* ctl;
};

__device__ __forceinline__ float4 f4_fma(float a, float4 x, float4 y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

// A batch of arcs of one row: lane l holds the column id (and weight) of the
// row's arc l, or of none.
struct ArcLoad {
  uint32_t c;
  float w;
};

__device__ __forceinline__ ArcLoad load_arcs(const uint32_t* __restrict__ col, const float* __restrict__ wn, uint64_t b,
                                             uint64_t e) {
  ArcLoad r{0u, 0.f};
  const uint64_t k = b + lane_id();
  if (k < e) {
    r.c = ldg(col + k);
    if (wn) r.w = ldg(wn + k);
  }
  return r;
}

// Rows of B floats handled by LPA lanes (4 columns each), G = 32 / LPA arcs
// per step; U steps in flight in the gradient (8 rows of 512 bytes at B = 128,
// at least two steps at small B; the iteration takes its own).
template <int LPA>
struct Wide {
  static constexpr int G = 32 / LPA;
  static constexpr int U = 8 / G > 2 ? 8 / G : 2;
};

// Sum over arcs [b, e) of wn * x[col] for this lane's 4 columns; `m` holds
// the row's first 32 arcs.  The first LPA lanes return the whole sum.
template <int LPA, int U>
__device__ __forceinline__ float4 row_sum(const IterArgs& a, const float* __restrict__ x, uint64_t b, uint64_t e,
                                          ArcLoad m) {
  constexpr int G = Wide<LPA>::G;
  const uint32_t lane = lane_id(), sub = lane % LPA, grp = lane / LPA;
  const bool act = 4 * sub < a.B;
  const float* __restrict__ xs = x + 4 * sub;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint64_t k0 = b; k0 < e; k0 += 32) {
    const uint32_t cnt = (uint32_t)(e - k0 < 32 ? e - k0 : 32);
    const ArcLoad nm = load_arcs(a.col, a.wn, k0 + 32, e);
    for (uint32_t u = 0; u < cnt; u += U * G) {
      float4 v[U];
      float w[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const uint32_t i = u + j * G + grp;
        const uint32_t c = __shfl_sync(kFull, m.c, i & 31);
        w[j] = __shfl_sync(kFull, m.w, i & 31);
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (act && i < cnt) v[j] = *reinterpret_cast<const float4*>(xs + (uint64_t)c * a.B);
        else w[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < U; ++j) acc = f4_fma(w[j], v[j], acc);
    }
    m = nm;
  }
  // lanes past a short row's arcs hold zeros: no step for them
  const uint32_t lanes = e - b < 32 / LPA ? (uint32_t)(e - b) * LPA : 32u;
#pragma unroll
  for (int o = LPA; o < 32; o <<= 1) {
    if (o >= lanes) break;  // uniform
    acc.x += __shfl_xor_sync(kFull, acc.x, o);
    acc.y += __shfl_xor_sync(kFull, acc.y, o);
    acc.z += __shfl_xor_sync(kFull, acc.z, o);
    acc.w += __shfl_xor_sync(kFull, acc.w, o);
  }
  return acc;
}

// Calls fn(row, first arc, end, its first 32 arcs) for the rows of a task of
// `rows` (a power of two, at most 32) consecutive rows that have between 1 and
// `tile` arcs; the next row's arcs are loaded before fn runs.
template <class Fn>
__device__ __forceinline__ void ppr_rows(const uint64_t* __restrict__ offs, const uint32_t* __restrict__ col,
                                         const float* __restrict__ wn, uint32_t n, uint64_t first, uint32_t rows,
                                         uint32_t tile, Fn&& fn) {
  const uint32_t lane = lane_id();
  uint64_t rb = 0;
  uint32_t rd = 0;
  if (lane < rows && first + lane < n) {
    rb = ldg(offs + first + lane);
    const uint64_t d = ldg(offs + first + lane + 1) - rb;
    rd = d <= tile ? (uint32_t)d : 0u;
  }
  unsigned todo = __ballot_sync(kFull, rd != 0);
  if (!todo) return;
  int k = __ffs(todo) - 1;
  uint64_t b = __shfl_sync(kFull, rb, k), e = b + __shfl_sync(kFull, rd, k);
  ArcLoad m = load_arcs(col, wn, b, e);
  while (true) {
    todo &= todo - 1;
    int k2 = 0;
    uint64_t b2 = 0, e2 = 0;
    ArcLoad m2{0u, 0.f};
    if (todo) {
      k2 = __ffs(todo) - 1;
      b2 = __shfl_sync(kFull, rb, k2), e2 = b2 + __shfl_sync(kFull, rd, k2);
      m2 = load_arcs(col, wn, b2, e2);
    }
    fn((uint32_t)(first + k), b, e, m);
    if (!todo) return;
    k = k2, b = b2, e = e2, m = m2;
  }
}

// Rows per task: 32, or fewer when there are too few rows for every warp; then
// half as many if that leaves fewer rows on the longest warp's path (a task's
// start, its offsets and then its first row's arcs, counted as two rows).  A
// 300 x 300 grid had 19 rows a warp in tasks of 16, so 32 for some: forward +
// adjoint, B = 4 / 128, 6.2 / 10.2 ms, now 4.9 / 8.2; 100 K vertices of mean
// degree 3 6.1 / 11.2, 4.8 / 9.2.
__device__ __forceinline__ uint32_t ppr_rows_per_task(uint32_t n, uint64_t nwarps) {
  uint32_t r = 32;
  while (r > 1 && (uint64_t)n < nwarps * r) r >>= 1;
  auto path = [&](uint32_t rows) { return ((uint64_t)n / rows + nwarps) / nwarps * (rows + 2); };
  return r >= 8 && path(r / 2) < path(r) ? r / 2 : r;
}

// LPA: lanes per row of B floats; 0 for B = 1 (lanes over arcs).
template <int LPA, int U, int MINB>
__global__ void __launch_bounds__(kPprBlock, MINB) ppr_iterate(IterArgs a) {
  constexpr bool WIDE = LPA != 0;
  constexpr int L = WIDE ? LPA : 1;
  __shared__ __align__(16) float s_diff[kPprWarps][128];  // written as float4
  __shared__ float s_acc[kPprWarps][32];  // B = 1: row sums of a task
  IterCtl* ctl = a.ctl;
  const uint64_t deadline = kernel_deadline();
  const uint64_t gtid = blockIdx.x * (uint64_t)kPprBlock + threadIdx.x;
  const uint64_t gthreads = (uint64_t)gridDim.x * kPprBlock;
  const uint64_t gwarp = gtid >> 5, nwarps = gthreads >> 5;
  const uint32_t lane = lane_id(), wib = threadIdx.x >> 5;
  const bool act = WIDE ? (lane < L && 4 * lane < a.B) : lane == 0;  // lanes that write a row
  const uint32_t tile = a.sched.tile;
  const uint32_t rpt = WIDE ? ppr_rows_per_task(a.n, nwarps) : 32;
  const uint64_t ntasks = a.sched.ntiles + ((uint64_t)a.n + rpt - 1) / rpt;
  s_acc[wib][lane] = 0.f;
  __syncwarp();
  for (uint32_t it = 0;; ++it) {
    const float* __restrict__ x = a.buf[it & 1];
    float* __restrict__ y = a.buf[(it + 1) & 1];
    if (blockIdx.x == 0 && threadIdx.x < 128) a.l1[((it + 1) % 3) * 128 + threadIdx.x] = 0.0;
    float4 dsum = make_float4(0.f, 0.f, 0.f, 0.f);
    auto finish = [&](uint32_t r, float4 acc, float4 o) {
      if (!act) return;
      const bool has_src = !a.flags || ((a.flags[r >> 5] >> (r & 31)) & 1u);
      const uint64_t base = (uint64_t)r * a.B + 4 * lane;
      float4 v = make_float4(a.alpha * acc.x, a.alpha * acc.y, a.alpha * acc.z, a.alpha * acc.w);
      if (has_src) v = f4_fma(a.src_scale, *reinterpret_cast<const float4*>(a.src + base), v);
      dsum.x += fabsf(v.x - o.x);
      dsum.y += fabsf(v.y - o.y);
      dsum.z += fabsf(v.z - o.z);
      dsum.w += fabsf(v.w - o.w);
      *reinterpret_cast<float4*>(y + base) = v;
    };
    auto finish1 = [&](uint32_t r, float acc) {
      float v = a.alpha * acc;
      if (!a.flags || ((a.flags[r >> 5] >> (r & 31)) & 1u)) v = fmaf(a.src_scale, a.src[r], v);
      dsum.x += fabsf(v - x[r]);
      y[r] = v;
    };
    auto old_row = [&](uint32_t r) {
      return act ? *reinterpret_cast<const float4*>(x + (uint64_t)r * a.B + 4 * lane)
                 : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    // this lane's columns of `cnt` partial rows, `step` tiles apart from tile t, in
    // order; stored in tile t's slot if asked
    auto sum_tiles = [&](uint64_t t, uint32_t cnt, uint32_t step, bool store) {
      float4* h = reinterpret_cast<float4*>(a.part + t * a.B) + lane;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (uint32_t k = 0; k < cnt; ++k) acc = f4_fma(1.f, h[(uint64_t)k * step * (a.B / 4)], acc);
      if (store) *h = acc;
      return acc;
    };
    for (uint64_t t = gwarp; t < ntasks; t += nwarps) {
      if (t < a.sched.ntiles) {  // one tile of a heavy row
        const uint2 tv = a.sched.tiles[t];
        const uint64_t vb = ldg(a.offs + tv.x), ve = ldg(a.offs + tv.x + 1);
        const uint64_t b = vb + (uint64_t)tv.y * tile, e = min(ve, b + tile);
        float* h = a.part + t * a.B;
        if constexpr (WIDE) {
          const float4 acc = row_sum<L, U>(a, x, b, e, load_arcs(a.col, a.wn, b, e));
          if (act) reinterpret_cast<float4*>(h)[lane] = acc;
        } else {
          float s = 0.f;
          for (uint64_t k = b + lane; k < e; k += 32) s = fmaf(ldg(a.wn + k), x[ldg(a.col + k)], s);
          s = warp_sum(s);
          if (lane == 0) *h = s;
        }
      } else if constexpr (WIDE) {
        ppr_rows(a.offs, a.col, a.wn, a.n, (t - a.sched.ntiles) * rpt, rpt, tile,
                 [&](uint32_t r, uint64_t b, uint64_t e, ArcLoad m) {
                   const float4 o = old_row(r);  // in flight beside the gathers
                   finish(r, row_sum<L, U>(a, x, b, e, m), o);
                 });
      } else {
        // 32 rows' arcs walked together, four steps of loads in flight; a
        // segmented sum per owner
        const uint64_t r = ((t - a.sched.ntiles) << 5) + lane;
        uint64_t b = 0;
        uint32_t d = 0;
        if (r < a.n) {
          b = ldg(a.offs + r);
          const uint64_t dd = ldg(a.offs + r + 1) - b;
          d = dd <= tile ? (uint32_t)dd : 0u;
        }
        warp_expand_mlp<4, float>(
            b, d, 0u, [&](bool valid, uint64_t e, uint32_t) { return valid ? ldg(a.col + e) : 0u; },
            [&](bool valid, uint64_t e, uint32_t c, uint32_t) { return valid ? ldg(a.wn + e) * x[c] : 0.f; },
            [&](bool valid, uint32_t owner, uint32_t, uint32_t, float v) {
              const uint32_t key = valid ? owner : 0xFFFFFFFFu;
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const float w = __shfl_down_sync(kFull, v, o);
                const uint32_t k2 = __shfl_down_sync(kFull, key, o);
                if (lane + o < 32 && k2 == key) v += w;
              }
              const uint32_t kp = __shfl_up_sync(kFull, key, 1);
              if (valid && (lane == 0 || kp != key)) s_acc[wib][owner] += v;
              __syncwarp();
            });
        const float sum = s_acc[wib][lane];
        s_acc[wib][lane] = 0.f;
        __syncwarp();
        if (d) finish1((uint32_t)r, sum);
      }
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    // rows of more than kPprSpan tiles: each span's sum, in tile order, into
    // its first tile's slot
    if (WIDE && a.sched.spans) {  // uniform
      for (uint64_t t = gwarp; t < a.sched.ntiles; t += nwarps) {
        const uint2 tv = a.sched.tiles[t];
        if (tv.y % kPprSpan != 0) continue;
        const uint64_t d = ldg(a.offs + tv.x + 1) - ldg(a.offs + tv.x);
        const uint32_t cnt = (uint32_t)((d + tile - 1) / tile);
        if (cnt > kPprSpan && act) sum_tiles(t, min(kPprSpan, cnt - tv.y), 1, true);
      }
      if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    }
    // heavy rows: their tiles follow one another from the one with k = 0
    for (uint64_t t = gwarp; t < a.sched.ntiles; t += nwarps) {
      const uint2 tv = a.sched.tiles[t];
      if (tv.y != 0) continue;
      const uint64_t d = ldg(a.offs + tv.x + 1) - ldg(a.offs + tv.x);
      const uint32_t cnt = (uint32_t)((d + tile - 1) / tile);
      if constexpr (WIDE) {
        if (!act) continue;
        const float4 o = old_row(tv.x);
        const float4 acc = cnt > kPprSpan ? sum_tiles(t, (cnt + kPprSpan - 1) / kPprSpan, kPprSpan, false)
                                          : sum_tiles(t, cnt, 1, false);
        finish(tv.x, acc, o);
      } else {
        float acc = 0.f;
        for (uint32_t k = lane; k < cnt; k += 32) acc += a.part[t + k];
        acc = warp_sum(acc);
        if (lane == 0) finish1(tv.x, acc);
      }
    }
    // per-column L1 change: block reduction, then one fp64 atomic per column
    if constexpr (WIDE) {
      if (act) *reinterpret_cast<float4*>(&s_diff[wib][4 * lane]) = dsum;
    } else {
      dsum.x = warp_sum(dsum.x);
      if (lane == 0) s_diff[wib][0] = dsum.x;
    }
    __syncthreads();
    if (threadIdx.x < a.B) {
      float sum = 0.f;
      for (int w = 0; w < kPprWarps; ++w) sum += s_diff[w][threadIdx.x];
      if (sum != 0.f) atomicAdd(&a.l1[(it % 3) * 128 + threadIdx.x], (double)sum);
    }
    if (!grid_barrier(&ctl->bar, gridDim.x, &ctl->err, deadline)) return;
    // converged when every column's L1 change is at most tol (times the
    // column's scale for the adjoint, whose source term is not normalised):
    // one thread per column
    bool done = true;
    if (threadIdx.x < a.B) {
      const double lim = (double)a.tol * (a.col_scale ? a.col_scale[threadIdx.x] : 1.0);
      done = *reinterpret_cast<volatile double*>(&a.l1[(it % 3) * 128 + threadIdx.x]) + a.l1[3 * 128 + threadIdx.x] <=
             lim;
    }
    done = __syncthreads_and(done);
    if (gtid == 0) ctl->iters = it + 1;
    if (done || it + 1 >= a.max_iter) break;
  }
}

// dL/dw for every arc of the CSR (rows = sources j):
//   g[e] = alpha/s_j * sum_b x_j^b (lam_i^b - mu_j^b),  mu_j = (lam_j - gx_j)/alpha
// Tasks as in ppr_iterate; the same number of lam rows in flight.
template <int LPA>
__global__ void __launch_bounds__(kPprBlock, LPA ? 3 : 4)
    ppr_grad_w(const uint64_t* __restrict__ offs, const uint32_t* __restrict__ col, const float* __restrict__ s,
               const float* __restrict__ x, const float* __restrict__ lam, const float* __restrict__ gx, uint32_t n,
               uint32_t B, float alpha, RowSched sched, float* __restrict__ grad_w) {
  constexpr bool WIDE = LPA != 0;
  constexpr int L = WIDE ? LPA : 1;
  const uint64_t gtid = blockIdx.x * (uint64_t)kPprBlock + threadIdx.x;
  const uint64_t gwarp = gtid >> 5, nwarps = ((uint64_t)gridDim.x * kPprBlock) >> 5;
  const uint32_t lane = lane_id();
  const float inv_alpha = 1.0f / alpha;
  auto run = [&](uint32_t j, uint64_t b, uint64_t e, ArcLoad m) {
    const float sj = s[j];
    const float scale = sj > 0.f ? alpha / sj : 0.f;
    if constexpr (WIDE) {
      constexpr int G = Wide<L>::G, U = Wide<L>::U;
      const uint32_t sub = lane % L, grp = lane / L;
      const bool act = 4 * sub < B;
      const float* __restrict__ ls = lam + 4 * sub;
      float4 xj = make_float4(0.f, 0.f, 0.f, 0.f), mj = xj;
      if (act) {
        const uint64_t base = (uint64_t)j * B + 4 * sub;
        xj = *reinterpret_cast<const float4*>(x + base);
        const float4 lj = *reinterpret_cast<const float4*>(lam + base);
        const float4 gj = *reinterpret_cast<const float4*>(gx + base);
        mj = make_float4((lj.x - gj.x) * inv_alpha, (lj.y - gj.y) * inv_alpha, (lj.z - gj.z) * inv_alpha,
                         (lj.w - gj.w) * inv_alpha);
      }
      for (uint64_t k0 = b; k0 < e; k0 += 32) {
        const uint32_t cnt = (uint32_t)(e - k0 < 32 ? e - k0 : 32);
        const ArcLoad nm = load_arcs(col, nullptr, k0 + 32, e);
        float out = 0.f;  // lane l: the gradient of arc k0 + l
        for (uint32_t u = 0; u < cnt; u += U * G) {
          float4 li[U];
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const uint32_t i = u + q * G + grp;
            const uint32_t c = __shfl_sync(kFull, m.c, i & 31);
            li[q] = mj;
            if (act && i < cnt) li[q] = *reinterpret_cast<const float4*>(ls + (uint64_t)c * B);
          }
#pragma unroll
          for (int q = 0; q < U; ++q) {
            float d = xj.x * (li[q].x - mj.x) + xj.y * (li[q].y - mj.y) + xj.z * (li[q].z - mj.z) +
                      xj.w * (li[q].w - mj.w);
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
            // arc u + q * G + g is held by group g: hand it to its lane
            const uint32_t at = lane - (u + q * G);  // wraps for lanes before it
            const float got = __shfl_sync(kFull, d, (at * L) & 31);
            if (at < (uint32_t)G) out = got;
          }
        }
        if (lane < cnt) grad_w[k0 + lane] = scale * out;
        m = nm;
      }
    } else {
      const float xj = x[j];
      const float mj = (lam[j] - gx[j]) * inv_alpha;
      for (uint64_t k = b + lane; k < e; k += 32) grad_w[k] = scale * xj * (lam[ldg(col + k)] - mj);
    }
  };
  const uint32_t rpt = ppr_rows_per_task(n, nwarps);
  const uint64_t ntasks = sched.ntiles + ((uint64_t)n + rpt - 1) / rpt;
  for (uint64_t t = gwarp; t < ntasks; t += nwarps) {
    if (t < sched.ntiles) {
      const uint2 tv = sched.tiles[t];
      const uint64_t vb = ldg(offs + tv.x), ve = ldg(offs + tv.x + 1);
      const uint64_t b = vb + (uint64_t)tv.y * sched.tile, e = min(ve, b + sched.tile);
      run(tv.x, b, e, load_arcs(col, nullptr, b, e));
    } else {
      ppr_rows(offs, col, nullptr, n, (t - sched.ntiles) * rpt, rpt, sched.tile, run);
    }
  }
}

// Lanes per row of B floats (0: one column).
int lanes_per_row(uint32_t B) {
  if (B == 1) return 0;
  int l = 1;
  while (4u * l < B) l *= 2;
  return l;
}

template <int LPA, int U, int MINB>
const void* iterate_ptr() {
  return reinterpret_cast<const void*>(&ppr_iterate<LPA, U, MINB>);
}

// Gathers in flight per warp against warps on the SM: four CTAs of 256 threads
// leave 64 registers, enough for four steps in flight (two for rows of at most
// 64 bytes), and hide more than three CTAs with twice the steps.  Forward +
// adjoint, edge factor 16, three CTAs / four, ms: RMAT-20 B = 128 187 / 173,
// 64 127 / 108, 32 106 / 76, 12 72 / 61, 8 57 / 51, 4 51 / 44; 30 K vertices
// B = 128 7.5 / 7.05, 32 3.95 / 3.6, 12 5.1 / 4.6.  At
// 16 lanes per row nothing is gained while the iterate fits L2 (B = 64, 200 K
// vertices 25.3 / 26.7, 90 K 9.8 / 10.0), and three CTAs stay.
constexpr uint64_t kL2Iterate = 126ull << 20;

const void* iterate_kernel(uint32_t B, uint32_t n) {
  switch (lanes_per_row(B)) {
    case 0: return iterate_ptr<0, 2, 4>();
    case 1: return iterate_ptr<1, 2, 4>();
    case 2: return iterate_ptr<2, 2, 4>();
    case 4: return iterate_ptr<4, 2, 4>();
    case 8: return iterate_ptr<8, 4, 4>();
    case 16: return sizeof(float) * B * (uint64_t)n > kL2Iterate ? iterate_ptr<16, 4, 4>() : iterate_ptr<16, 4, 3>();
    default: return iterate_ptr<32, 4, 4>();
  }
}

const void* grad_kernel(uint32_t B) {
  switch (lanes_per_row(B)) {
    case 0: return reinterpret_cast<const void*>(&ppr_grad_w<0>);
    case 1: return reinterpret_cast<const void*>(&ppr_grad_w<1>);
    case 2: return reinterpret_cast<const void*>(&ppr_grad_w<2>);
    case 4: return reinterpret_cast<const void*>(&ppr_grad_w<4>);
    case 8: return reinterpret_cast<const void*>(&ppr_grad_w<8>);
    case 16: return reinterpret_cast<const void*>(&ppr_grad_w<16>);
    default: return reinterpret_cast<const void*>(&ppr_grad_w<32>);
  }
}

// *any = 1 if some row has more than kPprSpan tiles.
__global__ void ppr_any_span(const uint2* __restrict__ tiles, uint32_t ntiles, uint32_t* any) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x)
    if (tiles[t].y == kPprSpan) *any = 1;
}

// out[c] = sum_r |src[r][c]| for the B columns of a vertex-major [n][B] array.
__global__ void ppr_colnorm(const float* __restrict__ src, uint32_t n, uint32_t B, double* out) {
  __shared__ double s_sum[128];
  for (uint32_t c = threadIdx.x; c < 128; c += blockDim.x) s_sum[c] = 0.0;
  __syncthreads();
  const uint32_t rows_per_pass = blockDim.x / B;  // threads past rows_per_pass * B stay idle
  const uint32_t c = threadIdx.x % B, r0 = threadIdx.x / B;
  double acc = 0.0;
  if (r0 < rows_per_pass)
    for (uint64_t r = (uint64_t)blockIdx.x * rows_per_pass + r0; r < n; r += (uint64_t)gridDim.x * rows_per_pass)
      acc += fabs((double)src[r * B + c]);
  if (r0 < rows_per_pass) atomicAdd(&s_sum[c], acc);
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < B; k += blockDim.x)
    if (s_sum[k] != 0.0) atomicAdd(&out[k], s_sum[k]);
}

__global__ void ppr_scale(const float* __restrict__ src, float scale, uint64_t count, float* __restrict__ dst) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < count; i += stride) dst[i] = scale * src[i];
}

int build_state(gb_graph* g, PprState* st, cudaStream_t s) {
  const uint32_t n = g->n;
  const uint64_t m = g->m;
  const uint32_t tile = ppr_tile(g);
  st->fwd.tile = st->bwd.tile = tile;
  for (RowSched* r : {&st->fwd, &st->bwd}) {
    uint32_t *heavy = nullptr, nheavy = 0;  // not needed: a heavy row is the tiles behind its first one
    const int rc = build_row_schedule(r == &st->fwd ? g->t_offs : g->offs, n, m, tile, tile, g->sm_count, g->pinned, s,
                                      &r->tiles, &heavy, &r->ntiles, &nheavy);
    cudaFree(heavy);
    if (rc != GB_OK) return rc;
  }
  const size_t ntiles = std::max<size_t>(1, std::max(st->fwd.ntiles, st->bwd.ntiles));
  GB_CUDA(cudaMalloc(&st->part, sizeof(float) * 128 * ntiles));
  GB_CUDA(cudaMalloc(&st->s, sizeof(float) * n));
  GB_CUDA(cudaMalloc(&st->wn, sizeof(float) * std::max<uint64_t>(m, 1)));
  GB_CUDA(cudaMalloc(&st->wn_t, sizeof(float) * std::max<uint64_t>(m, 1)));
  GB_CUDA(cudaMalloc(&st->flags, sizeof(uint32_t) * ((n + 31) / 32)));
  GB_CUDA(cudaMalloc(&st->l1, sizeof(double) * 4 * 128));
  GB_CUDA(cudaMalloc(&st->colnorm, sizeof(double) * 128));
  uint32_t* any = reinterpret_cast<uint32_t*>(st->l1);  // scratch until the first solve
  uint32_t* h_any = static_cast<uint32_t*>(g->pinned);
  GB_CUDA(cudaMemsetAsync(any, 0, 2 * sizeof(uint32_t), s));
  ppr_any_span<<<g->sm_count, 256, 0, s>>>(st->fwd.tiles, st->fwd.ntiles, any);
  ppr_any_span<<<g->sm_count, 256, 0, s>>>(st->bwd.tiles, st->bwd.ntiles, any + 1);
  GB_CUDA(cudaGetLastError());
  GB_CUDA(cudaMemcpyAsync(h_any, any, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GB_CUDA(cudaStreamSynchronize(s));
  st->fwd.spans = h_any[0] != 0;
  st->bwd.spans = h_any[1] != 0;
  return GB_OK;
}

int ensure_state(gb_graph* g, cudaStream_t s, PprState** out) {
  int rc = ensure_transpose(g, s);
  if (rc != GB_OK) return rc;
  if (!g->ppr_state) {
    PprState* st = new (std::nothrow) PprState();
    if (!st) GB_FAIL(GB_ERR_OOM, "ppr: host allocation failed");
    g->ppr_state = st;
    g->ppr_free = free_state;
    rc = build_state(g, st, s);
    if (rc != GB_OK) {  // whole or not at all: a later call may find the memory
      free_state(g);
      return rc;
    }
  }
  *out = static_cast<PprState*>(g->ppr_state);
  return GB_OK;
}

int prepare_weights(gb_graph* g, PprState* st, const float* w, cudaStream_t s) {
  if (!w) w = g->wf;
  if (!w) GB_FAIL(GB_ERR_ARG, "ppr: no arc weights (pass w or upload w_f32)");
  if (w != g->wf && !is_device_ptr(w)) GB_FAIL(GB_ERR_ARG, "ppr: w must be device memory");
  ppr_normalise<<<g->sm_count * 8, 256, 0, s>>>(g->offs, w, g->n, st->s, st->wn);
  ppr_permute<<<g->sm_count * 8, 256, 0, s>>>(st->wn, g->t_emap, g->m, st->wn_t);
  GB_CUDA(cudaGetLastError());
  return GB_OK;
}

// One Jacobi solve x = scale*src + alpha * M x (M = W~ or W~^T) into `out`.
int solve(gb_graph* g, PprState* st, bool adjoint, uint32_t B, const float* src, float scale, float alpha, float tol,
          uint32_t max_iter, float* out, float* tmp, IterCtl* ctl, uint32_t* iters, double* kernel_ms,
          cudaStream_t s) {
  IterArgs a{};
  a.offs = adjoint ? g->offs : g->t_offs;
  a.col = adjoint ? g->col : g->t_col;
  a.wn = adjoint ? st->wn : st->wn_t;
  a.sched = adjoint ? st->bwd : st->fwd;
  a.n = g->n;
  a.B = B;
  a.src = src;
  a.src_scale = scale;
  a.flags = adjoint ? nullptr : st->flags;
  a.buf[0] = out;
  a.buf[1] = tmp;
  a.alpha = alpha;
  a.tol = tol;
  a.max_iter = max_iter;
  a.part = st->part;
  a.l1 = st->l1;
  a.col_scale = adjoint ? st->colnorm : nullptr;
  a.ctl = ctl;
  if (adjoint) {
    // the adjoint's source term (the loss gradient) has arbitrary scale: stop
    // on the L1 change relative to each column's L1 norm
    GB_CUDA(cudaMemsetAsync(st->colnorm, 0, sizeof(double) * 128, s));
    ppr_colnorm<<<g->sm_count * 4, 256, 0, s>>>(src, g->n, B, st->colnorm);
  }
  GB_CUDA(cudaMemsetAsync(ctl, 0, sizeof(IterCtl), s));
  GB_CUDA(cudaMemsetAsync(st->l1, 0, sizeof(double) * 4 * 128, s));
  GB_CUDA(cudaMemsetAsync(st->flags, 0, sizeof(uint32_t) * ((g->n + 31) / 32), s));
  ppr_seed<<<g->sm_count * 8, 256, 0, s>>>(src, scale, g->n, B, st->flags, out, tmp, st->l1 + 3 * 128);  // x0 = scale * src
  GB_CUDA(cudaGetLastError());
  const void* kfn = iterate_kernel(B, g->n);
  int grid = coop_grid(g, kfn, kPprBlock, 0, 0);
  // no more CTAs than there is work for: every CTA takes part in the barriers
  const uint64_t work = a.sched.ntiles + (B > 1 ? (uint64_t)g->n : ((uint64_t)g->n + 31) / 32);
  grid = (int)std::min<uint64_t>(grid, (work + kPprWarps - 1) / kPprWarps);
  if (grid <= 0) GB_FAIL(GB_ERR_CUDA, "ppr: cannot size cooperative grid");
  void* args[] = {&a};
  KernelTimer kt(true, s);
  GB_CUDA(cudaLaunchCooperativeKernel(kfn, grid, kPprBlock, args, 0, s));
  kt.stop(s);
  IterCtl* hc = reinterpret_cast<IterCtl*>(static_cast<char*>(g->pinned) + 1024);
  GB_CUDA(cudaMemcpyAsync(hc, ctl, sizeof(IterCtl), cudaMemcpyDeviceToHost, s));
  GB_CUDA(cudaStreamSynchronize(s));
  if (hc->err) return dev_err_status(hc->err, "ppr");
  *iters = hc->iters;
  *kernel_ms += kt.ms();
  if (hc->iters & 1) GB_CUDA(cudaMemcpyAsync(out, tmp, sizeof(float) * (size_t)g->n * B, cudaMemcpyDeviceToDevice, s));
  return GB_OK;
}

// Rows of several columns are read and written 16 bytes at a time.
int check_aligned(uint32_t B, const float* p, const char* what) {
  if (B > 1 && reinterpret_cast<uintptr_t>(p) % 16 != 0)
    GB_FAIL(GB_ERR_ARG, "ppr: %s must start on a 16-byte boundary (B > 1)", what);
  return GB_OK;
}

int check_common(gb_graph* g, uint32_t B, float alpha, uint32_t max_iter) {
  // teleport / rank / arc-weight arrays are indexed by the caller's ids and arcs
  if (g->perm) GB_FAIL(GB_ERR_UNSUPPORTED, "ppr: graph was relabelled; PPR needs file order");
  if (!(B == 1 || (B % 4 == 0 && B >= 4 && B <= 128))) GB_FAIL(GB_ERR_ARG, "ppr: B must be 1 or a multiple of 4 <= 128");
  if (!(alpha > 0.f && alpha < 1.f)) GB_FAIL(GB_ERR_ARG, "ppr: alpha must be in (0,1)");
  if (max_iter == 0) GB_FAIL(GB_ERR_ARG, "ppr: max_iter must be > 0");
  if (g->m >= (1ull << 32)) GB_FAIL(GB_ERR_UNSUPPORTED, "ppr: limited to < 2^32 arcs");
  return GB_OK;
}

}  // namespace
}  // namespace gb

extern "C" int gb_ppr_forward(gb_graph* g, uint32_t B, const float* teleport, const float* w, float alpha, float tol,
                              uint32_t max_iter, float* x_out, uint32_t* iters_out, gb_stats* stats, void* stream) {
  using namespace gb;
  clear_error();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!g || !teleport || !x_out) GB_FAIL(GB_ERR_ARG, "gb_ppr_forward: null argument");
  int rc = check_common(g, B, alpha, max_iter);
  if (rc != GB_OK) return rc;
  GB_CUDA(cudaSetDevice(g->device));
  if (!is_device_ptr(teleport) || !is_device_ptr(x_out)) GB_FAIL(GB_ERR_ARG, "gb_ppr_forward: arrays must be device memory");
  if ((rc = check_aligned(B, teleport, "teleport")) != GB_OK) return rc;
  if ((rc = check_aligned(B, x_out, "x_out")) != GB_OK) return rc;
  PprState* st = nullptr;
  if ((rc = ensure_state(g, s, &st)) != GB_OK) return rc;
  if ((rc = prepare_weights(g, st, w, s)) != GB_OK) return rc;
  const size_t need = carve_size<IterCtl>(1) + carve_size<float>((size_t)g->n * B);
  if ((rc = ws_reserve(g, need, s)) != GB_OK) return rc;
  Carver cv(g->ws);
  IterCtl* ctl = cv.take<IterCtl>(1);
  float* tmp = cv.take<float>((size_t)g->n * B);
  uint32_t iters = 0;
  double ms = 0.0;
  if ((rc = solve(g, st, false, B, teleport, 1.0f - alpha, alpha, tol, max_iter, x_out, tmp, ctl, &iters, &ms, s)) != GB_OK)
    return rc;
  if (iters_out) *iters_out = iters;
  if (stats) {
    GB_CUDA(cudaStreamSynchronize(s));
    *stats = gb_stats{};
    stats->rounds = iters;
    stats->edges_reached = g->m;
    stats->vertices_reached = g->n;
    stats->launches = 5;
    stats->kernel_ms = ms;
  }
  if (iters >= max_iter) {
    set_error("gb_ppr_forward: failed to converge in %u iterations", iters);
    return GB_ERR_NOT_CONVERGED;
  }
  return GB_OK;
}

extern "C" int gb_ppr_backward(gb_graph* g, uint32_t B, const float* x, const float* gx, const float* w, float alpha,
                               float tol, uint32_t max_iter, float* grad_teleport, float* grad_w, uint32_t* iters_out,
                               gb_stats* stats, void* stream) {
  using namespace gb;
  clear_error();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!g || !x || !gx) GB_FAIL(GB_ERR_ARG, "gb_ppr_backward: null argument");
  int rc = check_common(g, B, alpha, max_iter);
  if (rc != GB_OK) return rc;
  GB_CUDA(cudaSetDevice(g->device));
  if (!is_device_ptr(x) || !is_device_ptr(gx) || (grad_teleport && !is_device_ptr(grad_teleport)) ||
      (grad_w && !is_device_ptr(grad_w)))
    GB_FAIL(GB_ERR_ARG, "gb_ppr_backward: arrays must be device memory");
  if ((rc = check_aligned(B, x, "x")) != GB_OK) return rc;
  if ((rc = check_aligned(B, gx, "gx")) != GB_OK) return rc;
  PprState* st = nullptr;
  if ((rc = ensure_state(g, s, &st)) != GB_OK) return rc;
  if ((rc = prepare_weights(g, st, w, s)) != GB_OK) return rc;
  const size_t nb = (size_t)g->n * B;
  const size_t need = carve_size<IterCtl>(1) + 2 * carve_size<float>(nb);
  if ((rc = ws_reserve(g, need, s)) != GB_OK) return rc;
  Carver cv(g->ws);
  IterCtl* ctl = cv.take<IterCtl>(1);
  float* lam = cv.take<float>(nb);
  float* tmp = cv.take<float>(nb);
  uint32_t iters = 0;
  double ms = 0.0;
  rc = solve(g, st, true, B, gx, 1.0f, alpha, tol, max_iter, lam, tmp, ctl, &iters, &ms, s);
  if (rc != GB_OK) return rc;
  KernelTimer kt(stats != nullptr, s);
  if (grad_teleport) ppr_scale<<<g->sm_count * 8, 256, 0, s>>>(lam, 1.0f - alpha, nb, grad_teleport);
  if (grad_w) {
    void* args[] = {&g->offs, &g->col, &st->s, &x, &lam, &gx, &g->n, &B, &alpha, &st->bwd, &grad_w};
    GB_CUDA(cudaLaunchKernel(grad_kernel(B), g->sm_count * 8, kPprBlock, args, 0, s));
  }
  kt.stop(s);
  GB_CUDA(cudaGetLastError());
  if (iters_out) *iters_out = iters;
  if (stats) {
    GB_CUDA(cudaStreamSynchronize(s));
    *stats = gb_stats{};
    stats->rounds = iters;
    stats->edges_reached = g->m;
    stats->vertices_reached = g->n;
    stats->launches = 7;
    stats->kernel_ms = ms + kt.ms();
  }
  if (iters >= max_iter) {
    set_error("gb_ppr_backward: failed to converge in %u iterations", iters);
    return GB_ERR_NOT_CONVERGED;
  }
  return GB_OK;
}
