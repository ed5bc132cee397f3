// Many disjoint graphs in one launch: BFS + CC over a block-diagonal packing.
//
// Config of the reference build plan: 512 uneven Erdos-Renyi graphs with BFS
// and CC per graph.  Looping gb_bfs / gb_cc per graph pays two launches and a
// host round trip per small graph; here the graphs share ONE device mirror
// (vertex ranges graph_first[k] .. graph_first[k+1]-1, no arc crossing a
// range) and
//   * BFS runs once from the super-source {graph_first[k] + local_src[k]}:
//     since no arc leaves a graph, every vertex gets exactly the level it has
//     in its own graph's BFS (lonestar/analytics/cpu/bfs/bfs.cpp:244-293);
//   * CC labels every vertex with the minimum GLOBAL id of its component,
//     which is graph_first[k] plus the minimum LOCAL id -- the label LabelProp
//     converges to per graph (ConnectedComponents.cpp:183-230) -- so one
//     subtraction localises it.  When the levels are asked for too, what the
//     BFS reached in graph k IS the component of its source: its label is its
//     least id, no arc is read for it, and union-find (larger root under the
//     smaller) runs over the arcs of the unreached vertices only.  512
//     Erdos-Renyi graphs of 1 K - 200 K vertices, mean degree 8: union-find
//     over every arc took 4.1 of 5.5 ms; the call now takes 1.5 ms.  A call
//     for the labels alone runs union-find over all arcs.
// After the first call on a layout (validation, buffer set-up) the call
// issues only stream-ordered work when the outputs are device pointers, so it
// can be captured in a CUDA graph and replayed.

#include <cstring>
#include <vector>

#include "device_common.cuh"
#include "device_graph.cuh"
#include "sweep.cuh"
#include "union_find.cuh"

namespace gb {

int run_bfs_sources(gb_graph* g, const uint32_t* d_srcs, uint32_t k, uint32_t* d_level, cudaStream_t s);
int run_cc(gb_graph* g, int algo, uint32_t* label_out, gb_stats* stats, cudaStream_t s);

namespace {

__device__ __forceinline__ uint32_t graph_of(const uint32_t* __restrict__ gf, uint32_t ng, uint32_t v) {
  uint32_t lo = 0, hi = ng;  // largest k with gf[k] <= v
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (gf[mid] <= v) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void mg_validate(const uint64_t* __restrict__ offs, const uint32_t* __restrict__ col, uint32_t n,
                            const uint32_t* __restrict__ gf, uint32_t ng, int* bad) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = tid; v < n; v += stride) {
    const uint32_t k = graph_of(gf, ng, (uint32_t)v);
    const uint32_t lo = gf[k], hi = gf[k + 1];
    for (uint64_t e = offs[v]; e < offs[v + 1]; ++e) {
      const uint32_t u = col[e];
      if (u < lo || u >= hi) {
        atomicOr(bad, 1);
        break;
      }
    }
  }
}

__global__ void mg_localize(uint32_t* __restrict__ label, uint32_t n, const uint32_t* __restrict__ gf, uint32_t ng) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = tid; v < n; v += stride) label[v] -= gf[graph_of(gf, ng, (uint32_t)v)];
}

// Walks the chunks of 32 consecutive vertices of this warp's contiguous share
// of [0, n): fn(v, valid, k) with k the graph of v, by all lanes.
template <class Fn>
__device__ __forceinline__ void mg_walk(uint32_t n, const uint32_t* __restrict__ gf, uint32_t ng, Fn&& fn) {
  const uint64_t gwarp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nchunks = ((uint64_t)n + 31) >> 5;
  const uint64_t per = (nchunks + nwarps - 1) / nwarps;
  const uint64_t c0 = gwarp * per, c1 = c0 + per < nchunks ? c0 + per : nchunks;
  if (c0 >= c1) return;
  uint32_t k = graph_of(gf, ng, (uint32_t)(c0 << 5));
  for (uint64_t c = c0; c < c1; ++c) {
    const uint64_t v = (c << 5) + lane_id();
    const bool valid = v < n;
    if (valid)
      while (gf[k + 1] <= v) ++k;
    fn((uint32_t)v, valid, k);
    k = __shfl_sync(kFull, k, 0);  // the next chunk starts at or after this one's first graph
  }
}

// root[k] = least id that the BFS reached in graph k; unreached vertices
// become their own parents.  Every warp but the first of a graph finds
// root[k] at or below its own ids, so few atomics are sent.
__global__ void mg_roots(const uint32_t* __restrict__ level, uint32_t n, const uint32_t* __restrict__ gf, uint32_t ng,
                         uint32_t* root, uint32_t* __restrict__ p) {
  mg_walk(n, gf, ng, [&](uint32_t v, bool valid, uint32_t k) {
    const bool reached = valid && level[v] != kInf;
    if (valid && !reached) p[v] = v;
    if (reached && v < *reinterpret_cast<volatile uint32_t*>(&root[k])) atomicMin(&root[k], v);
  });
}

// Union-find over the arcs of the unreached vertices (their neighbours are
// unreached too: the graphs are symmetric, so each edge is taken once): tasks
// of 32 consecutive rows, then the heavy rows' tiles, so that no warp walks
// the row of an unreached hub alone (the call on one graph of 1 M vertices
// whose unreached component is a star: 10.9 ms by a warp per row, 0.086 with
// tiles; eight of 100 K 1.12 / 0.083).
__global__ void mg_link(const uint32_t* __restrict__ level, const uint64_t* __restrict__ offs,
                        const uint32_t* __restrict__ col, uint32_t n, SweepSched sched, uint32_t* p) {
  const uint64_t gwarp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nchunks = ((uint64_t)n + 31) >> 5;
  for (uint64_t c = gwarp; c < nchunks + sched.ntiles; c += nwarps) {
    if (c >= nchunks) {
      const uint2 tv = sched.tiles[c - nchunks];
      if (level[tv.x] != kInf) continue;
      const uint64_t vb = ldg(offs + tv.x), ve = ldg(offs + tv.x + 1);
      const uint64_t b = vb + (uint64_t)tv.y * sched.tile, e = min(ve, b + sched.tile);
      for (uint64_t j = b + lane_id(); j < e; j += 32) {
        const uint32_t u = ldg(col + j);
        if (u < tv.x) link(p, tv.x, u);
      }
      continue;
    }
    const uint64_t v = (c << 5) + lane_id();
    const bool mine = v < n && level[v] == kInf;
    if (!__any_sync(kFull, mine)) continue;
    uint64_t b = 0;
    uint32_t d = 0;
    if (mine) {
      b = ldg(offs + v);
      const uint64_t dd = ldg(offs + v + 1) - b;
      d = dd > sched.heavy ? 0u : (uint32_t)dd;
    }
    warp_expand(b, d, (uint32_t)v, [&](bool on, uint64_t e, uint32_t, uint32_t x) {
      if (!on) return;
      const uint32_t u = ldg(col + e);
      if (u < x) link(p, x, u);
    });
  }
}

__global__ void mg_label(const uint32_t* __restrict__ level, uint32_t n, const uint32_t* __restrict__ gf, uint32_t ng,
                         const uint32_t* __restrict__ root, const uint32_t* __restrict__ p,
                         uint32_t* __restrict__ label) {
  mg_walk(n, gf, ng, [&](uint32_t v, bool valid, uint32_t k) {
    if (!valid) return;
    uint32_t r;
    if (level[v] != kInf) {
      r = root[k];
    } else {
      r = v;
      while (p[r] != r) r = p[r];
    }
    label[v] = r - gf[k];
  });
}

// CC labels of every graph from its BFS levels (see the file comment).
int cc_from_levels(gb_graph* g, const uint32_t* d_level, uint32_t ng, uint32_t* d_label, cudaStream_t s) {
  // the heavy rows' tiles, when some row needs them (built once per graph; a
  // call that is captured before that was done walks every row by a warp)
  const gb_tuning t = effective_tuning(g);
  SweepSched sched{};
  sched.heavy = 0xFFFFFFFFu;
  if (g->max_degree > t.heavy_degree) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool built = g->sweep_tiles && g->sweep_heavy == t.heavy_degree && g->sweep_tile == t.tile_edges;
    if (!built) GB_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap == cudaStreamCaptureStatusNone) {
      const int rc = ensure_sweep_schedule(g, t.heavy_degree, t.tile_edges, s, &sched);
      if (rc != GB_OK) return rc;
    }
  }
  // after the BFS: its workspace is free again, and holds two queues of n ids
  const size_t need = carve_size<uint32_t>(ng) + carve_size<uint32_t>(g->n);
  int st = ws_reserve(g, need, s);
  if (st != GB_OK) return st;
  Carver cv(g->ws);
  uint32_t* root = cv.take<uint32_t>(ng);
  uint32_t* p = cv.take<uint32_t>(g->n);
  GB_CUDA(cudaMemsetAsync(root, 0xFF, sizeof(uint32_t) * ng, s));
  const int blocks = g->sm_count * 8;
  mg_roots<<<blocks, 256, 0, s>>>(d_level, g->n, g->mg_first, ng, root, p);
  mg_link<<<blocks, 256, 0, s>>>(d_level, g->offs, g->col, g->n, sched, p);
  mg_label<<<blocks, 256, 0, s>>>(d_level, g->n, g->mg_first, ng, root, p, d_label);
  GB_CUDA(cudaGetLastError());
  return GB_OK;
}

uint64_t fnv1a(const uint32_t* p, size_t k) {
  uint64_t h = 1469598103934665603ull;
  for (size_t i = 0; i < k; ++i) {
    h ^= p[i];
    h *= 1099511628211ull;
  }
  return h;
}

// Validate and cache the layout (first call for a layout only).
int prepare_layout(gb_graph* g, const uint32_t* gf, uint32_t ng, cudaStream_t s) {
  const uint64_t h = fnv1a(gf, (size_t)ng + 1) ^ ng;
  if (g->mg_first && g->mg_ngraphs == ng && g->mg_hash == h) return GB_OK;
  if (gf[0] != 0 || gf[ng] != g->n) GB_FAIL(GB_ERR_ARG, "multi-graph: graph_first must start at 0 and end at n");
  for (uint32_t k = 0; k < ng; ++k)
    if (gf[k + 1] <= gf[k]) GB_FAIL(GB_ERR_ARG, "multi-graph: graph %u is empty or ranges are not increasing", k);
  cudaFree(g->mg_first);
  cudaFree(g->mg_src);
  cudaFree(g->mg_level);
  cudaFree(g->mg_label);
  if (g->mg_stage) cudaFreeHost(g->mg_stage);
  g->mg_first = g->mg_src = g->mg_level = g->mg_label = g->mg_stage = nullptr;
  g->mg_ngraphs = 0;
  GB_CUDA(cudaMalloc(&g->mg_first, sizeof(uint32_t) * (ng + 1)));
  GB_CUDA(cudaMalloc(&g->mg_src, sizeof(uint32_t) * ng));
  GB_CUDA(cudaMalloc(&g->mg_level, sizeof(uint32_t) * g->n));
  GB_CUDA(cudaMalloc(&g->mg_label, sizeof(uint32_t) * g->n));
  GB_CUDA(cudaMallocHost(&g->mg_stage, sizeof(uint32_t) * (2 * (size_t)ng + 1)));
  GB_CUDA(cudaMemcpyAsync(g->mg_first, gf, sizeof(uint32_t) * (ng + 1), cudaMemcpyHostToDevice, s));
  int* dbad = reinterpret_cast<int*>(g->mg_src);  // scratch before sources are written
  GB_CUDA(cudaMemsetAsync(dbad, 0, sizeof(int), s));
  mg_validate<<<g->sm_count * 4, 256, 0, s>>>(g->offs, g->col, g->n, g->mg_first, ng, dbad);
  int hbad = 0;
  GB_CUDA(cudaMemcpyAsync(&hbad, dbad, sizeof(int), cudaMemcpyDeviceToHost, s));
  GB_CUDA(cudaStreamSynchronize(s));
  if (hbad) GB_FAIL(GB_ERR_FORMAT, "multi-graph: an arc leaves its graph's vertex range");
  g->mg_ngraphs = ng;
  g->mg_hash = h;
  return GB_OK;
}

}  // namespace
}  // namespace gb

extern "C" int gb_multi_graph_bfs_cc(gb_graph* g, const uint32_t* graph_first, uint32_t ngraphs,
                                     const uint32_t* local_src, uint32_t* level_out, uint32_t* label_out,
                                     gb_stats* stats, void* stream) {
  using namespace gb;
  clear_error();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!g || !graph_first || !local_src || (!level_out && !label_out))
    GB_FAIL(GB_ERR_ARG, "gb_multi_graph_bfs_cc: null argument");
  if (ngraphs == 0 || ngraphs > g->n) GB_FAIL(GB_ERR_ARG, "gb_multi_graph_bfs_cc: bad graph count %u", ngraphs);
  if (!g->symmetric) GB_FAIL(GB_ERR_UNSUPPORTED, "gb_multi_graph_bfs_cc: needs symmetric graphs");
  if (g->perm) GB_FAIL(GB_ERR_UNSUPPORTED, "gb_multi_graph_bfs_cc: the block-diagonal layout needs file order (graph was relabelled)");
  if (is_device_ptr(graph_first) || is_device_ptr(local_src))
    GB_FAIL(GB_ERR_ARG, "gb_multi_graph_bfs_cc: graph_first and local_src are host arrays");
  GB_CUDA(cudaSetDevice(g->device));
  int st = prepare_layout(g, graph_first, ngraphs, s);
  if (st != GB_OK) return st;
  for (uint32_t k = 0; k < ngraphs; ++k)
    if (local_src[k] >= graph_first[k + 1] - graph_first[k])
      GB_FAIL(GB_ERR_ARG, "gb_multi_graph_bfs_cc: local source %u of graph %u out of range", local_src[k], k);
  for (uint32_t k = 0; k < ngraphs; ++k) g->mg_stage[k] = graph_first[k] + local_src[k];
  KernelTimer kt(stats != nullptr, s);
  GB_CUDA(cudaMemcpyAsync(g->mg_src, g->mg_stage, sizeof(uint32_t) * ngraphs, cudaMemcpyHostToDevice, s));
  const bool lev_dev = level_out && is_device_ptr(level_out);
  const bool lab_dev = label_out && is_device_ptr(label_out);
  uint32_t* d_level = lev_dev ? level_out : g->mg_level;
  uint32_t* d_label = lab_dev ? label_out : g->mg_label;
  if (level_out) {
    st = run_bfs_sources(g, g->mg_src, ngraphs, d_level, s);
    if (st != GB_OK) return st;
  }
  if (label_out && level_out) {
    st = cc_from_levels(g, d_level, ngraphs, d_label, s);
    if (st != GB_OK) return st;
  } else if (label_out) {
    st = run_cc(g, GB_CC_UNIONFIND, d_label, nullptr, s);
    if (st != GB_OK) return st;
    mg_localize<<<g->sm_count * 4, 256, 0, s>>>(d_label, g->n, g->mg_first, ngraphs);
    GB_CUDA(cudaGetLastError());
  }
  kt.stop(s);
  if (level_out && !lev_dev) GB_CUDA(cudaMemcpyAsync(level_out, d_level, sizeof(uint32_t) * g->n, cudaMemcpyDefault, s));
  if (label_out && !lab_dev) GB_CUDA(cudaMemcpyAsync(label_out, d_label, sizeof(uint32_t) * g->n, cudaMemcpyDefault, s));
  if (stats || (level_out && !lev_dev) || (label_out && !lab_dev)) {
    GB_CUDA(cudaStreamSynchronize(s));
    const int err = static_cast<int*>(g->pinned)[8];
    if (level_out && err) return dev_err_status(err, "gb_multi_graph_bfs_cc");
    if (stats) {
      *stats = gb_stats{};
      stats->vertices_reached = g->n;
      stats->edges_reached = g->m;
      stats->launches = (level_out ? 3 : 0) + (label_out ? 3 : 0);
      stats->kernel_ms = kt.ms();
    }
  }
  return GB_OK;
}
