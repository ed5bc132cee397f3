"""GPU parity: BFS, SSSP, CC and PageRank kernels (through the C ABI) against
the CPU oracle on the same seeded inputs.  Integer results are bit-exact;
PageRank tolerances are stated per test."""
import numpy as np
import pytest

import oracle
from galois_b200 import (GB_CC_AFFOREST, GB_CC_LABELPROP, GB_CC_UNIONFIND, DeviceGraph, GbError, HostCSR,
                         assign_weights_u32, erdos_renyi, grid2d, rmat)
from galois_b200 import _lib

pytestmark = pytest.mark.gpu
INF = oracle.INF


def path_graph(n):
    s = list(range(n - 1)) + list(range(1, n))
    d = list(range(1, n)) + list(range(n - 1))
    return HostCSR.from_edges(n, s, d)


def star_graph(k):
    return HostCSR.from_edges(k + 1, [0] * k + list(range(1, k + 1)), list(range(1, k + 1)) + [0] * k)


def grid8(rows, cols):
    """rows x cols grid with the 8 king-move neighbours (degree <= 8)."""
    s, d = [], []
    for r in range(rows):
        for c in range(cols):
            for dr in (-1, 0, 1):
                for dc in (-1, 0, 1):
                    if (dr or dc) and 0 <= r + dr < rows and 0 <= c + dc < cols:
                        s.append(r * cols + c)
                        d.append((r + dr) * cols + c + dc)
    return HostCSR.from_edges(rows * cols, s, d)


def union(*gs):
    """Block-diagonal union of host graphs."""
    off = 0
    ends, cols = [], []
    base = 0
    for g in gs:
        ends.append(g.end_offs.astype(np.uint64) + np.uint64(base))
        cols.append(g.col.astype(np.uint32) + np.uint32(off))
        off += g.n
        base += g.m
    return HostCSR(np.concatenate(ends), np.concatenate(cols))


# ---- BFS ----------------------------------------------------------------------

@pytest.mark.parametrize("scale,ef", [(10, 4), (14, 16)])
def test_bfs_rmat_sym_bit_exact(cuda_device, scale, ef):
    g, _ = rmat(scale, ef, seed=scale)
    deg = g.degrees()
    with DeviceGraph(g, symmetric=True) as dg:
        for src in (int(np.argmax(deg)), int(np.flatnonzero(deg == 1)[0]) if (deg == 1).any() else 1,
                    int(np.flatnonzero(deg == 0)[0]) if (deg == 0).any() else 2):
            got, st = dg.bfs(src, stats=True)
            want = oracle.bfs_serial(g, src)
            assert (got == want).all(), f"src {src}"
            assert st["vertices_reached"] == int((want != INF).sum())


def test_bfs_push_only_and_pull_heavy(cuda_device):
    g, _ = rmat(13, 16, seed=21)
    src = int(np.argmax(g.degrees()))
    want = oracle.bfs_serial(g, src)
    with DeviceGraph(g, symmetric=True) as dg:
        dg.set_tuning(direction_opt=2)
        got, st = dg.bfs(src, stats=True)
        assert (got == want).all() and st["pull_rounds"] == 0
        dg.set_tuning(direction_opt=0, do_alpha=1e6, do_beta=1e-6, heavy_degree=32, tile_edges=64)
        got, st = dg.bfs(src, stats=True)
        assert (got == want).all() and st["pull_rounds"] > 0


def test_bfs_directed_push_and_transpose_pull(cuda_device):
    g, perm = rmat(12, 8, seed=3, symmetrize=False)
    src = int(perm[0])
    want = oracle.bfs_serial(g, src)
    with DeviceGraph(g, symmetric=False) as dg:
        assert (dg.bfs(src) == want).all()
        dg.build_transpose()
        dg.set_tuning(do_alpha=1e6, do_beta=1e-6)
        got, st = dg.bfs(src, stats=True)
        assert (got == want).all()


def test_bfs_small_shapes(cuda_device):
    for g, src in ((path_graph(300), 0), (path_graph(300), 150), (star_graph(5000), 0), (star_graph(5000), 17),
                   (HostCSR(np.zeros(1, np.uint64), np.zeros(0, np.uint32)), 0),
                   (grid2d(40, 33), 0)):
        with DeviceGraph(g, symmetric=True) as dg:
            assert (dg.bfs(src) == oracle.bfs_serial(g, src)).all()


def test_bfs_device_output_and_errors(cuda_device):
    import torch

    g, _ = rmat(11, 8, seed=1)
    src = int(np.argmax(g.degrees()))
    with DeviceGraph(g, symmetric=True) as dg:
        out = torch.empty(g.n, dtype=torch.int32, device="cuda")
        dg.bfs(src, out=out)
        torch.cuda.synchronize()
        assert (out.cpu().numpy().view(np.uint32) == oracle.bfs_serial(g, src)).all()
        with pytest.raises(GbError) as e:
            dg.bfs(g.n)
        assert e.value.status == _lib.GB_ERR_ARG


# ---- BFS parents (bfsDirectionOpt output) --------------------------------------

@pytest.mark.parametrize("sym,reorder", [(True, 0), (False, 0), (True, 1), (False, 1)])
def test_bfs_parent_bit_exact(cuda_device, sym, reorder):
    g, perm = rmat(13, 16, seed=9, symmetrize=sym)
    src = int(perm[0])
    lv_want = oracle.bfs_serial(g, src)
    want = oracle.bfs_parent_min(g, src, lv_want)
    with DeviceGraph(g, symmetric=sym, reorder=reorder) as dg:
        # small tiles so the hubs' rows take the tile kernel
        dg.set_tuning(heavy_degree=32, tile_edges=64)
        lv = np.empty(g.n, np.uint32)
        got, st = dg.bfs_parent(src, level_out=lv, stats=True)
    assert (lv == lv_want).all()
    assert (got == want).all()
    assert oracle.verify_bfs_parent(g, src, lv_want, got) == 0
    assert st["vertices_reached"] == int((lv_want != INF).sum())


def test_bfs_parent_small_shapes_and_device_output(cuda_device):
    import torch

    for g, src in ((path_graph(300), 150), (star_graph(5000), 17), (star_graph(5000), 0),
                   (HostCSR(np.zeros(1, np.uint64), np.zeros(0, np.uint32)), 0), (grid2d(40, 33), 5)):
        lv = oracle.bfs_serial(g, src)
        with DeviceGraph(g, symmetric=True) as dg:
            out = torch.empty(g.n, dtype=torch.int32, device="cuda")
            dg.bfs_parent(src, out=out)
            torch.cuda.synchronize()
            got = out.cpu().numpy().view(np.uint32)
        assert (got == oracle.bfs_parent_min(g, src, lv)).all()
        assert got[src] == 0
    with DeviceGraph(path_graph(10), symmetric=True) as dg:
        with pytest.raises(GbError) as e:
            dg.bfs_parent(10)
        assert e.value.status == _lib.GB_ERR_ARG


@pytest.mark.parametrize("alpha", [1e-3, 2.0, 15.0, 1e6])
@pytest.mark.parametrize("heavy,tile", [(16, 32), (0, 0)])
def test_bfs_queue_edges(cuda_device, alpha, heavy, tile):
    """Levels whose vertices have rows of 0 to `heavy` + 1 arcs and of 8, 9 and
    many tiles side by side (a lane writes up to 8 tiles of its own, the warp
    the longer runs), with direction switch points at which every warp queues
    its part of the next level, some do, or none does."""
    rng = np.random.default_rng(7)
    n, hubs = 30000, 300
    deg = rng.integers(0, 40, hubs)
    deg[:12] = [0, 1, 15, 16, 17, 32, 33, 8 * 32, 8 * 32 + 1, 9 * 32, 40 * 32, 9000]
    rng.shuffle(deg)
    src = np.repeat(np.arange(1, hubs + 1), deg)
    dst = rng.integers(hubs + 1, n, len(src))
    more = rng.integers(hubs + 1, n, (2, n))  # the levels after them
    a = np.concatenate([np.zeros(hubs, np.int64), src, more[0]])
    b = np.concatenate([np.arange(1, hubs + 1), dst, more[1]])
    g = HostCSR.from_edges(n, np.concatenate([a, b]), np.concatenate([b, a]))
    for order in (0, 1):
        with DeviceGraph(g, symmetric=True, reorder=order) as dg:
            dg.set_tuning(do_alpha=alpha, heavy_degree=heavy, tile_edges=tile)
            for s in (0, 5, n - 1):
                want = oracle.bfs_serial(g, s)
                for _ in range(2):
                    assert (dg.bfs(s) == want).all(), (order, s)


# ---- SSSP ---------------------------------------------------------------------

@pytest.mark.parametrize("shift", [0, 5, 13, 31])
def test_sssp_rmat_directed_bit_exact(cuda_device, shift):
    g, perm = rmat(13, 16, seed=8, symmetrize=False)
    assign_weights_u32(g, 1, 255, seed=8)
    src = int(perm[0])
    with DeviceGraph(g) as dg:
        got, st = dg.sssp(src, shift, stats=True)
    want = oracle.sssp_dijkstra(g, src)
    assert (got == want).all()
    assert st["vertices_reached"] == int((want != INF).sum())


@pytest.mark.parametrize("local_depth,block", [(-1, 256), (8, 256), (64, 1024)])
def test_sssp_grid_many_buckets(cuda_device, local_depth, block):
    """The phase-synchronous kernel (sssp_async = -1: the default would take
    regions for the widest buckets) without local queues, with queues and
    with large blocks."""
    g = grid2d(96, 80)
    assign_weights_u32(g, 1, 255, seed=3)
    want = oracle.sssp_dijkstra(g, 0)
    with DeviceGraph(g, symmetric=True) as dg:
        dg.set_tuning(local_depth=local_depth, block_threads=block, sssp_async=-1)
        for shift in (13, 8, 3):
            got, st = dg.sssp(0, shift, stats=True)
            assert (got == want).all() and st["pull_rounds"] == 0
            if shift <= 8:
                assert st["buckets"] > 10


@pytest.mark.parametrize("shift", [13, 6, 0])
def test_sssp_async_buckets_bit_exact(cuda_device, shift):
    """Asynchronous buckets (bounded-degree graphs with local queues) against
    Dijkstra and against the phase-synchronous kernel, on a grid, a sparse
    Erdos-Renyi graph with isolated vertices, a path and a disjoint union
    (unreachable part), from several sources."""
    er = erdos_renyi(30000, 3.0, seed=9)
    cases = [(grid2d(120, 70), (0, 4321)), (er, (0, 12345)), (path_graph(2000), (0, 999)),
             (union(grid2d(30, 30), path_graph(100)), (5, 950)), (grid8(90, 60), (0, 2999))]
    for g, srcs in cases:
        assign_weights_u32(g, 1, 255, seed=int(g.n))
        assert g.degrees().max() <= 32
        with DeviceGraph(g, symmetric=True) as dg:
            for src in srcs:
                want = oracle.sssp_dijkstra(g, src)
                # 1: asynchronous buckets; 2: the same over fixed-width rows
                # (degree <= 4 or <= 8; the Erdos-Renyi graph's degree is above 8, so it
                # takes the plain asynchronous kernel); 3: regions in shared memory
                # (the Erdos-Renyi graph's regions hold too many arcs: asynchronous kernel)
                for mode in (1, 2, 3):
                    dg.set_tuning(local_depth=8, sssp_async=mode)
                    got, st = dg.sssp(src, shift, stats=True)
                    assert (got == want).all(), f"async {mode} n={g.n} src={src}"
                    assert st["vertices_reached"] == int((want != INF).sum())
                dg.set_tuning(sssp_async=-1)
                got, st = dg.sssp(src, shift, stats=True)
                assert (got == want).all() and st["pull_rounds"] == 0, f"phase-synchronous n={g.n} src={src}"


def test_sssp_async_small_ring_and_blocks(cuda_device):
    """One CTA per SM (few warps share the ring) and a graph whose source has
    no arcs (nothing is published)."""
    g = grid2d(200, 150)
    assign_weights_u32(g, 1, 255, seed=77)
    want = oracle.sssp_dijkstra(g, 777)
    with DeviceGraph(g, symmetric=True) as dg:
        for mode in (1, 2):
            dg.set_tuning(local_depth=4, blocks_per_sm=1, sssp_async=mode)
            assert (dg.sssp(777, 13) == want).all()
        # the rows carry the weights: new weights rebuild them
        dg.assign_weights_u32(1, 255, 78)
        g.w_u32 = None
        assign_weights_u32(g, 1, 255, seed=78)
        assert (dg.sssp(777, 13) == oracle.sssp_dijkstra(g, 777)).all()
    iso = union(path_graph(1), grid2d(10, 10))
    iso.w_u32 = np.ones(iso.m, np.uint32)
    with DeviceGraph(iso, symmetric=True) as dg:
        for mode in (1, 2):
            dg.set_tuning(sssp_async=mode)
            got = dg.sssp(0, 13)
            assert got[0] == 0 and (got[1:] == INF).all()


@pytest.mark.parametrize("shift", [13, 8, 0])
def test_sssp_regions_bit_exact(cuda_device, shift):
    """Regions of 2048 consecutive ids relaxed in shared memory (tuning
    sssp_async = 3) against Dijkstra: grids of many regions in file order and
    in locality order (compact regions), a ragged last region, an
    unreachable part, and a grid whose regions hold too many arcs (8
    neighbours: the other kernels run)."""
    from galois_b200._lib import GB_ORDER_LOCALITY
    cases = [(grid2d(300, 290), (0, 45000, 86999)), (union(grid2d(150, 100), path_graph(5000)), (7, 16000)),
             (grid2d(64, 64), (0,)), (grid8(120, 90), (0, 5000))]
    for g, srcs in cases:
        assign_weights_u32(g, 1, 255, seed=int(g.n) + shift)
        for order in (0, GB_ORDER_LOCALITY):
            with DeviceGraph(g, symmetric=True) as dg:
                if order:
                    dg.reorder(order)
                dg.set_tuning(sssp_async=3)
                for src in srcs:
                    want = oracle.sssp_dijkstra(g, src)
                    got, st = dg.sssp(src, shift, stats=True)
                    assert (got == want).all(), f"regions n={g.n} order={order} src={src}"
                    assert st["vertices_reached"] == int((want != INF).sum())
                    # a second call reuses the cached region check and the workspace
                    assert (dg.sssp(src, shift) == want).all()


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
def test_sssp_regions_output_at_any_word(cuda_device, offset):
    """A device output that starts 4, 8, 12 or 16 bytes into an allocation:
    the region kernel (the default on a grid in file order, and asked for)
    loads distances 16 bytes at a time.  Graphs of degree 4 and 5 (rows of
    slots, offsets), several regions and a ragged last one; the words around
    the output stay as they were."""
    import torch

    grid = grid2d(70, 61)
    a = np.repeat(np.arange(grid.n), grid.degrees())
    v = np.arange(0, grid.n - 62, 500)
    more = HostCSR.from_edges(grid.n, np.concatenate([a, v, v + 62]), np.concatenate([grid.col, v + 62, v]))
    assert more.degrees().max() > 4 and grid.degrees().max() == 4
    for g in (grid, more):
        assign_weights_u32(g, 1, 255, seed=5)
        with DeviceGraph(g, symmetric=True) as dg:
            for mode in (0, 3):
                dg.set_tuning(sssp_async=mode)
                for src in (0, g.n - 1):
                    want = oracle.sssp_dijkstra(g, src)
                    buf = torch.full((g.n + offset + 4,), -7, dtype=torch.int32, device="cuda")
                    out = buf[offset:offset + g.n]
                    dg.sssp(src, 13, out=out)
                    assert (out.cpu().numpy().view(np.uint32) == want).all()
                    out.fill_(-7)
                    _, st = dg.sssp(src, 13, out=out, stats=True)
                    assert st["pull_rounds"] > 0  # the region kernel
                    assert (out.cpu().numpy().view(np.uint32) == want).all()
                    assert (buf[:offset] == -7).all() and (buf[offset + g.n:] == -7).all()


def test_sssp_local_queues_rmat(cuda_device):
    g, perm = rmat(14, 16, seed=12, symmetrize=False)
    assign_weights_u32(g, 1, 255, seed=12)
    src = int(perm[0])
    want = oracle.sssp_dijkstra(g, src)
    with DeviceGraph(g) as dg:
        for depth in (1, 32, 256):
            dg.set_tuning(local_depth=depth)
            assert (dg.sssp(src, 13) == want).all()


def test_sssp_heavy_tiles_and_unreachable(cuda_device):
    g = union(star_graph(3000), path_graph(50))
    g.w_u32 = (np.arange(g.m) % 255 + 1).astype(np.uint32)
    with DeviceGraph(g, symmetric=True) as dg:
        dg.set_tuning(heavy_degree=64, tile_edges=128)
        for src in (0, 5, 3010):
            assert (dg.sssp(src, 4) == oracle.sssp_dijkstra(g, src)).all()


def test_sssp_needs_weights(cuda_device):
    g, _ = rmat(8, 4, seed=1)
    with DeviceGraph(g) as dg:
        with pytest.raises(GbError) as e:
            dg.sssp(0)
        assert e.value.status == _lib.GB_ERR_ARG


# ---- CC -----------------------------------------------------------------------

@pytest.mark.parametrize("algo", [GB_CC_LABELPROP, GB_CC_UNIONFIND, GB_CC_AFFOREST])
def test_cc_min_labels(cuda_device, algo):
    for g in (rmat(14, 8, seed=31)[0], erdos_renyi(20000, 1.1, seed=2), union(path_graph(500), star_graph(2000)),
              grid2d(50, 70)):
        want = oracle.cc_union_find(g)
        with DeviceGraph(g, symmetric=True) as dg:
            got, st = dg.cc(algo, stats=True)
        assert (got == want).all()


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("arcs_per_row", [0.5, 1.24, 1.25, 1.26, 2.0])
def test_cc_sparse_first_round(cuda_device, arcs_per_row, order):
    """Symmetric graphs on both sides of 1.25 arcs per row, from which on the
    first round takes two arcs a row: a hub of many tiles, small components
    and isolated vertices."""
    n, hub = 40000, 9000
    rng = np.random.default_rng(3)
    edges = int(n * arcs_per_row / 2)
    a = np.concatenate([np.full(hub, 77), rng.integers(n // 3, n, edges - hub)])
    b = np.concatenate([rng.permutation(n // 3)[:hub], rng.integers(n // 3, n, edges - hub)])
    g = HostCSR.from_edges(n, np.concatenate([a, b]), np.concatenate([b, a]))
    assert abs(g.m - arcs_per_row * n) <= 2
    want = oracle.cc_union_find(g)
    with DeviceGraph(g, symmetric=True, reorder=order) as dg:
        for _ in range(3):
            assert (dg.cc(GB_CC_LABELPROP) == want).all()


def test_cc_directed_is_weak(cuda_device):
    g, _ = rmat(12, 4, seed=5, symmetrize=False)
    sym = HostCSR.from_edges(g.n, np.concatenate([np.repeat(np.arange(g.n), g.degrees()), g.col]),
                             np.concatenate([g.col, np.repeat(np.arange(g.n), g.degrees())]))
    want = oracle.cc_union_find(sym)
    with DeviceGraph(g, symmetric=False) as dg:
        for algo in (GB_CC_LABELPROP, GB_CC_UNIONFIND):
            assert (dg.cc(algo) == want).all()
        with pytest.raises(GbError):
            dg.cc(GB_CC_AFFOREST)


# ---- PageRank -------------------------------------------------------------------

def test_pagerank_pull_vs_fp64(cuda_device):
    g, _ = rmat(14, 16, seed=41)
    want, it64 = oracle.pr_pull_topo_f64(g, 0.85, 1e-6, 1000)
    with DeviceGraph(g, symmetric=True) as dg:
        got, st = dg.pagerank_pull(0.85, 1e-6, 1000, stats=True)
    # tolerance: 1e-5 L-inf (absolute), and 1e-4 relative on every vertex
    assert np.abs(got - want).max() < 1e-5
    assert (np.abs(got - want) / want).max() < 1e-4
    assert abs(st["iterations"] - it64) <= 2


def test_pagerank_pull_heavy_tiles(cuda_device):
    g = union(star_graph(20000), path_graph(100))
    want, it64 = oracle.pr_pull_topo_f64(g, 0.85, 1e-7, 1000)
    with DeviceGraph(g, symmetric=True) as dg:
        dg.set_tuning(heavy_degree=64, tile_edges=256)
        got, st = dg.pagerank_pull(0.85, 1e-7, 1000, stats=True)
    assert (np.abs(got - want) / want).max() < 1e-4


def test_pagerank_pull_not_converged_status(cuda_device):
    g, _ = rmat(10, 8, seed=2)
    with DeviceGraph(g, symmetric=True) as dg:
        got, st = dg.pagerank_pull(0.85, 0.0, 5, stats=True)
        assert st["iterations"] == 5 and not st["converged"]
        with pytest.raises(GbError) as e:
            dg.pagerank_pull(0.85, 0.0, 5, allow_not_converged=False)
        assert e.value.status == _lib.GB_ERR_NOT_CONVERGED


def _rel(got, want):
    """Largest |got - want| / max(|want|, 1): absolute below 1, relative
    above (the residual variants' values are unnormalised, ~1 on average and
    up to ~100 on the hubs, where fp32 accumulation dominates)."""
    return float((np.abs(got.astype(np.float64) - want) / np.maximum(np.abs(want), 1.0)).max())


def check_residual_parity(got, want, tol, what):
    """Residual PageRank against the FP64 restatement of the same rounds at
    the same tolerance.  Every vertex within 1e-5 relative (absolute below
    1), except where a residual lying within fp32 rounding of tol was taken
    on one side and not on the other (a threshold flip, possible because the
    GPU sums in another order): the value there differs by that residual,
    at most tol, and its out-neighbours' by alpha / nout of it (push Sync also
    activates them one round apart).  Such vertices must be rare (at most 1 %
    of them; measured 0.19 % for push Sync on RMAT-14 at tol 1e-4) and stay
    within 1e-5 relative + 2 tol."""
    err = np.abs(got.astype(np.float64) - want)
    scale = np.maximum(np.abs(want), 1.0)
    flipped = int((err > 1e-5 * scale).sum())
    assert flipped <= max(10, 1e-2 * want.size), f"{what}: {flipped} vertices beyond 1e-5 relative"
    assert float((err - 1e-5 * scale).max()) <= 2 * tol, f"{what}: max error {float(err.max()):.3e}"


RESIDUAL = [("pull-residual", "pagerank_pull_residual", oracle.pr_pull_residual),
            ("push-sync", "pagerank_push", oracle.pr_push_sync)]


@pytest.mark.parametrize("reorder", [0, 1])
@pytest.mark.parametrize("name,method,restated", RESIDUAL)
@pytest.mark.parametrize("scale,ef,seed,tol", [(12, 8, 19, 1e-3), (12, 8, 17, 1e-4), (14, 16, 41, 1e-4)])
def test_pagerank_residual_vs_restatement(cuda_device, name, method, restated, scale, ef, seed, tol, reorder):
    """The residual variants against the oracle's FP64 restatement of the same
    rounds (PageRank-pull.cpp:132-190, PageRank-push.cpp:103-188) at the same
    tolerance, as check_residual_parity states, and the same number of
    rounds within 2; both vertex orders."""
    g, _ = rmat(scale, ef, seed=seed)
    want, it64 = restated(g, 0.85, tol, 1000, f64=True)
    # reorder 1: the degree-ordered graph (the flat light-row sweep for pull-residual)
    with DeviceGraph(g, symmetric=True, reorder=reorder) as dg:
        got, st = getattr(dg, method)(0.85, tol, 1000, stats=True)
    check_residual_parity(got, want, tol, name)
    assert abs(st["iterations"] - it64) <= 2, f"{name}: {st['iterations']} rounds vs {it64}"


def _star_with_path(k, plen):
    """A star of k leaves (one hub with k arcs each way) plus a detached path."""
    s = [0] * k + list(range(1, k + 1)) + list(range(k + 1, k + plen)) + list(range(k + 2, k + plen + 1))
    d = list(range(1, k + 1)) + [0] * k + list(range(k + 2, k + plen + 1)) + list(range(k + 1, k + plen))
    return HostCSR.from_edges(k + plen + 1, s, d)


@pytest.mark.parametrize("case", ["hub-split", "directed", "single-partition", "many-partitions"])
def test_pagerank_binned_layout(cuda_device, case):
    """Degree-ordered graphs run PageRank pull and pull-residual over the
    binned layout (blocks of 32 768 sources, runs of arcs into one
    destination, 256-arc chunks).  Shapes that exercise it: a hub whose run
    spans whole chunks of several tasks and whose own block is split over
    tasks, a directed graph with rows that have no arcs but sources that do, a
    graph smaller than one block, and one of several blocks.  Pull against the FP64 Jacobi oracle (<= 1e-5,
    iterations within 2) and against the file-order row sweep (<= 1e-6);
    pull-residual against the FP64 restatement of its rounds
    (check_residual_parity, rounds within 2)."""
    tol = 1e-6
    if case == "hub-split":
        # fp32 Jacobi on a 150 K-leaf star settles into a rounding limit cycle
        # whose L1 change stays near 2-3e-6 (the row sweep's near 3e-6 to 2e-5):
        # a 1e-6 tolerance is never met there, by either kernel
        g, sym = _star_with_path(150000, 3000), True
        tol = 1e-5
    elif case == "directed":
        g, _ = rmat(14, 8, seed=5, symmetrize=False)
        sym = False
    elif case == "single-partition":
        g, sym = grid2d(100, 120), True
    else:
        g, _ = rmat(17, 8, seed=6)
        sym = True
    want, it64 = oracle.pr_pull_topo_f64(g, 0.85, tol, 1000)
    with DeviceGraph(g, symmetric=sym) as plain:
        ref = plain.pagerank_pull(0.85, tol, 1000)
    with DeviceGraph(g, symmetric=sym, reorder=_lib.GB_ORDER_DEGREE) as dg:
        for _ in range(2):  # the second call reuses the cached layout
            got, st = dg.pagerank_pull(0.85, tol, 1000, stats=True)
            assert np.max(np.abs(got.astype(np.float64) - want)) <= 1e-5, case
            assert abs(st["iterations"] - it64) <= 2, (case, st["iterations"], it64)
            assert np.max(np.abs(got - ref)) <= 1e-5, case
        rwant, rit = oracle.pr_pull_residual(g, 0.85, 1e-4, 1000, f64=True)
        rgot, rst = dg.pagerank_pull_residual(0.85, 1e-4, 1000, stats=True)
        check_residual_parity(rgot, rwant, 1e-4, f"pull-residual {case}")
        assert abs(rst["iterations"] - rit) <= 2, case


@pytest.mark.parametrize("heavy", [2, 4, 128])
def test_pagerank_binned_more_heavy_rows_than_hubs(cuda_device, heavy):
    """The binned layout adds the largest rows up in 64 bits, at most 16 384 of
    them: with low degree thresholds a graph of 40 K vertices has more heavy
    rows than that, with the default fewer.  Against the FP64 oracles as in
    the layout's other test."""
    g = erdos_renyi(40000, 9.0, seed=4)
    assert (g.degrees() > 4).sum() > 16384 > (g.degrees() > 128).sum()
    want, it64 = oracle.pr_pull_topo_f64(g, 0.85, 1e-6, 1000)
    rwant, rit = oracle.pr_pull_residual(g, 0.85, 1e-4, 1000, f64=True)
    with DeviceGraph(g, symmetric=True, reorder=_lib.GB_ORDER_DEGREE) as dg:
        dg.set_tuning(heavy_degree=heavy)
        for _ in range(2):
            got, st = dg.pagerank_pull(0.85, 1e-6, 1000, stats=True)
            assert np.max(np.abs(got.astype(np.float64) - want)) <= 1e-5
            assert np.allclose(got, want, rtol=1e-4, atol=0)
            assert abs(st["iterations"] - it64) <= 2
        rgot, rst = dg.pagerank_pull_residual(0.85, 1e-4, 1000, stats=True)
        check_residual_parity(rgot, rwant, 1e-4, f"pull-residual heavy={heavy}")
        assert abs(rst["iterations"] - rit) <= 2


@pytest.mark.parametrize("n", [4097, 20000])
@pytest.mark.parametrize("shift,tile,order", [(13, 0, 0), (13, 96, 1), (13, 512, 0), (7, 0, 1), (5, 256, 0)])
def test_sssp_bitmap_phases(cuda_device, n, shift, tile, order):
    """Bitmap phases over rows of 0, 1 and up to a warp's steps and tiles'
    edges (128/129 arcs: light/heavy; 255-257, 512/513: tiles), hubs of many
    tiles, words with one and with all 32 vertices active; with small deltas
    also the far pile.  Exact against Dijkstra, twice."""
    rng = np.random.default_rng(n + shift)
    deg = np.where(rng.random(n) < 0.6, rng.integers(0, 8, n), rng.integers(0, 140, n))
    deg[64:128] = 0
    deg[:16] = np.minimum([0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 3000, 4000], n - 1)
    src = np.repeat(rng.permutation(n), deg)
    g = HostCSR.from_edges(n, src, rng.integers(0, n, len(src)))
    assign_weights_u32(g, 1, 255, seed=3)
    with DeviceGraph(g, symmetric=False, reorder=order) as dg:
        if tile:
            dg.set_tuning(tile_edges=tile)
        for s in (int(np.argmax(g.degrees())), int(np.flatnonzero(g.degrees())[-1])):
            want = oracle.sssp_dijkstra(g, s)
            for _ in range(2):
                assert (dg.sssp(s, shift) == want).all()


@pytest.mark.parametrize("n", [31, 49152, 49153, 70001])
@pytest.mark.parametrize("order", [0, 1])
def test_pagerank_row_sweep_edges(cuda_device, n, order):
    """Row sweeps of graphs at and above the size from which file order renames
    the columns (arcs leaning on a few vertices), the same in degree order;
    rows of 0 to 9, 127-129 and 255-257 arcs and hubs of many tiles."""
    rng = np.random.default_rng(n)
    perm = rng.permutation(n)
    deg = np.minimum(rng.zipf(1.6, n), 300)
    deg[:16] = np.minimum([0, 1, 8, 9, 127, 128, 129, 255, 256, 257, 8192, 8193, 8449, 20000, 31, 33], n - 1)
    src = np.repeat(perm, deg)
    dst = perm[np.minimum((n * rng.random(len(src)) ** 8).astype(np.int64), n - 1)]
    g = HostCSR.from_edges(n, src, dst)
    want, it64 = oracle.pr_pull_topo_f64(g, 0.85, 1e-6, 1000)
    rwant, rit = oracle.pr_pull_residual(g, 0.85, 1e-4, 1000, f64=True)
    with DeviceGraph(g, symmetric=False, reorder=order) as dg:
        for _ in range(2):
            got, st = dg.pagerank_pull(0.85, 1e-6, 1000, stats=True)
            assert np.max(np.abs(got.astype(np.float64) - want)) <= 1e-5  # the bound of the other pull tests
            assert abs(st["iterations"] - it64) <= 2
        rgot, rst = dg.pagerank_pull_residual(0.85, 1e-4, 1000, stats=True)
        check_residual_parity(rgot, rwant, 1e-4, f"pull-residual n={n} order={order}")
        assert abs(rst["iterations"] - rit) <= 2


@pytest.mark.parametrize("k,n_giant", [(3, 40), (1000, 500), (30000, 20000)])
def test_cc_giant_goes_under_smaller_roots(cuda_device, k, n_giant):
    """k triangles whose least ids are below the giant component's hang on it
    by their third arcs, which the first round does not read: in the second
    round every triangle hooks the giant's root at once (joins that go on
    through several labels), so its label falls while the rows are walked.
    Ids: k triangles' first and second vertices, the head of the giant, the
    triangles' third vertices, the rest of the giant; rows are sorted, so a
    row's first two arcs stay inside its triangle or the giant's head."""
    head = 2 * k
    third = head + n_giant
    rest = third + k
    n = rest + max(n_giant, k)
    i = np.arange(k)
    h = np.arange(head, third)
    g = np.arange(rest, n)
    rng = np.random.default_rng(k)
    hang = rng.permutation(g)[:k]  # the giant's end of each triangle's arc
    a = np.concatenate([i, i, k + i, h[:-1], g, g, third + i])
    b = np.concatenate([k + i, third + i, third + i, h[1:], head + (g - rest) % n_giant,
                        head + (g - rest + 1) % n_giant, hang])
    src, dst = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((dst, src))
    csr = HostCSR.from_edges(n, src[order], dst[order])
    for algo in (GB_CC_LABELPROP, GB_CC_AFFOREST):
        with DeviceGraph(csr, symmetric=True) as dg:
            for _ in range(5):
                assert (dg.cc(algo) == 0).all()


@pytest.mark.parametrize("method,kw", [("pagerank_pull_residual", {}), ("pagerank_push", {}),
                                       ("pagerank_push", {"algo": "async"})])
def test_pagerank_residual_converges_to_fixed_point(cuda_device, method, kw):
    """At tolerance 1e-9 the residual variants -- pull-residual, push Sync and
    push Async (PageRank-push.cpp:68-101, whose schedule no serial
    restatement fixes) -- reach the PageRank fixed point
    x = (1 - alpha) + alpha * sum x[u] / nout[u] (the FP64 Jacobi solution
    scaled by n) within 1e-5 relative per vertex (absolute below 1)."""
    g, _ = rmat(14, 16, seed=41)
    xstar, _ = oracle.pr_pull_topo_f64(g, 0.85, 1e-15, 5000)
    xstar *= g.n
    with DeviceGraph(g, symmetric=True) as dg:
        got = getattr(dg, method)(0.85, 1e-9, 1000, **kw)
    assert _rel(got, xstar) <= 1e-5, (method, kw)


def test_pagerank_push_async_app_tolerance_and_shapes(cuda_device):
    """Async push at the app's default tolerance 1e-3: every vertex ends
    within the leftover-residual bound of the fixed point (below 1e-2
    relative on these graphs; the Sync restatement at the same tolerance is
    as far), on a graph with hubs split into tiles, a directed graph with
    dangling vertices, and a path."""
    g, _ = rmat(13, 16, seed=23)
    xstar, _ = oracle.pr_pull_topo_f64(g, 0.85, 1e-15, 5000)
    xstar *= g.n
    want_sync, _ = oracle.pr_push_sync(g, 0.85, 1e-3, 1000)
    with DeviceGraph(g, symmetric=True) as dg:
        dg.set_tuning(heavy_degree=32, tile_edges=64)
        got, st = dg.pagerank_push(0.85, 1e-3, 1000, stats=True, algo="async")
    assert st["iterations"] == 1
    assert _rel(got, xstar) <= 1e-2 and _rel(want_sync, xstar) <= 1e-2
    # a directed graph: the push goes along out-arcs; its fixed point is the
    # transposed graph's pull solution
    gd, _ = rmat(11, 8, seed=4, symmetrize=False)
    from galois_b200 import transpose

    gt, _ = transpose(gd)
    xd, _ = oracle.pr_pull_topo_f64(gt, 0.85, 1e-15, 5000)
    xd *= gd.n
    with DeviceGraph(gd, symmetric=False) as dg:
        got = dg.pagerank_push(0.85, 1e-9, 1000, algo="async")
    assert _rel(got, xd) <= 1e-5
    with DeviceGraph(path_graph(500), symmetric=True) as dg:
        got = dg.pagerank_push(0.85, 1e-9, 1000, algo="async")
    xp, _ = oracle.pr_pull_topo_f64(path_graph(500), 0.85, 1e-15, 5000)
    assert _rel(got, xp * 500) <= 1e-5
