"""Many disjoint graphs in one launch (gb_multi_graph_bfs_cc) against per-graph
CPU oracles, bit-exact; plus CUDA-graph capture and replay of the call."""
import numpy as np
import pytest

import oracle
from galois_b200 import DeviceGraph, GbError, HostCSR, erdos_renyi
from galois_b200 import _lib
from galois_b200.graph import pack_graphs

pytestmark = pytest.mark.gpu


def make_graphs(k, seed=0, lo=50, hi=3000):
    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(np.log(lo), np.log(hi), k)).astype(int)
    return [erdos_renyi(int(n), 8.0 if i % 3 else 1.5, seed=seed * 1000 + i) for i, n in enumerate(sizes)]


def expected(graphs, local_src):
    levels, labels = [], []
    for g, s in zip(graphs, local_src):
        levels.append(oracle.bfs_serial(g, int(s)))
        labels.append(oracle.cc_union_find(g))
    return np.concatenate(levels), np.concatenate(labels)


def test_multigraph_matches_per_graph_oracle(cuda_device):
    graphs = make_graphs(64, seed=3)
    packed, first = pack_graphs(graphs)
    rng = np.random.default_rng(5)
    local = np.array([rng.integers(0, g.n) for g in graphs], np.uint32)
    want_lv, want_lb = expected(graphs, local)
    with DeviceGraph(packed, symmetric=True) as dg:
        lv, lb = dg.multi_graph_bfs_cc(first, local)
        assert np.array_equal(lv, want_lv)
        assert np.array_equal(lb, want_lb)
        # a second layout on the same handle (validation cache refresh)
        local2 = np.zeros(len(graphs), np.uint32)
        lv2, _ = dg.multi_graph_bfs_cc(first, local2)
        assert np.array_equal(lv2, expected(graphs, local2)[0])


@pytest.mark.parametrize("sizes", [[1], [1, 1, 1], [31, 33, 1, 64], [5] * 100, [2000, 1, 3]])
def test_multigraph_labels_from_levels(cuda_device, sizes):
    """Labels taken from the BFS levels: graphs smaller than a warp's chunk, a
    source in the giant component, in a small one (the giant is unreached) and
    without arcs."""
    graphs = [erdos_renyi(n, 3.0, seed=i) if n > 1 else HostCSR(np.zeros(1), np.zeros(0)) for i, n in enumerate(sizes)]
    packed, first = pack_graphs(graphs)
    for pick in (np.argmax, np.argmin, lambda d: len(d) // 2):
        local = np.array([int(pick(g.degrees())) for g in graphs], np.uint32)
        want_lv, want_lb = expected(graphs, local)
        with DeviceGraph(packed, symmetric=True) as dg:
            lv, lb = dg.multi_graph_bfs_cc(first, local)
            assert np.array_equal(lv, want_lv) and np.array_equal(lb, want_lb)


@pytest.mark.parametrize("hub_at", [2, 700, 40000])
@pytest.mark.parametrize("heavy,tile", [(0, 0), (16, 32)])
def test_multigraph_unreached_hubs(cuda_device, hub_at, heavy, tile):
    """Sources in small components beside unreached ones with hubs of many
    tiles (most neighbours' ids above the hub's, some, or none), rows of
    exactly the heavy degree, a graph whose hub is reached, and a captured
    call."""
    import torch

    n = 40001
    arcs = [(0, 1)] + [(hub_at, v) for v in range(2, n) if v != hub_at and v % 7]
    arcs += [(v, v + 7) for v in range(7, n - 700, 7)][:5000]
    arcs += [(3, v) for v in range(8, 8 + 7 * 16, 7) if v != hub_at]  # a row of 17 or so
    src, dst = np.array(arcs + [(b, a) for a, b in arcs]).T
    order = np.lexsort((dst, src))
    hub = HostCSR.from_edges(n, src[order], dst[order])
    reached = HostCSR.from_edges(900, [0] * 899 + list(range(1, 900)), list(range(1, 900)) + [0] * 899)
    graphs = [hub, reached, erdos_renyi(50, 2.0, seed=1), hub]
    packed, first = pack_graphs(graphs)
    local = np.array([0, 5, 0, 1], np.uint32)
    want_lv, want_lb = expected(graphs, local)
    with DeviceGraph(packed, symmetric=True) as dg:
        if heavy:
            dg.set_tuning(heavy_degree=heavy, tile_edges=tile)
        lv, lb = dg.multi_graph_bfs_cc(first, local)
        assert np.array_equal(lv, want_lv) and np.array_equal(lb, want_lb)
        d_lv = torch.zeros(packed.n, dtype=torch.int32, device="cuda")
        d_lb = torch.zeros(packed.n, dtype=torch.int32, device="cuda")
        dg.multi_graph_bfs_cc(first, local, level_out=d_lv, label_out=d_lb)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            dg.multi_graph_bfs_cc(first, local, level_out=d_lv, label_out=d_lb)
        d_lv.fill_(-1), d_lb.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(d_lv.cpu().numpy().view(np.uint32), want_lv)
        assert np.array_equal(d_lb.cpu().numpy().view(np.uint32), want_lb)


def test_multigraph_rejects_crossing_arcs_and_bad_sources(cuda_device):
    graphs = make_graphs(4, seed=1)
    packed, first = pack_graphs(graphs)
    bad_first = first.copy()
    bad_first[1] += 1  # vertex ranges no longer match the packing
    with DeviceGraph(packed, symmetric=True) as dg:
        with pytest.raises(GbError) as e:
            dg.multi_graph_bfs_cc(bad_first, np.zeros(4, np.uint32))
        assert e.value.status == _lib.GB_ERR_FORMAT
        with pytest.raises(GbError):
            dg.multi_graph_bfs_cc(first, np.array([0, 0, 0, graphs[3].n], np.uint32))


def test_multigraph_cuda_graph_replay(cuda_device):
    import torch

    graphs = make_graphs(32, seed=7)
    packed, first = pack_graphs(graphs)
    local = np.zeros(len(graphs), np.uint32)
    want_lv, want_lb = expected(graphs, local)
    with DeviceGraph(packed, symmetric=True) as dg:
        lv = torch.empty(packed.n, dtype=torch.int32, device="cuda")
        lb = torch.empty(packed.n, dtype=torch.int32, device="cuda")
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            dg.multi_graph_bfs_cc(first, local, lv, lb)  # warm-up: layout, workspace, schedule
            torch.cuda.synchronize()
            cg = torch.cuda.CUDAGraph()
            with torch.cuda.graph(cg, stream=s):
                dg.multi_graph_bfs_cc(first, local, lv, lb)
        lv.fill_(-1)
        lb.fill_(-1)
        for _ in range(3):
            cg.replay()
        torch.cuda.synchronize()
        assert np.array_equal(lv.cpu().numpy().view(np.uint32), want_lv)
        assert np.array_equal(lb.cpu().numpy().view(np.uint32), want_lb)
        del cg
