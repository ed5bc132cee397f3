"""GPU parity for batched personalised PageRank, its adjoint and the autograd
wrapper, against the FP64 oracle (oracle/ppr.py).

Tolerances: the fp32 Jacobi solve stops at a per-column L1 change <= tol
(1e-7 here); the remaining error is about tol * alpha / (1 - alpha) in L1, so
forward values are compared with atol 1e-6 + rtol 1e-4.  Gradients are
compared to the FP64 adjoint with rtol 1e-3 relative to the largest entry."""
import numpy as np
import pytest

from galois_b200 import DeviceGraph, HostCSR, assign_weights_f32, rmat
from oracle import ppr as oppr

pytestmark = pytest.mark.gpu
ALPHA = 0.85


def setup(scale=10, B=4, seed=5, nnz=8):
    g, _ = rmat(scale, 8, seed=seed, symmetrize=False)
    assign_weights_f32(g, seed=seed)
    rng = np.random.default_rng(seed)
    T = np.zeros((g.n, B), np.float32)
    for b in range(B):
        T[rng.choice(g.n, nnz, replace=False), b] = 1.0 / nnz
    c = rng.standard_normal((g.n, B)).astype(np.float32)
    return g, T, c


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-30))


@pytest.mark.parametrize("B", [1, 4, 128])
def test_forward_backward_vs_fp64(cuda_device, B):
    import torch

    from galois_b200 import _lib

    g, T, c = setup(B=B)
    w64 = g.w_f32.astype(np.float64)
    x_ref = oppr.forward(g, T.astype(np.float64), w64, ALPHA)
    gT_ref, gw_ref = oppr.backward(g, x_ref, c.astype(np.float64), w64, ALPHA)
    with DeviceGraph(g) as dg:
        Tt = torch.from_numpy(T).cuda()
        x = torch.empty_like(Tt)
        import ctypes as C

        st = _lib.lib.gb_ppr_forward(dg.handle, B, C.c_void_p(Tt.data_ptr()), None, ALPHA, 1e-7, 1000,
                                     C.c_void_p(x.data_ptr()), None, None, None)
        assert st == 0, _lib.last_error()
        xh = x.cpu().numpy().astype(np.float64)
        assert np.allclose(xh, x_ref, atol=1e-6, rtol=1e-4)
        ct = torch.from_numpy(c).cuda()
        gT = torch.empty_like(Tt)
        gw = torch.empty(g.m, dtype=torch.float32, device="cuda")
        st = _lib.lib.gb_ppr_backward(dg.handle, B, C.c_void_p(x.data_ptr()), C.c_void_p(ct.data_ptr()), None,
                                      ALPHA, 1e-7, 1000, C.c_void_p(gT.data_ptr()), C.c_void_p(gw.data_ptr()),
                                      None, None, None)
        assert st == 0, _lib.last_error()
        assert rel(gT.cpu().numpy(), gT_ref) < 1e-3
        assert rel(gw.cpu().numpy(), gw_ref) < 1e-3


@pytest.mark.parametrize("B", [1, 4, 8, 12, 20, 32, 36, 64, 68, 100])
def test_row_and_tile_edges(cuda_device, B):
    """Every lanes-per-row variant over rows of 0, 1, 7-9, 31-33 and 63-65
    arcs (a small graph's tile is 32 arcs), a hub of many tiles and a ragged
    vertex count; two runs give the same bits."""
    import torch

    from galois_b200.ppr import ppr

    rng = np.random.default_rng(3)
    n, src, dst = 517, [], []
    for j, d in enumerate((0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 400)):
        to = rng.choice(n, d, replace=False)
        src += [j] * d + list(to)  # the same counts as out-rows and as in-rows
        dst += list(to) + [j] * d
    g = HostCSR.from_edges(n, src, dst)
    assign_weights_f32(g, seed=4)
    T = rng.random((n, B)).astype(np.float32) * (rng.random((n, B)) < 0.1)
    T /= np.maximum(T.sum(0), 1e-30)
    c = rng.standard_normal((n, B)).astype(np.float32)
    w64 = g.w_f32.astype(np.float64)
    x_ref = oppr.forward(g, T.astype(np.float64), w64, ALPHA)
    gT_ref, gw_ref = oppr.backward(g, x_ref, c.astype(np.float64), w64, ALPHA)
    runs = []
    with DeviceGraph(g) as dg:
        for _ in range(2):
            Tt = torch.from_numpy(T).cuda().requires_grad_(True)
            w = torch.from_numpy(g.w_f32).cuda().requires_grad_(True)
            x = ppr(dg, Tt, w, ALPHA, 1e-7)
            runs.append((x, *torch.autograd.grad((torch.from_numpy(c).cuda() * x).sum(), (Tt, w))))
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    x, gT, gw = (t.detach().cpu().numpy() for t in runs[0])
    assert np.allclose(x, x_ref, atol=1e-6, rtol=1e-4)
    assert rel(gT, gT_ref) < 1e-3
    assert rel(gw, gw_ref) < 1e-3


@pytest.mark.parametrize("rows,cols", [(97, 31), (300, 257), (401, 500)])
@pytest.mark.parametrize("B", [4, 8, 128])
def test_grid_rows_per_task(cuda_device, rows, cols, B):
    """Rows of two to four arcs, for which a row's sum takes fewer steps over
    the lanes, and vertex counts that give a task 1, 8 and 16 rows, ragged at
    the end: the forward solve against 64 bits, and each column's sum, which it
    keeps."""
    import torch

    from galois_b200 import grid2d
    from galois_b200.ppr import ppr

    g = grid2d(rows, cols)
    assign_weights_f32(g, seed=3)
    rng = np.random.default_rng(rows)
    T = np.zeros((g.n, B), np.float32)
    T[rng.integers(0, g.n, 8 * B), np.tile(np.arange(B), 8)] = 0.125
    x_ref = oppr.forward(g, T.astype(np.float64), g.w_f32.astype(np.float64), ALPHA)
    with DeviceGraph(g) as dg:
        w = torch.from_numpy(g.w_f32).cuda()
        x = ppr(dg, torch.from_numpy(T).cuda(), w, ALPHA, 1e-7)
        # every vertex has out-arcs, so the solve keeps each column's sum
        assert np.allclose(x.double().sum(0).cpu().numpy(), T.astype(np.float64).sum(0), rtol=1e-5)
    assert np.allclose(x.cpu().numpy(), x_ref, atol=1e-6, rtol=1e-4)


@pytest.mark.parametrize("B", [1, 4, 20, 128])
def test_hub_spans(cuda_device, B):
    """Hubs of exactly 512 tiles of 32 arcs, one arc more, 1024 tiles and one
    arc more (512 tiles make a span, added up before the spans' sums are), in
    both directions, beside light rows; two runs give the same bits."""
    import torch

    from galois_b200.ppr import ppr

    rng = np.random.default_rng(5)
    n, src, dst = 33001, [], []
    for j, d in enumerate((16384, 16385, 32768, 32769)):
        to = rng.choice(np.arange(4, n), d, replace=False)
        src += [np.full(d, j), to]
        dst += [to, np.full(d, j)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    g = HostCSR.from_edges(n, src, dst)
    assert g.m < 148 * 32 * 16 * 64  # tiles of 32 arcs
    assign_weights_f32(g, seed=6)
    T = rng.random((n, B)).astype(np.float32) * (rng.random((n, B)) < 0.1)
    T /= np.maximum(T.sum(0), 1e-30)
    c = rng.standard_normal((n, B)).astype(np.float32)
    w64 = g.w_f32.astype(np.float64)
    x_ref = oppr.forward(g, T.astype(np.float64), w64, ALPHA)
    gT_ref, gw_ref = oppr.backward(g, x_ref, c.astype(np.float64), w64, ALPHA)
    runs = []
    with DeviceGraph(g) as dg:
        for _ in range(2):
            Tt = torch.from_numpy(T).cuda().requires_grad_(True)
            w = torch.from_numpy(g.w_f32).cuda().requires_grad_(True)
            x = ppr(dg, Tt, w, ALPHA, 1e-7)
            runs.append((x, *torch.autograd.grad((torch.from_numpy(c).cuda() * x).sum(), (Tt, w))))
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    x, gT, gw = (t.detach().cpu().numpy() for t in runs[0])
    assert np.allclose(x, x_ref, atol=1e-6, rtol=1e-4)
    assert rel(gT, gT_ref) < 1e-3
    assert rel(gw, gw_ref) < 1e-3


def test_heavy_rows_tiled(cuda_device):
    import torch

    from galois_b200.ppr import ppr

    # a hub with in- and out-degree above the tiling threshold
    n = 3000
    src = [0] * (n - 1) + list(range(1, n)) + list(range(1, n - 1))
    dst = list(range(1, n)) + [0] * (n - 1) + list(range(2, n))
    g = HostCSR.from_edges(n, src, dst)
    assign_weights_f32(g, seed=2)
    rng = np.random.default_rng(1)
    B = 8
    T = np.zeros((n, B), np.float32)
    for b in range(B):
        T[rng.choice(n, 4, replace=False), b] = 0.25
    x_ref = oppr.forward(g, T.astype(np.float64), g.w_f32.astype(np.float64), ALPHA)
    with DeviceGraph(g) as dg:
        x = ppr(dg, torch.from_numpy(T).cuda(), torch.from_numpy(g.w_f32).cuda())
        assert np.allclose(x.cpu().numpy(), x_ref, atol=1e-6, rtol=1e-4)


def test_autograd_matches_fp64_and_finite_differences(cuda_device):
    import torch

    from galois_b200.ppr import ppr

    g, T, c = setup(scale=9, B=8)
    w = torch.from_numpy(g.w_f32.copy()).cuda().requires_grad_(True)
    Tt = torch.from_numpy(T).cuda().requires_grad_(True)
    ct = torch.from_numpy(c).cuda()
    with DeviceGraph(g) as dg:
        x = ppr(dg, Tt, w, ALPHA, 1e-7)
        loss = (ct * x).sum()
        loss.backward()
        w64 = g.w_f32.astype(np.float64)
        x_ref = oppr.forward(g, T.astype(np.float64), w64, ALPHA)
        gT_ref, gw_ref = oppr.backward(g, x_ref, c.astype(np.float64), w64, ALPHA)
        assert rel(Tt.grad.cpu().numpy(), gT_ref) < 1e-3
        assert rel(w.grad.cpu().numpy(), gw_ref) < 1e-3
        # central finite differences of the fp32 GPU forward on a few weights
        rng = np.random.default_rng(4)
        for e in rng.choice(np.flatnonzero(np.abs(gw_ref) > 0.05 * np.abs(gw_ref).max()), 4, replace=False):
            h = 1e-2 * float(g.w_f32[e])
            with torch.no_grad():
                wp = w.detach().clone()
                wp[e] += h
                wm = w.detach().clone()
                wm[e] -= h
                lp = float((ct * ppr(dg, Tt.detach(), wp, ALPHA, 1e-7)).sum())
                lm = float((ct * ppr(dg, Tt.detach(), wm, ALPHA, 1e-7)).sum())
            fd = (lp - lm) / (2 * h)
            assert abs(fd - gw_ref[e]) <= 5e-2 * abs(gw_ref[e]) + 1e-4


def test_ppr_sharded_single_rank_matches_autograd(cuda_device):
    """galois_b200.distributed.ppr_sharded over a one-rank NCCL group gives
    the plain autograd result (the multi-rank split and the all-reduce of
    grad_w are covered by the gloo tests)."""
    import datetime
    import os
    import socket

    import torch
    import torch.distributed as dist

    from galois_b200.distributed import ppr_sharded
    from galois_b200.ppr import ppr

    with socket.socket() as sk:
        sk.bind(("127.0.0.1", 0))
        port = sk.getsockname()[1]
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("nccl", rank=0, world_size=1, timeout=datetime.timedelta(seconds=60),
                            device_id=torch.device("cuda", 0))
    try:
        g, T, c = setup(scale=10, B=8)
        with DeviceGraph(g) as dg:
            Tt = torch.from_numpy(T).cuda()
            ct = torch.from_numpy(c).cuda()
            w = torch.from_numpy(g.w_f32).cuda()
            x, cols, gt, gw, loss = ppr_sharded(dg, Tt, w, ct, ALPHA, 1e-7)
            wr = w.clone().requires_grad_(True)
            Tr = Tt.clone().requires_grad_(True)
            xr = ppr(dg, Tr, wr, ALPHA, 1e-7)
            lr = (ct * xr).sum()
            lr.backward()
        assert cols == (0, 8)
        assert torch.allclose(x, xr.detach())
        assert torch.allclose(gt, Tr.grad)
        assert torch.allclose(gw, wr.grad)
        assert abs(float(loss) - float(lr.detach())) <= 1e-5 * max(1.0, abs(float(lr.detach())))
    finally:
        dist.destroy_process_group()


def test_no_memory_then_memory(cuda_device):
    """First calls on a device without memory for the transpose, then for the
    solve's own arrays, fail and leave nothing half-made: the next calls fail
    the same way, and with memory again the result is another handle's."""
    import torch

    from galois_b200 import _lib, erdos_renyi
    from galois_b200.ppr import ppr

    g = erdos_renyi(400000, 8.0, seed=3)
    assign_weights_f32(g, seed=4)
    T = torch.rand((g.n, 4), device="cuda") / g.n
    x = torch.empty_like(T)
    with DeviceGraph(g) as dg:
        want = ppr(dg, T, None, ALPHA, 1e-6)
    _lib.check(_lib.lib.gb_pool_trim(), "gb_pool_trim")

    def call(dg):
        return _lib.lib.gb_ppr_forward(dg.handle, 4, T.data_ptr(), None, ALPHA, 1e-6, 1000, x.data_ptr(), None, None,
                                       None)

    def take_all():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held = []
        for mb in (8192, 1024, 128, 16, 2):
            while torch.cuda.mem_get_info()[0] > (mb + 4) << 20:
                try:
                    held.append(torch.empty(mb << 20, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        return held

    for transposed in (False, True):
        with DeviceGraph(g) as dg:
            if transposed:
                dg.build_transpose()
            held = take_all()
            for _ in range(2):
                assert call(dg) == _lib.GB_ERR_OOM
            del held
            torch.cuda.empty_cache()
            assert call(dg) == _lib.GB_OK
            torch.cuda.synchronize()
            assert torch.allclose(x, want, atol=1e-9, rtol=1e-5)


@pytest.mark.parametrize("B", [1, 4, 128])
def test_inputs_at_any_word(cuda_device, B):
    """Teleport and loss-gradient tensors that start 4 to 12 bytes into an
    allocation: the autograd entry point copies them, the C entry points
    refuse what the kernels cannot read 16 bytes at a time."""
    import torch

    from galois_b200 import _lib
    from galois_b200.ppr import ppr

    g, T, c = setup(B=4)
    n = g.n
    T = torch.from_numpy(np.tile(T, (1, 32))[:, :B].copy()).cuda()
    c = torch.from_numpy(np.tile(c, (1, 32))[:, :B].copy()).cuda()
    w = torch.from_numpy(g.w_f32).cuda()

    def at(t, words):
        buf = torch.empty(t.numel() + words, device="cuda")
        buf[words:] = t.flatten()
        return buf[words:].view(t.shape)

    with DeviceGraph(g) as dg:
        runs = []
        for words in (0, 1, 2, 3):
            Tt, wt = at(T, words).requires_grad_(True), w.clone().requires_grad_(True)
            assert Tt.data_ptr() % 16 == 4 * words
            x = ppr(dg, Tt, wt, ALPHA, 1e-7)
            runs.append((x, *torch.autograd.grad(x, (Tt, wt), grad_outputs=at(c, words))))
        for r in runs[1:]:
            assert all(torch.equal(a, b) for a, b in zip(r, runs[0]))
        x = torch.empty((n, B), device="cuda")
        gw = torch.empty(g.m, device="cuda")
        ok = _lib.GB_OK if B == 1 else _lib.GB_ERR_ARG

        def forward(t, out):
            return _lib.lib.gb_ppr_forward(dg.handle, B, t.data_ptr(), None, ALPHA, 1e-7, 1000, out.data_ptr(), None,
                                           None, None)

        def backward(xs, gx):
            return _lib.lib.gb_ppr_backward(dg.handle, B, xs.data_ptr(), gx.data_ptr(), None, ALPHA, 1e-7, 1000, None,
                                            gw.data_ptr(), None, None, None)

        assert forward(T, x) == _lib.GB_OK and backward(x, c) == _lib.GB_OK
        assert forward(at(T, 1), x) == ok and forward(T, at(x, 3)) == ok
        assert backward(at(x, 2), c) == ok and backward(x, at(c, 1)) == ok
        torch.cuda.synchronize()
