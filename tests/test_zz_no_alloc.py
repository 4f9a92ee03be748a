"""bp_residual_noalloc: the residual entry point that allocates nothing.

It exists for callers that own all device memory themselves (a fixed pool
or budget, or code that must not hit the implicit device synchronisation of
cudaMalloc/cudaFree during a time step): they hand in their own device
buffers and the kernel keeps its reduction scratch in a fixed file-scope
device array.  This test calls it through the C ABI with device buffers
(allocated here, by the test, with torch) and checks its residual and norms
against the existing bp_matvec entry point, on two calls in a row (the
second call reuses the shared scratch left by the first).  This file is
named so that pytest collects it last.
"""
import ctypes as C

import numpy as np
import pytest

from cism_b200 import configs, solver

from helpers import oracle_system, owned_active_rows, random_state

pytestmark = pytest.mark.gpu

_dp = C.c_void_p


@pytest.mark.parametrize("m", [configs.slab(n=24), configs.dome()], ids=lambda m: m.name)
def test_noalloc_residual_matches_matvec(ctx, m):
    import torch

    lib = solver.lib()
    lib.bp_residual_noalloc.argtypes = [C.c_int] * 4 + [_dp] * 13
    lib.bp_residual_noalloc.restype = C.c_int
    su, _, _, A, bu, bv, _ = oracle_system(m, seed=11)
    xu, xv = random_state(m, su, seed=12, scale=5.0)
    # expected through the existing entry point
    yu, yv = ctx.matvec(m, su["active_vertex"], A, xu, xv)
    rows = owned_active_rows(m, su["active_vertex"])
    eu = np.where(rows[..., None], yu - bu, 0.0)
    ev = np.where(rows[..., None], yv - bv, 0.0)
    enr = np.sqrt(np.sum(eu ** 2 + ev ** 2))
    enb = np.sqrt(np.sum(np.where(rows[..., None], bu ** 2 + bv ** 2, 0.0)))
    dev = torch.device("cuda:0")
    t = lambda a, dt=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dt)
    dA = [t(a) for a in A]
    dxu, dxv, dbu, dbv = t(xu), t(xv), t(bu), t(bv)
    dav = t(su["active_vertex"], torch.int32)
    stream = torch.cuda.current_stream(dev).cuda_stream
    for call in range(2):
        dru = torch.full(m.vshape3, np.nan, device=dev, dtype=torch.float64)
        drv = torch.full(m.vshape3, np.nan, device=dev, dtype=torch.float64)
        dn = torch.full((3,), np.nan, device=dev, dtype=torch.float64)
        rc = lib.bp_residual_noalloc(m.nx, m.ny, m.nz, m.periodic, dav.data_ptr(),
                                     *[a.data_ptr() for a in dA], dxu.data_ptr(), dxv.data_ptr(),
                                     dbu.data_ptr(), dbv.data_ptr(), dru.data_ptr(), drv.data_ptr(),
                                     dn.data_ptr(), stream)
        assert rc == 0
        torch.cuda.synchronize(dev)
        ru, rv, nrm = dru.cpu().numpy(), drv.cpu().numpy(), dn.cpu().numpy()
        scale = np.max(np.abs(eu)) + np.max(np.abs(ev))
        assert np.max(np.abs(ru - eu)) <= 1e-13 * scale, call
        assert np.max(np.abs(rv - ev)) <= 1e-13 * scale, call
        assert abs(nrm[0] - enr) <= 1e-13 * enr, call
        assert abs(nrm[1] - enb) <= 1e-13 * enb, call
        assert abs(nrm[2] - enr / enb) <= 1e-12 * (enr / enb), call


def test_noalloc_rejects_oversize(ctx):
    lib = solver.lib()
    lib.bp_residual_noalloc.argtypes = [C.c_int] * 4 + [_dp] * 13
    # 4100 x 4100 x 1 rows exceed the fixed scratch; rejected before any launch
    one = C.c_void_p(1)
    rc = lib.bp_residual_noalloc(4101, 4101, 1, 1, *([one] * 12), None)
    assert rc == 10


@pytest.mark.parametrize("dims", [(6, 6, 1, 1), (6, 9, 3, 0), (9, 7, 3, 1), (40, 23, 11, 1), (64, 64, 15, 0)],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("offset", [0, 1])
def test_noalloc_residual_chunk_edges(dims, offset):
    """Chunks of 32 rows: odd and even numbers of rows, one level, rows whose
    chunk ends the arrays, no active vertex, matrix pointers 16-byte aligned
    (bulk copies) and not (plain loads), more chunks than resident blocks.
    27 products of random values in [-1, 1] per row and block: rounding below
    60 x 2^-53 x 108 < 1e-12 absolute; the norms to the same, relative."""
    import torch

    nx, ny, nz, periodic = dims
    lib = solver.lib()
    lib.bp_residual_noalloc.argtypes = [C.c_int] * 4 + [_dp] * 13
    rng = np.random.default_rng(sum(dims) + offset)
    V, W = nx - 1, ny - 1
    A = [rng.uniform(-1, 1, (W, V, nz, 27)) for _ in range(4)]
    xu, xv, bu, bv = (rng.uniform(-1, 1, (W, V, nz)) for _ in range(4))
    for share in (0.0, 0.5, 1.0):
        av = (rng.uniform(size=(W, V)) < share).astype(np.int32)
        lo = 2 if periodic else 1
        rows = np.zeros((W, V), bool)
        rows[lo:ny - 2, lo:nx - 2] = True
        rows &= av.astype(bool)
        eu, ev = np.zeros((W, V, nz)), np.zeros((W, V, nz))
        X = [np.pad(a, 1) for a in (xu, xv)]
        for m in range(27):
            i, j, k = m % 3, (m // 3) % 3, m // 9
            su, sv = (a[j:j + W, i:i + V, k:k + nz] for a in X)
            eu += A[0][..., m] * su + A[1][..., m] * sv
            ev += A[2][..., m] * su + A[3][..., m] * sv
        eu = np.where(rows[..., None], eu - bu, 0.0)
        ev = np.where(rows[..., None], ev - bv, 0.0)
        dev = torch.device("cuda:0")

        def up(a, off=0):  # off: start the array 8 bytes past a 16-byte boundary
            t = torch.zeros(a.size + 2, device=dev, dtype=torch.float64)
            t[off:off + a.size] = torch.from_numpy(a.reshape(-1))
            return t[off:off + a.size]

        dA = [up(a, offset) for a in A]
        d = [up(a) for a in (xu, xv, bu, bv)]
        dav = torch.from_numpy(av).to(dev)
        out = [torch.full((W * V * nz,), np.nan, device=dev, dtype=torch.float64) for _ in range(2)]
        dn = torch.full((3,), np.nan, device=dev, dtype=torch.float64)
        rc = lib.bp_residual_noalloc(nx, ny, nz, periodic, dav.data_ptr(), *[a.data_ptr() for a in dA],
                                     *[a.data_ptr() for a in d], *[a.data_ptr() for a in out], dn.data_ptr(),
                                     torch.cuda.current_stream(dev).cuda_stream)
        assert rc == 0
        ru, rv = (o.cpu().numpy().reshape(W, V, nz) for o in out)
        assert np.max(np.abs(ru - eu)) <= 1e-12 and np.max(np.abs(rv - ev)) <= 1e-12
        r3 = rows[..., None]
        nr = np.sqrt(np.sum(eu ** 2 + ev ** 2))
        nb = np.sqrt(np.sum(np.where(r3, bu ** 2 + bv ** 2, 0.0)))
        nrm = dn.cpu().numpy()
        assert abs(nrm[0] - nr) <= 1e-12 * max(nr, 1.0) and abs(nrm[1] - nb) <= 1e-12 * max(nb, 1.0)
        assert abs(nrm[2] - (nr / nb if nb > 0 else 0.0)) <= 1e-11


def test_noalloc_calls_after_an_overlap():
    """Calls of different sizes that overlap on two streams spoil each other's
    norms (the header says so); the calls after them, direct ones and replays of
    a captured one, give what they gave before: bitwise, as the sums' order is
    fixed."""
    import torch

    lib = solver.lib()
    lib.bp_residual_noalloc.argtypes = [C.c_int] * 4 + [_dp] * 13
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)
    sizes = [(9, 7, 3, 1), (160, 161, 11, 0), (33, 20, 10, 1)]
    calls = []
    for nx, ny, nz, periodic in sizes:
        n = nz * (nx - 1) * (ny - 1)
        A = [torch.rand(n * 27, generator=g, device=dev, dtype=torch.float64) for _ in range(4)]
        d = [torch.rand(n, generator=g, device=dev, dtype=torch.float64) for _ in range(4)]
        av = torch.ones((nx - 1) * (ny - 1), device=dev, dtype=torch.int32)
        out = [torch.empty(n, device=dev, dtype=torch.float64) for _ in range(2)]
        norms = torch.empty(3, device=dev, dtype=torch.float64)
        calls.append((nx, ny, nz, periodic, av, A, d, out, norms))

    def call(c, stream):
        nx, ny, nz, periodic, av, A, d, out, norms = c
        rc = lib.bp_residual_noalloc(nx, ny, nz, periodic, av.data_ptr(), *[a.data_ptr() for a in A],
                                     *[a.data_ptr() for a in d], *[a.data_ptr() for a in out], norms.data_ptr(),
                                     stream.cuda_stream)
        assert rc == 0

    main = torch.cuda.current_stream(dev)
    streams = [torch.cuda.Stream(dev) for _ in sizes]
    graphs = []
    want = []
    for c in calls:
        c[-1].fill_(float("nan"))
        call(c, main)
        torch.cuda.synchronize(dev)
        want.append(c[-1].clone())
        assert not bool(want[-1].isnan().any())
    for c in calls:
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            call(c, torch.cuda.current_stream(dev))
        graphs.append(gr)
    for turn in range(20):
        for _ in range(5):
            for c, s in zip(calls, streams):
                call(c, s)
        if turn % 2:
            for gr, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    gr.replay()
        torch.cuda.synchronize(dev)
        for replay in (False, True):
            for c, gr, w in zip(calls, graphs, want):
                c[-1].fill_(float("nan"))
                gr.replay() if replay else call(c, main)
                torch.cuda.synchronize(dev)
                assert torch.equal(c[-1], w), (turn, replay, c[:3])
