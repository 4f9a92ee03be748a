"""GPU tests of the engine's execution paths: the device-resident Picard
loop against the host-driven one, and the learned guess behind the C ABI
against the network's Python forward.

Tolerances: device loop vs host loop, bitwise (the same kernels in the
same order); the C-ABI guess vs the Python forward of the same weights,
1e-6 relative
(identical arithmetic and BF16 rounding points; a last-bit difference of
log10 can move one BF16 input by one unit).
"""
import os

import numpy as np
import pytest

from cism_b200 import configs, solver

from helpers import rel_l2, small_models

pytestmark = pytest.mark.gpu

MODELS = {m.name: m for m in small_models()}


class _Env:
    """Set environment switches the engine reads when it builds a problem or
    starts a run, and restore them."""

    def __init__(self, **kw):
        self.kw = kw
        self.old = {}

    def __enter__(self):
        for k, v in self.kw.items():
            self.old[k] = os.environ.get(k)
            os.environ[k] = v

    def __exit__(self, *a):
        for k, v in self.old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


@pytest.mark.parametrize("precision", [solver.FP64, solver.MIXED])
def test_device_loop_equals_host_loop(ctx, precision):
    m = configs.marine(n=40, dx=4000.0).copy(pcg_maxiters=2000, which_resid=configs.RESID_L2NORM_RELATIVE,
                                             which_precond=configs.PRECOND_SIA)
    prep, u0, v0 = solver.prepare(m, precision=precision)
    out = {}
    for loop in ("0", "1"):
        with _Env(BP_DEVICE_LOOP=loop):
            prob = ctx.problem([prep])
            prob.set_guess([u0], [v0])
            prob.run()  # first run: the autotuner, then the device loop takes over
            prob.set_guess([u0], [v0])
            st = prob.run()[0]  # a whole run in the device loop
            u, v, _ = prob.get()
            prob.close()
        out[loop] = (u[0], v[0], st)
    (ua, va, sa), (ub, vb, sb) = out["0"], out["1"]
    assert sa["status"] == sb["status"] == 0
    assert (sa["picard_iters"], sa["pcg_iters_total"]) == (sb["picard_iters"], sb["pcg_iters_total"])
    assert np.array_equal(ua, ub) and np.array_equal(va, vb)


def _random_network(seed=3, n_in=6):
    from cism_b200 import net

    model = net.UNet(n_out=24, seed=seed, n_in=n_in)
    model.in_shift = np.array([1.0, 0.1, -0.1, 2.5, 0.0, 4.0][:n_in], np.float32)
    model.in_scale = np.array([0.8, 0.5, 0.5, 1.2, 1.0, 2.0][:n_in], np.float32)
    model.out_scale = 35.0
    return model


@pytest.mark.parametrize("n_in", [5, 6])
def test_learned_guess_c_abi_matches_python(ctx, tmp_path, n_in):
    """Five inputs, or six with the flow-law factor channel."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net

    model = _random_network(n_in=n_in)
    path = str(tmp_path / "net.npz")
    model.save(path)
    ctx.load_guess(path)
    ms = [configs.marine(n=40, dx=4000.0, seed=s) for s in (11, 12)]
    preps = [solver.prepare(m, guess_mode=solver.GUESS_LEARNED)[0] for m in ms]
    prob = ctx.problem(preps)
    n0 = ctx.guess_launches()
    prob.set_guess([None, None], [None, None])
    assert ctx.guess_launches() > n0
    gu, gv = prob.get_guess()
    prob.close()
    # the Python forward of the same weights on the same features
    F = np.stack([net.normalized_input(model, net.pad_grid(net.input_features(m, p.arrays, n_in)))
                  for m, p in zip(ms, preps)])
    x = torch.tensor(F, dtype=torch.float32, device="cuda").to(torch.bfloat16).contiguous()
    out = model.forward(x, int(ms[0].periodic), train=False).cpu().numpy() * model.out_scale
    for m, p, o, u, v in zip(ms, preps, out, gu, gv):
        pu, pv = net.guess_from_grid(m, o, p.arrays["active_vertex"])
        av = p.arrays["active_vertex"].astype(bool)
        assert np.abs(pu).max() > 0.0
        assert rel_l2([u[av], v[av]], [pu[av], pv[av]]) < 1e-6


def test_learned_start_converges_to_the_plain_answer(ctx, tmp_path):
    pytest.importorskip("torch")
    model = _random_network(seed=4)
    path = str(tmp_path / "net.npz")
    model.save(path)
    ctx.load_guess(path)
    m = configs.marine(n=40, dx=4000.0, seed=7).copy(pcg_maxiters=2000, which_resid=configs.RESID_L2NORM_RELATIVE)
    prep, u0, v0 = solver.prepare(m)
    u, v, _, st = ctx.solve_prepared(prep, u0, v0, want_efvs=False)
    prep_l, _, _ = solver.prepare(m, precision=solver.MIXED, guess_mode=solver.GUESS_LEARNED)
    ul, vl, _, stl = ctx.solve_prepared(prep_l, np.zeros_like(u0), np.zeros_like(v0), want_efvs=False)
    assert st["status"] == stl["status"] == 0
    # the relative-residual criterion ends both at the same point
    assert rel_l2([ul, vl], [u, v]) < 1e-6


def test_learned_guess_needs_a_network():
    c = solver.Context(0)
    try:
        m = configs.marine(n=40, dx=4000.0)
        prep, u0, v0 = solver.prepare(m, guess_mode=solver.GUESS_LEARNED)
        with pytest.raises(solver.BPError) as e:
            c.solve_prepared(prep, u0, v0)
        assert e.value.code == 10
        with pytest.raises(solver.BPError):
            c.load_guess("/nonexistent/weights.bin")
    finally:
        c.close()


@pytest.mark.parametrize("name", ["marine", "slab"])
def test_element_centric_assembly_equals_row_form(ctx, name):
    """k_asm_elem + the gathering row kernel against the row-integrating
    kernel (BP_ASM_ELEM=0) on the same state: bitwise the same matrix,
    right-hand side and viscosity."""
    m = (configs.marine(n=40, dx=4000.0) if name == "marine" else configs.slab(n=24))
    prep, u0, v0 = solver.prepare(m)
    rng = np.random.default_rng(5)
    u = u0 + 50.0 * rng.standard_normal(u0.shape)
    v = v0 + 50.0 * rng.standard_normal(v0.shape)
    outs = []
    for flag in ("0", "1"):
        with _Env(BP_ASM_ELEM=flag):
            A, bu, bv, efvs = ctx.assemble(prep, u, v)
        outs.append(A + [bu, bv, efvs])
    assert np.count_nonzero(outs[0][0]) > 0
    for a, b in zip(*outs):
        assert np.array_equal(a, b)


def _resident_models():
    """Sizes around the resident PCG's edges: one tile, a last tile of one
    column, 64 levels (tiles of four columns), 256-node tiles, the 2-D solves
    (256-column tiles), the most tiles that fit (144 and 147 of 11 levels) and
    the first that does not (the launched kernels run both times)."""
    cap = dict(pcg_maxiters=60, maxiter_nonlinear=3)
    return [configs.dome(n=9, nz=3, radius=4.0e3).copy(**cap), configs.dome(n=21, nz=8, radius=15.0e3).copy(**cap),
            configs.dome(n=13, nz=64, radius=7.0e3).copy(**cap), configs.slab(n=17, nz=11).copy(**cap),
            configs.slab(n=49, ny_cells=48, nz=11).copy(**cap), configs.slab(n=48, nz=11).copy(**cap),
            configs.slab(n=52, nz=11).copy(**cap), configs.marine(n=40, dx=4000.0).copy(**cap),
            configs.marine(n=36, dx=4000.0).copy(approx_2d=configs.APPROX_SSA, **cap),
            configs.slab(n=36).copy(approx_2d=configs.APPROX_DIVA, **cap)]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
@pytest.mark.parametrize("precond", [configs.PRECOND_NONE, configs.PRECOND_DIAG, configs.PRECOND_SIA])
def test_resident_pcg_equals_launched(ctx, variant, precond, mixed):
    """The resident PCG against the launched kernels (a timing run launches
    every step): the same arithmetic in the same order, so bitwise the same
    velocities, iterations and norms; also for a batch of uneven instances
    that end at different iterations, and with a check every 1, 3 and 5."""
    models = [m for m in _resident_models() if not (m.approx_2d and precond == configs.PRECOND_SIA)]
    groups = [[m] for m in models]
    groups.append([configs.slab(n=16).copy(pcg_maxiters=40, maxiter_nonlinear=4),
                   configs.dome(n=15, nz=11, radius=11.0e3).copy(pcg_maxiters=400, maxiter_nonlinear=3),
                   configs.dome(n=9, nz=11, radius=4.0e3).copy(pcg_maxiters=7, maxiter_nonlinear=2)])
    for i, ms in enumerate(groups):
        ncheck = (5, 1, 3)[i % 3]
        ms = [m.copy(which_sparse=variant, which_precond=precond, pcg_ncheck=ncheck, pcg_tol=1e-5) for m in ms]
        preps = [solver.prepare(m, precision=solver.MIXED if mixed else solver.FP64)[0] for m in ms]
        prob = ctx.problem(preps)
        zero = [np.zeros(m.vshape3) for m in ms]
        got = []
        for timing in (False, False, True):
            prob.timing(timing)
            prob.set_guess(zero, zero)
            st = prob.run()
            u, v, e = prob.get(want_efvs=True)
            got.append((u, v, e, st))
        prob.timing(False)
        prob.close()
        keys = ("status", "picard_iters", "pcg_iters_total", "pcg_iters_last", "refine_steps_total", "converged",
                "pcg_err_last", "resid_velo", "L2_norm", "L2_norm_relative")
        for other in got[1:]:
            for a, b in zip(got[0][:3], other[:3]):
                assert all(np.array_equal(x, y) for x, y in zip(a, b)), (ms[0].name, ncheck)
            for s, r in zip(got[0][3], other[3]):
                assert {k: s[k] for k in keys} == {k: r[k] for k in keys}, (ms[0].name, ncheck)


def _staged_models():
    """Past the resident PCG's sizes: odd rows (tiles that wrap from one row to
    the next), a front, an outflow domain with ice at its edges, sheets with
    scattered holes (tiles cut into many rows, some past a descriptor's halo),
    tiles of 256 (8 levels), 224 (14), 160 (5) and 132 nodes (33 levels), and
    columns too short for the staged kernel (2 levels: the per-node kernel)."""
    cap = dict(pcg_maxiters=25, maxiter_nonlinear=2)
    holes = configs.slab(n=90, nz=11)
    rng = np.random.default_rng(8)
    keep = rng.uniform(size=holes.thck.shape) < 0.55
    thin = holes.copy(thck=configs.halo_fill_cells(np.where(keep, holes.thck, 0.0)), **cap)
    return [configs.slab(n=75, ny_cells=71, nz=11).copy(**cap), configs.marine(n=100, dx=4000.0).copy(**cap),
            configs.marine(n=100, dx=4000.0, radius_frac=0.7).copy(periodic=0, **cap), thin,
            configs.slab(n=101, nz=8).copy(**cap), configs.slab(n=75, nz=14).copy(**cap),
            configs.slab(n=111, nz=5).copy(**cap), configs.slab(n=41, nz=33).copy(**cap),
            configs.slab(n=210, nz=2).copy(**cap)]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
def test_staged_matvec_equals_per_node(ctx, variant, mixed):
    """The staged Krylov matvec against the per-node kernels: the same
    arithmetic in the same order, so bitwise the same solves; also a batch
    whose instances end at different iterations."""
    groups = [[m] for m in _staged_models()]
    groups.append([configs.slab(n=64).copy(pcg_maxiters=40, maxiter_nonlinear=3),
                   configs.dome(n=31, nz=11).copy(pcg_maxiters=12, maxiter_nonlinear=2),
                   configs.slab(n=50).copy(pcg_maxiters=7, maxiter_nonlinear=4)])
    for i, ms in enumerate(groups):
        pc = (configs.PRECOND_SIA, configs.PRECOND_DIAG)[i % 2]
        ms = [m.copy(which_sparse=variant, which_precond=pc, pcg_tol=1e-6) for m in ms]
        preps = [solver.prepare(m, precision=solver.MIXED if mixed else solver.FP64)[0] for m in ms]
        zero = [np.zeros(m.vshape3) for m in ms]
        got = []
        for config in ("0,0,0,0,0", "0,0,0,0,1", "0,0,0,37,1"):
            with _Env(BP_MV_CONFIG=config):
                prob = ctx.problem(preps)
                prob.set_guess(zero, zero)
                prob.run()
                st = prob.run()
                u, v, _ = prob.get()
                prob.close()
            got.append((u, v, st))
        keys = ("status", "picard_iters", "pcg_iters_total", "refine_steps_total", "pcg_err_last", "L2_norm")
        for other in got[1:]:
            for a, b in zip(got[0][:2], other[:2]):
                assert all(np.array_equal(x, y) for x, y in zip(a, b)), ms[0].name
            for s, r in zip(got[0][2], other[2]):
                assert {k: s[k] for k in keys} == {k: r[k] for k in keys}, ms[0].name


@pytest.mark.parametrize("dims", [(9, 8, 2, 1, 0.5), (40, 33, 7, 0, 0.8), (110, 97, 11, 1, 0.7), (64, 20, 31, 0, 1.0)])
def test_matvec_of_a_callers_matrix(ctx, dims):
    """bp_matvec on matrices the device puts in node order in chunks of at
    most 38,836 rows: one chunk, a last warp of a few rows, and four chunks in
    turn in the two halves of the staging buffer.  Products of values in
    [-1, 1], 54 a row: rounding below 54 x 54 x 2^-53 < 1e-12."""
    nx, ny, nz, periodic, share = dims
    rng = np.random.default_rng(nx * nz)
    V, W = nx - 1, ny - 1
    A = [rng.uniform(-1, 1, (W, V, nz, 27)) for _ in range(4)]
    av = (rng.uniform(size=(W, V)) < share).astype(np.int32)
    m = configs.slab(n=nx - 4, ny_cells=ny - 4, nz=nz).copy(periodic=periodic)
    assert (m.nx, m.ny) == (nx, ny)
    xu, xv = (configs.halo_fill_stag(rng.uniform(-1, 1, (W, V, nz)), periodic) for _ in range(2))
    avh = configs.halo_fill_stag(av.astype(float), periodic)
    yu, yv = ctx.matvec(m, av, A, xu, xv)
    js, is_ = m.owned_vertex_slices()
    own = np.zeros((W, V), bool)
    own[js, is_] = True
    # a neighbour counts where it is an owned active vertex or the image of one
    X = [np.pad(np.where(avh[..., None] != 0, a, 0.0), 1) for a in (xu, xv)]
    eu, ev = np.zeros((W, V, nz)), np.zeros((W, V, nz))
    for q in range(27):
        i, j, k = q % 3, (q // 3) % 3, q // 9
        su, sv = (a[j:j + W, i:i + V, k:k + nz] for a in X)
        eu += A[0][..., q] * su + A[1][..., q] * sv
        ev += A[2][..., q] * su + A[3][..., q] * sv
    rows = (own & (av != 0))[..., None]
    assert np.max(np.abs(yu - np.where(rows, eu, 0.0))) <= 1e-12
    assert np.max(np.abs(yv - np.where(rows, ev, 0.0))) <= 1e-12


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
def test_staged_sums_of_many_and_of_large_instances(ctx, variant, mixed):
    """The staged matvec's last CTA: 45 instances whose sums all end in one CTA
    (more than one list of 32, more tiles than threads), and an instance whose
    partials pass shared memory in several chunks.  Bitwise the per-node
    kernels' solves, as above."""
    many = [configs.slab(n=22 + i % 3, nz=11) for i in range(45)]
    for ms, grid in ((many, 1), ([configs.slab(n=250, nz=11)], 0)):
        ms = [m.copy(which_sparse=variant, which_precond=configs.PRECOND_SIA, pcg_tol=1e-6, pcg_maxiters=6 + i % 4,
                     maxiter_nonlinear=1) for i, m in enumerate(ms)]
        preps = [solver.prepare(m, precision=solver.MIXED if mixed else solver.FP64)[0] for m in ms]
        zero = [np.zeros(m.vshape3) for m in ms]
        got = []
        for config in ("0,0,0,0,0", f"0,0,0,{grid},1"):
            with _Env(BP_MV_CONFIG=config):
                prob = ctx.problem(preps)
                prob.set_guess(zero, zero)
                st = prob.run()
                u, v, _ = prob.get()
                prob.close()
            got.append((u, v, st))
        for a, b in zip(got[0][:2], got[1][:2]):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
        keys = ("status", "pcg_iters_total", "refine_steps_total", "pcg_err_last", "L2_norm")
        for s, r in zip(got[0][2], got[1][2]):
            assert {k: s[k] for k in keys} == {k: r[k] for k in keys}
