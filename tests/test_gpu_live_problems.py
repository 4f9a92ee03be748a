"""GPU tests of problems that are alive beside each other: what a launch may
ask for (its shared memory above all) must not depend on which problem was
created last, on this context or on another thread's.  Every comparison is
bitwise with the solve of the problem alone.
"""
import threading

import numpy as np
import pytest

from cism_b200 import configs, solver

from test_gpu_engine import _Env

pytestmark = pytest.mark.gpu

KEYS = ("status", "picard_iters", "pcg_iters_total", "refine_steps_total", "pcg_err_last", "L2_norm")


def _prep(m, mixed):
    return solver.prepare(m, precision=solver.MIXED if mixed else solver.FP64)[0]


def _run(prob, m):
    z = [np.zeros(m.vshape3)]
    prob.set_guess(z, z)
    st = prob.run()[0]
    u, v, _ = prob.get()
    return u[0], v[0], {k: st[k] for k in KEYS}


def _alone(ctx, m, mixed, runs=2):
    prob = ctx.problem([_prep(m, mixed)])
    out = [_run(prob, m) for _ in range(runs)][-1]
    prob.close()
    return out


def _same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
def test_resident_problems_beside_each_other(ctx, variant, mixed):
    """A problem of the resident PCG (10 levels, SIA factors) before and after
    one that needs less shared memory of the same kernel (9 levels, so tiles of
    144 nodes and not 160, no factors) is created; the third problem is tuned
    and captured after a fourth, smaller one was made."""
    cap = dict(pcg_maxiters=60, maxiter_nonlinear=3, which_sparse=variant)
    big = configs.dome(n=21, nz=10, radius=15.0e3).copy(which_precond=configs.PRECOND_SIA, **cap)
    small = configs.dome(n=15, nz=9, radius=11.0e3).copy(which_precond=configs.PRECOND_DIAG, **cap)
    ref_big, ref_small = _alone(ctx, big, mixed), _alone(ctx, small, mixed)
    A = ctx.problem([_prep(big, mixed)])
    assert _same(_run(A, big), ref_big)
    B = ctx.problem([_prep(small, mixed)])
    assert _same(_run(A, big), ref_big)
    assert _same(_run(B, small), ref_small)
    C = ctx.problem([_prep(big, mixed)])
    D = ctx.problem([_prep(small, mixed)])
    for prob, m, ref in ((C, big, ref_big), (D, small, ref_small), (A, big, ref_big), (C, big, ref_big)):
        assert _same(_run(prob, m), ref)
    for prob in (A, B, C, D):
        prob.close()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
def test_staged_problems_beside_each_other(ctx, variant, mixed):
    """The same for the staged matvec: 11 levels, then 10 of the same kernel.
    One Picard iteration, so that the run after the second problem's creation
    is the one that captures the loop."""
    cap = dict(pcg_maxiters=25, maxiter_nonlinear=1, which_sparse=variant, which_precond=configs.PRECOND_SIA)
    big, small = (configs.slab(n=75, nz=nz).copy(**cap) for nz in (11, 10))
    with _Env(BP_MV_CONFIG="0,0,0,0,1"):
        ref_big, ref_small = _alone(ctx, big, mixed), _alone(ctx, small, mixed)
        A = ctx.problem([_prep(big, mixed)])
        assert _same(_run(A, big), ref_big)
        B = ctx.problem([_prep(small, mixed)])
        assert _same(_run(A, big), ref_big)
        for prob, m, ref in ((B, small, ref_small), (B, small, ref_small), (A, big, ref_big)):
            assert _same(_run(prob, m), ref)
        A.close()
        B.close()


@pytest.mark.parametrize("mixed", [False, True])
def test_two_contexts_on_two_threads(mixed):
    """Distinct contexts on distinct threads, each making and running resident
    problems of different sizes in turn."""
    cap = dict(pcg_maxiters=60, maxiter_nonlinear=3, which_sparse=configs.SPARSE_PCG_STANDARD)
    models = [configs.dome(n=n, nz=nz, radius=r).copy(which_precond=pc, **cap)
              for n, nz, r, pc in ((21, 10, 15.0e3, configs.PRECOND_SIA), (15, 9, 11.0e3, configs.PRECOND_DIAG),
                                   (31, 10, 22.0e3, configs.PRECOND_SIA), (9, 3, 4.0e3, configs.PRECOND_NONE))]
    preps = [_prep(m, mixed) for m in models]
    with solver.Context(0) as c:
        refs = [_alone(c, m, mixed) for m in models]
    bad = []

    def work(first):
        try:
            with solver.Context(0) as c:
                for i in range(12):
                    j = (first + i) % len(models)
                    prob = c.problem([preps[j]])
                    got = [_run(prob, models[j]) for _ in range(2)]
                    prob.close()
                    bad.extend((first, i, models[j].nz) for g in got if not _same(g, refs[j]))
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            bad.append((first, repr(e)))

    th = [threading.Thread(target=work, args=(t,)) for t in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
