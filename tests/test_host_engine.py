"""CPU tests of the host engine (cism_b200/csrc/bp_engine.cpp) on a fake CUDA
runtime (tests/hostemu/hostengine.cpp): "device" memory is host memory, every
linear solve and Picard loop ends at its first update, and launches can be
refused, to see what the engine makes of an error code."""
import ctypes as C
import os

import numpy as np
import pytest

from cism_b200 import configs, solver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_dp = solver._dp
OK, ERR_CUDA, ERR_ARGS = 0, 6, 10


class Engine:
    """The few calls of the C ABI that the tests need, on the fake."""

    def __init__(self):
        self.L = C.CDLL(os.path.join(ROOT, "tests", "hostemu", "libhostengine.so"))
        self.L.fake_nonzero_holes.restype = C.c_long
        self.L.bp_last_error.restype = C.c_char_p
        self.L.fake_refuse(0)
        self.h = C.c_void_p()
        assert self.L.bp_create(0, C.byref(self.h)) == OK

    def close(self):
        assert self.L.bp_destroy(self.h) == OK

    def problem(self, models, **kw):
        preps = [solver.prepare(m, **kw)[0] for m in models]
        arr = (solver.Inputs * len(preps))(*[p.inputs for p in preps])
        P = C.c_void_p()
        assert self.L.bp_problem_create(self.h, len(preps), arr, C.byref(P)) == OK
        return P

    @staticmethod
    def ptrs(arrays):
        return (_dp * len(arrays))(*[C.cast(None, _dp) if a is None else a.ctypes.data_as(_dp) for a in arrays])

    def set_guess(self, P, us, vs):
        return self.L.bp_problem_set_guess(P, self.ptrs(us), self.ptrs(vs))

    def run(self, P, n=1):
        return self.L.bp_problem_run(P, (solver.Stats * n)())

    def free(self, P):
        self.L.bp_problem_destroy(P)


@pytest.fixture()
def eng():
    e = Engine()
    yield e
    e.close()


def _slab(n, nz=11, **kw):
    return configs.slab(n=n, nz=nz).copy(maxiter_nonlinear=2, **kw)


def _zero(m):
    return [np.zeros(m.vshape3)], [np.zeros(m.vshape3)]


@pytest.mark.parametrize("variant", [configs.SPARSE_PCG_STANDARD, configs.SPARSE_PCG_CHRONGEAR])
@pytest.mark.parametrize("precision", [solver.FP64, solver.MIXED])
def test_refused_launch_in_a_capture_ends_the_run(eng, variant, precision):
    """A Krylov matvec that is refused while a graph is captured: the run ends
    with BP_ERR_CUDA, nothing captured without it is launched, then or later,
    and no capture stays open; without the refusal the problem runs."""
    m = _slab(60, which_sparse=variant)
    P = eng.problem([m], precision=precision)
    assert eng.set_guess(P, *_zero(m)) == OK
    g0 = eng.L.fake_graph_launches()
    eng.L.fake_refuse(1)
    for _ in range(2):
        assert eng.run(P) == ERR_CUDA
        assert eng.L.fake_capturing() == 0
        assert eng.L.fake_graph_launches() == g0
    eng.L.fake_refuse(0)
    assert eng.run(P) in (0, 3, 4)
    assert eng.set_guess(P, *_zero(m)) == OK
    eng.free(P)


def test_refused_launch_outside_a_capture_ends_the_run(eng):
    m = _slab(60)
    P = eng.problem([m])
    assert eng.set_guess(P, *_zero(m)) == OK
    eng.L.fake_refuse(2)
    assert eng.run(P) == ERR_CUDA
    eng.L.fake_refuse(0)
    assert eng.run(P) in (0, 3, 4)
    eng.free(P)


def test_velocity_transfers_leave_the_node_vectors_holes_at_zero(eng):
    """The columns' scratch on the way in and out is no node vector: the slots
    of the vectors that belong to no column stay zero (make_view)."""
    ms = [_slab(13), _slab(10)]
    P = eng.problem(ms)
    rng = np.random.default_rng(4)
    us, vs = ([rng.standard_normal(m.vshape3) for m in ms] for _ in range(2))
    assert eng.set_guess(P, us, vs) == OK
    assert eng.L.fake_nonzero_holes() == 0
    out = [[np.zeros(m.vshape3) for m in ms] for _ in range(2)]
    assert eng.L.bp_problem_get_guess(P, eng.ptrs(out[0]), eng.ptrs(out[1])) == OK
    assert eng.L.fake_nonzero_holes() == 0
    for a, b, m in zip(us + vs, out[0] + out[1], ms + ms):
        js, is_ = m.owned_vertex_slices()
        assert np.array_equal(a[js, is_], b[js, is_])  # a periodic slab: every owned vertex is active
    assert eng.run(P, 2) in (0, 3, 4)
    assert eng.L.bp_problem_get(P, eng.ptrs(out[0]), eng.ptrs(out[1]), None) == OK
    assert eng.L.fake_nonzero_holes() == 0
    eng.free(P)


@pytest.mark.parametrize("n,halo", [(48, True), (49, False)])
def test_halo_tables_are_built_only_where_tiles_may_fit(eng, n, halo):
    """144 tiles fit the fake's 148 CTAs, 151 do not: the halo's tables (0.3 ms
    of host time at 600 tiles) are not built to be thrown away."""
    P = eng.problem([_slab(n)])
    assert (eng.L.fake_resident_halo() > 0) == halo
    eng.free(P)


def test_timing_runs_of_a_resident_problem(eng):
    """A timing run launches the PCG's steps one by one; one of the kernels
    that run untimed (2) has one PCG launch per Picard iteration.  A problem
    that is not resident is timed the same way in both."""
    for n, resident in ((20, 1), (60, 0)):
        m = _slab(n)
        P = eng.problem([m])
        assert eng.L.bp_problem_resident(P) == resident
        count = {}
        for mode in (1, 2):
            assert eng.set_guess(P, *_zero(m)) == OK
            assert eng.L.bp_problem_timing(P, mode) == OK
            assert eng.run(P) in (0, 3, 4)
            ms, k = (C.c_double * 9)(), (C.c_int * 9)()
            assert eng.L.bp_problem_kernel_times(P, ms, k) == OK
            count[mode] = list(k)
        assert count[1][0] > 1 and count[1][1] > 1  # matvecs, updates
        assert count[2][:2] == ([1, 0] if resident else count[1][:2])
        assert count[2][2:] == count[1][2:] or resident
        eng.free(P)


def test_a_call_that_fails_ends_synchronised(eng):
    """A batch of a given and a learned guess without a network: the call is
    refused with no copy from the context's staging buffer still on its way
    (the next call writes there)."""
    ms = [_slab(12), _slab(13)]
    preps = [solver.prepare(m, guess_mode=g)[0] for m, g in zip(ms, (solver.GUESS_GIVEN, solver.GUESS_LEARNED))]
    arr = (solver.Inputs * 2)(*[p.inputs for p in preps])
    P = C.c_void_p()
    assert eng.L.bp_problem_create(eng.h, 2, arr, C.byref(P)) == OK
    z = np.zeros(ms[0].vshape3)
    assert eng.set_guess(P, [z, None], [z, None]) == ERR_ARGS
    assert b"bp_guess_load" in eng.L.bp_last_error(eng.h)
    assert eng.L.fake_copies_open() == 0
    eng.free(P)
