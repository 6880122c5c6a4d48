"""What a failed inner iteration leaves behind: the status word is cleared and
the hand-over buffers hold the sentinel again before the call returns, on the
stream of the passes, so the next call runs normally.

The timeout is forced with a wait limit of 0 polls (see test_failure.py).
Grids: 12 x 2 CTAs of 4 rows x 32 columns along x and y, in clusters of up to 8
along x, so products cross inside clusters, between clusters and between
column blocks.  The compared context applies the boundary conditions once by
hand, which is all that the failed iteration leaves in the state (the halo
planes' wall ghost rows lag by one application), and must then give the same
words."""
import os
import re

import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cgli_fu_flow_b200", "csrc")
ETIMEOUT = -6
LIMIT = 4194304
DIMS = (45, 40, 16)


def test_no_fill_on_the_default_stream():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "capi.cu")).read())
    assert not re.search(r"\bcudaMemset\(", text)


def words(g):
    return g.q().view(np.int64)


def boundaries(g):
    g.halo_x()
    g.y_boundary_condition()
    g.x_boundary_condition()
    g.z_boundary_condition()


def time_out(call):
    from cgli_fu_flow_b200.solver import CgliError
    with pytest.raises(CgliError) as ei:
        call()
    assert ei.value.code == ETIMEOUT


@pytest.mark.gpu
@pytest.mark.parametrize("queued", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_retry_right_after_a_timeout(cuda_lib, precision, queued):
    import torch
    from cgli_fu_flow_b200.solver import Solver
    g, h = Solver(Channel(*DIMS), precision), Solver(Channel(*DIMS), precision)
    g.init()
    h.init()
    boundaries(h)
    h.step(3)
    g.set_wait_limit(0)
    if queued:   # some 30 ms of the caller's work on the default stream
        a = torch.ones(4096, 4096, device="cuda", dtype=torch.bfloat16)
        torch.cuda.synchronize()
        for _ in range(300):
            torch.matmul(a, a)
    time_out(g.inner_iteration)
    g.set_wait_limit(LIMIT)
    g.step(3)
    torch.cuda.synchronize()
    assert np.array_equal(words(g), words(h))
    g.close()
    h.close()


def routine_fluxes(g):
    boundaries(g)
    g.flux_x()
    g.flux_y()
    g.flux_z()
    g.viscous_terms()


@pytest.mark.gpu
@pytest.mark.parametrize("reps", [1, 2])
def test_profile_reports_a_timeout_and_the_routines_after_it_are_right(cuda_lib, reps):
    from cgli_fu_flow_b200.solver import Solver
    g, h = Solver(Channel(*DIMS)), Solver(Channel(*DIMS))
    g.init()
    h.init()
    boundaries(h)
    g.set_wait_limit(0)
    time_out(lambda: g.profile_stages(reps))
    g.set_wait_limit(LIMIT)
    for routine in ("dplusgs", "dual_time_stepping"):
        for s in (g, h):
            routine_fluxes(s)
        eg, eh = getattr(g, routine)(), getattr(h, routine)()
        assert np.array_equal(eg, eh) and np.all(eg > 0)
        assert np.array_equal(words(g), words(h))
    assert all(t > 0 for t in g.profile_stages(1).values())
    g.close()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["lusgs", "dplur"])
def test_divergence_leaves_its_norms(cuda_lib, solver):
    import ctypes
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(8, 12, 8)
    q = ch.initial_conserved().copy()
    q[2, 4, 5, 3] = np.nan
    g = Solver(ch)
    g.set_inner_solver(solver)
    calls = {"iteration": lambda er: g.L.cgli_inner_iteration(g.h, er),
             "fixed": lambda er: g.L.cgli_step(g.h, 4, 1e-3, 30, ctypes.byref(ctypes.c_int()), er),
             "drop": lambda er: g.L.cgli_step(g.h, 0, 1e-3, 30, ctypes.byref(ctypes.c_int()), er)}
    for name, call in calls.items():
        g.init(q)
        er = (ctypes.c_double * 5)(*[7.0] * 5)
        assert call(er) == -5, name
        assert 7.0 not in er[:] and not np.all(np.isfinite(er[:])), (name, er[:])
    g.close()


OPEN = dict(x_open=True, nx_inlet=4, nx_outlet=5, buoyancy=True, twall_lo=343.0592)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kw", [{}, dict(wavy=True, wave=0.01), OPEN], ids=["flat", "wavy", "open"])
def test_iterations_behind_a_timeout_leave_the_state_alone(cuda_lib, kw, precision):
    """A step whose first iteration times out, with nine more behind it, leaves
    the words of one iteration that timed out (ghost cells included), and so
    does the retry."""
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(*DIMS, **kw)
    g, h = Solver(ch, precision), Solver(ch, precision)
    g.init()
    h.init()
    for s, call in ((g, lambda: g.step(10)), (h, h.inner_iteration)):
        s.set_wait_limit(0)
        time_out(call)
        s.set_wait_limit(LIMIT)
    assert np.array_equal(words(g), words(h))
    g.step(2)
    h.step(2)
    assert np.array_equal(words(g), words(h))
    g.close()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["lusgs", "dplur"])
@pytest.mark.parametrize("kw", [{}, OPEN], ids=["flat", "open"])
def test_iterations_behind_a_divergence_leave_the_state_alone(cuda_lib, kw, solver):
    from cgli_fu_flow_b200.solver import CgliError, Solver
    ch = Channel(17, 12, 8, **kw)
    q = ch.initial_conserved().copy()
    q[2, 8, 5, 3] = np.nan
    out = []
    for fixed in (True, False):
        g = Solver(ch)
        g.set_inner_solver(solver)
        g.init(q)
        with pytest.raises(CgliError) as ei:
            g.step(10) if fixed else g.inner_iteration()
        assert ei.value.code == -5
        out.append(words(g))
        g.close()
    assert np.array_equal(out[0], out[1])
