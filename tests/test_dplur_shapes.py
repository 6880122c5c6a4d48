"""The DP-LUR relaxation at the edges of its blocks (8 rows x 32 columns) and
of the grid, whose outer neighbours contribute nothing, on the three forms of
grid (channel metrics, general metrics, open ends).  FP64 throughout, so the
bar is that of the other parity tests for three inner iterations: 1e-12
relative L2 per variable (fused multiply-adds and refined reciprocals, a few
units in the last place per iteration)."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel


@pytest.mark.gpu
@pytest.mark.parametrize("grid", ["flat", "wavy", "open"])
@pytest.mark.parametrize("dims", [(3, 6, 4), (5, 8, 33), (4, 9, 31), (17, 25, 65)])
def test_iterations_match_oracle(cuda_lib, dims, grid):
    from cgli_fu_flow_b200.solver import Solver
    from oracle.oracle import Oracle
    kw = {}
    if grid == "wavy":
        kw = dict(wavy=True, wave=0.01)
    elif grid == "open":
        kw = dict(x_open=True, nx_inlet=1, nx_outlet=1, buoyancy=True, twall_lo=343.0592)
    ch = Channel(*dims, **kw)
    g, o = Solver(ch), Oracle(ch, inner_solver="dplur")
    g.init()
    o.init()
    g.set_inner_solver("dplur")
    for _ in range(3):
        g.inner_iteration()
        o.inner_iteration()
    sl = np.s_[:, 3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]
    qg, qo = g.q()[sl], o.q()[sl]
    g.close()
    errs = [np.linalg.norm(qg[v] - qo[v]) / np.linalg.norm(qo[v]) for v in range(5)]
    assert max(errs) <= 1e-12, errs
