"""The LU-SGS passes at the edges of their work split: a warp owns one x row of
32 columns, a CTA a few rows.  Grids with one row or column more or less than
a whole number of those, the smallest grid, and few steps along k; against the
CPU oracle after three inner iterations.

Tolerance: the bars of the other parity tests, 1e-12 relative L2 per variable
for FP64 (fused multiply-adds and refined reciprocals, a few units in the last
place per iteration) and 1e-6 for the FP32 passes (6e-8 of increments that,
from the random start, are as large as the transverse momenta themselves)."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

pytestmark = pytest.mark.gpu

SHAPES = [(3, 6, 4), (4, 31, 5), (7, 32, 4), (8, 33, 40), (9, 64, 6), (17, 65, 37), (33, 12, 70)]


def rel_l2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("grid", ["flat", "wavy", "open"])
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-6)])
@pytest.mark.parametrize("dims", SHAPES)
def test_iterations_match_oracle(cuda_lib, dims, precision, tol, grid):
    from cgli_fu_flow_b200.solver import Solver
    from oracle.oracle import Oracle
    kw = {}
    if grid == "wavy":
        kw = dict(wavy=True, wave=0.01)
    elif grid == "open":
        kw = dict(x_open=True, nx_inlet=1, nx_outlet=1, buoyancy=True, twall_lo=343.0592)
    ch = Channel(*dims, **kw)
    g, o = Solver(ch, precision), Oracle(ch)
    g.init()
    o.init()
    for _ in range(3):
        g.inner_iteration()
        o.inner_iteration()
    sl = np.s_[:, 3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]
    qg, qo = g.q()[sl], o.q()[sl]
    g.close()
    errs = [rel_l2(qg[v], qo[v]) for v in range(5)]
    assert max(errs) <= tol, errs
