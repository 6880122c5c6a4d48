"""The inviscid fluxes over their forms: the channel's metrics and general ones,
rows of faces that fill blocks of 64 and rows that do not (a plane's faces as
one run), one face per thread and, on the last grid, four along the stencil
with a remainder.  The bar is that of the routine-by-routine parity test:
1e-12 of the largest value (the same sums with fused multiply-adds and refined
reciprocals)."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel


@pytest.mark.gpu
@pytest.mark.parametrize("grid", ["flat", "wavy", "open"])
@pytest.mark.parametrize("dims", [(3, 6, 4), (5, 9, 33), (6, 10, 64), (7, 12, 63), (130, 126, 113)])
def test_fluxes_match_oracle(cuda_lib, dims, grid):
    from cgli_fu_flow_b200.solver import Solver
    from oracle.oracle import Oracle
    kw = {}
    if grid == "wavy":
        kw = dict(wavy=True, wave=0.01)
    elif grid == "open":
        kw = dict(x_open=True, nx_inlet=1, nx_outlet=1, buoyancy=True, twall_lo=343.0592)
    ch = Channel(*dims, **kw)
    g, o = Solver(ch), Oracle(ch)
    g.init()
    o.init()
    g.halo_x(); g.y_boundary_condition()
    if ch.x_open:
        g.x_boundary_condition()
    g.z_boundary_condition()
    for n in ("halo_x", "bc_y", "bc_x", "bc_z") if ch.x_open else ("halo_x", "bc_y", "bc_z"):
        o.call(n)
    g.flux_x(); g.flux_y(); g.flux_z()
    for n in ("flux_x", "flux_y", "flux_z"):
        o.call(n)
    nx, ny, nz = dims
    reg = {"x": np.s_[2:nx + 3, 1:ny + 1, 1:nz + 1], "y": np.s_[2:nx + 2, 1:ny + 2, 1:nz + 1],
           "z": np.s_[2:nx + 2, 1:ny + 1, 1:nz + 2]}
    for ax, sl in reg.items():
        for v in range(1, 6):
            a, b = g.get(f"inF{ax}{v}")[sl], o.array(f"inF{ax}{v}")[sl]
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), (ax, v)
    g.close()
