"""The viscous terms at the edges of their tiles (13 rows x 32 columns, chunks
of x planes chosen by the grid with a remainder) on the three forms of grid.
The bar is that of the routine-by-routine parity test: 1e-11 of the largest
value (second differences of rounded velocities)."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel


@pytest.mark.gpu
@pytest.mark.parametrize("grid", ["flat", "wavy", "open"])
@pytest.mark.parametrize("dims", [(3, 6, 4), (4, 13, 32), (5, 14, 33), (31, 27, 31), (41, 65, 65)])
def test_viscous_terms_match_oracle(cuda_lib, dims, grid):
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
    g.inner_iteration()   # fills the halos and moves the field off its start
    o.inner_iteration()
    g.halo_x(); g.y_boundary_condition()
    for n in ("halo_x", "bc_y", "bc_x", "bc_z") if ch.x_open else ("halo_x", "bc_y", "bc_z"):
        o.call(n)
    if ch.x_open:
        g.x_boundary_condition()
    g.z_boundary_condition()
    g.viscous_terms()
    o.call("viscous")
    sl = np.s_[3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]
    for v in range(2, 6):
        a, b = g.get(f"vF{v}")[sl], o.array(f"vF{v}")[sl]
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max(), v
    g.close()
