"""The wavefront passes' hand-over of products between CTAs in every
combination: a CTA holds 4 rows of 32 columns, up to 8 CTAs along x form a
cluster, so a grid of more than 32 planes and more than 32 rows passes products
inside clusters (pushed), between clusters and between column blocks (both
polled through memory), with a last cluster that is partly filled (45 planes: 8
+ 4 CTAs along x; 70: 8 + 8 + 2) and column blocks that are (8 columns; 1).

Three inner iterations against the CPU oracle, with the bars of
test_sweep_shapes.py (1e-12 relative L2 for FP64, 1e-6 for the FP32 passes), and
the same words after a forced timeout (a wait limit of 0 polls) as without."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

pytestmark = pytest.mark.gpu

SHAPES = [(45, 40, 16), (70, 65, 20)]
GRIDS = {"flat": {}, "wavy": dict(wavy=True, wave=0.01),
         "open": dict(x_open=True, nx_inlet=1, nx_outlet=1, buoyancy=True, twall_lo=343.0592)}


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-6)])
@pytest.mark.parametrize("dims", SHAPES)
def test_iterations_match_oracle(cuda_lib, dims, precision, tol, grid):
    from cgli_fu_flow_b200.solver import Solver
    from oracle.oracle import Oracle
    ch = Channel(*dims, **GRIDS[grid])
    g, o = Solver(ch, precision), Oracle(ch)
    g.init()
    o.init()
    for _ in range(3):
        g.inner_iteration()
        o.inner_iteration()
    sl = np.s_[:, 3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]
    qg, qo = g.q()[sl], o.q()[sl]
    g.close()
    errs = [np.linalg.norm(qg[v] - qo[v]) / np.linalg.norm(qo[v]) for v in range(5)]
    assert max(errs) <= tol, errs


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", SHAPES)
def test_iterations_after_a_timeout(cuda_lib, dims, precision, grid):
    """Every wait between CTAs gives up, twice; then the state is the one of
    before (its boundaries applied), and so are the iterations that follow."""
    from cgli_fu_flow_b200.solver import CgliError, Solver
    ch = Channel(*dims, **GRIDS[grid])
    g, h = Solver(ch, precision), Solver(ch, precision)
    g.init()
    h.init()
    for _ in range(2):
        g.set_wait_limit(0)
        with pytest.raises(CgliError) as ei:
            g.inner_iteration()
        assert ei.value.code == -6
        g.set_wait_limit(4194304)
        h.halo_x()
        h.y_boundary_condition()
        h.x_boundary_condition()
        h.z_boundary_condition()
        assert np.array_equal(g.q().view(np.int64), h.q().view(np.int64))
    g.step(3)
    h.step(3)
    assert np.array_equal(g.q().view(np.int64), h.q().view(np.int64))
    g.close()
    h.close()


@pytest.mark.parametrize("grid", list(GRIDS))
@pytest.mark.parametrize("precision", [0, 1])
def test_nan_products_are_values(cuda_lib, precision, grid):
    """The polls through memory wait for a bit pattern that no arithmetic
    produces: products that are NaN arrive like any other, so a state that is
    not finite is a divergence, not a timeout."""
    from cgli_fu_flow_b200.solver import CgliError, Solver
    ch = Channel(*SHAPES[0], **GRIDS[grid])
    q = ch.initial_conserved().copy()
    q[2, 4, 5, 3] = np.nan
    g = Solver(ch, precision)
    for sign in (1, -1):
        q[2, 4, 5, 3] = np.copysign(np.nan, sign)
        g.init(q)
        with pytest.raises(CgliError) as ei:
            g.step(4)
        assert ei.value.code == -5
    g.close()
