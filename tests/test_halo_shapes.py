"""The iteration's one boundary kernel against the three routines that it
stands for (x halo, wall rows, z copies), whose ghost cells depend on one
another: the ghost cells that an inner iteration leaves equal, bit by bit, those
that the routines give on the state it started from.  The grids include the
smallest one, on which a plane is both images' source."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel


@pytest.mark.gpu
@pytest.mark.parametrize("wavy", [False, True])
@pytest.mark.parametrize("dims", [(3, 6, 4), (4, 7, 5), (5, 31, 33), (9, 12, 126)])
def test_iteration_ghost_cells_equal_the_routines(cuda_lib, dims, wavy):
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(*dims, **(dict(wavy=True, wave=0.01) if wavy else {}))
    a, b = Solver(ch), Solver(ch)
    a.init()
    b.init()
    for _ in range(2):
        a.inner_iteration()
    for v in range(1, 6):
        b.set(f"U{v}_", a.get(f"U{v}_"))
    a.inner_iteration()
    b.halo_x(); b.y_boundary_condition(); b.z_boundary_condition()
    nx, ny, nz = dims
    for v in range(1, 6):
        x, y = a.get(f"U{v}_"), b.get(f"U{v}_")
        x[3:nx + 3, 2:ny + 2, 2:nz + 2] = y[3:nx + 3, 2:ny + 2, 2:nz + 2]
        # as words: the unused corner cells hold the NaN of the initial field's 0 / 0
        assert np.array_equal(x.view(np.int64), y.view(np.int64)), v
    a.close()
    b.close()
