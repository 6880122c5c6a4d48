"""The filter's levels at the edges of their work split: tiles of 8 rows x 32
columns and chunks of x planes chosen by the grid (one plane a CTA on a small
grid, several with a remainder on a longer one).  The arithmetic is that of
Filter.cpp in its order with correctly rounded operations, so the sensitivity
fields are equal to the oracle's bit by bit."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel
from oracle import filter_oracle as F

E_HIGH, E_LOW = 0.1, 0.01


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(3, 6, 4), (5, 8, 33), (23, 17, 31), (150, 33, 65)])
def test_filter_matches_oracle_bit_by_bit(cuda_lib, dims):
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(*dims)
    g = Solver(ch)
    g.init()
    g.halo_x(); g.y_boundary_condition(); g.z_boundary_condition()
    U = [g.get(f"U{v}_") for v in range(1, 6)]
    J, yp = g.get("J"), ch.y_point()
    M = F.face_masks(ch.nx, ch.ny, ch.nz, J.shape)
    crit = float(np.median(F.sensor(U, J, yp, ch.nx, ch.ny, ch.nz)[0][M[0]]))
    got = g.filter(yp, crit, E_HIGH, E_LOW)
    want, _, _ = F.filter_ep(U, J, yp, ch.nx, ch.ny, ch.nz, crit, E_HIGH, E_LOW)
    g.close()
    for f in range(3):
        assert np.array_equal(got[f][M[f]], want[f][M[f]]), "XYZ"[f]
