"""The step-ordered metric terms of a general grid belong to the wavefront
passes: contexts that run none (DP-LUR, the routines, the filter, restart
files) hold no room for them, and new metrics reach the passes."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

CH = Channel(11, 20, 9, wavy=True, wave=0.01)
STREAM_WORDS = 9 * CH.nx * 32 * (CH.nz + 31)            # one block of 32 columns
RECORD_BYTES = 11 * int(np.prod(CH.shape)) * 8          # DP-LUR's coefficient records


@pytest.mark.gpu
def test_only_the_passes_allocate_the_metric_stream(cuda_lib):
    from cgli_fu_flow_b200.solver import Solver
    g = Solver(CH)
    g.init()
    b0 = g.device_bytes
    g.halo_x()
    g.flux_x()
    g.viscous_terms()
    g.dual_time_stepping()
    assert g.device_bytes == b0
    g.set_inner_solver("dplur")
    g.step(2, update_force=False)
    assert g.device_bytes == b0 + RECORD_BYTES
    g.set_inner_solver("lusgs")
    g.step(2, update_force=False)
    assert g.device_bytes == b0 + RECORD_BYTES + 8 * STREAM_WORDS
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["step", "profile", "dplur"])
def test_new_metrics_reach_the_passes(cuda_lib, first):
    """A context that ran on one wavy grid and then gets another's metrics gives
    the words of a context that only ever had those (the driving force held, which
    a step would otherwise adapt)."""
    from cgli_fu_flow_b200.solver import METRIC_NAMES, Solver, channel_metric_host
    other = Channel(11, 20, 9, wavy=True, wave=0.02)
    out = []
    for used in (True, False):
        g = Solver(CH)
        if used:
            g.init()
            if first == "profile":
                g.profile_stages(1)
            else:
                g.set_inner_solver("dplur" if first == "dplur" else "lusgs")
                g.step(2, update_force=False)
                g.set_inner_solver("lusgs")
        for n in METRIC_NAMES:
            g.set(n, channel_metric_host(other, n))
        g.init()
        g.step(2, update_force=False)
        out.append(g.q().view(np.int64))
        g.close()
    assert np.array_equal(out[0], out[1])
