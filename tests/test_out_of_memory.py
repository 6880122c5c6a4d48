"""An allocation that cannot be had is reported by the call that asked for it
and by no later one: cudaMalloc leaves its error for the next check of a kernel
launch.  The requests are larger than the device's memory, so nothing is taken
and every one of them is refused at once."""
import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

ENOMEM = -3


def refused(call):
    from cgli_fu_flow_b200.solver import CgliError
    with pytest.raises(CgliError) as ei:
        call()
    assert ei.value.code == ENOMEM


@pytest.mark.gpu
def test_a_refused_allocation_is_reported_once(cuda_lib):
    import torch
    from cgli_fu_flow_b200.cnn import Network
    from cgli_fu_flow_b200.solver import Params, Solver, load_library
    ch = Channel(8, 12, 32)
    g, net = Solver(ch), Network(8, 12, 32)
    g.init()
    net.reserve_levels(4)
    p = Params(30000, 1000, 1000, 1., 1., 1., 1e-3, 1e-4, 1e-5, 0.72, 300., 300., 0., 0, 0, 0, 0, 0, 0, 1.)
    assert 30000 * 1000 * 1000 * 8 > torch.cuda.get_device_properties(0).total_memory
    import ctypes
    h = ctypes.c_void_p()
    L = load_library()
    assert L.cgli_create(ctypes.byref(p), ctypes.byref(h)) == ENOMEM and not h
    g.step(2)
    refused(lambda: Network(30000, 1000, 1024))
    g.step(2)
    net.push_level(g)
    assert np.all(np.isfinite(g.step(2)[1]))
    g.close()
    net.close()
