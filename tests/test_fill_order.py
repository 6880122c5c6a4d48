"""Buffers that a context allocates when it first needs them are zeroed on the
context's own stream.  That stream is a non-blocking one: a fill on the default
stream (asynchronous to the host, and behind whatever the caller has queued
there) has no order against the kernels that write the buffer, and could zero
what they wrote.

The GPU tests queue ordinary work on the default stream (torch's) before the
call, and compare with a context that ran without it: the same kernels on the
same inputs, so the same words."""
import os
import re

import numpy as np
import pytest

from cgli_fu_flow_b200.channel import Channel

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cgli_fu_flow_b200", "csrc")


def test_context_fills_are_on_a_stream():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "capi.cu")).read())
    body = text[text.index("int alloc(cgli_ctx"):]
    body = body[:body.index("\n}\n")]
    assert not re.search(r"\bcudaMemset\(", body), "alloc fills on the default stream"
    assert re.search(r"cudaMemsetAsync\([^;]*c->stream\)", body)


def queue_work():
    """Some 30 ms of matrix products on the default stream, not waited for."""
    import torch
    a = torch.ones(4096, 4096, device="cuda", dtype=torch.bfloat16)
    for _ in range(300):
        torch.matmul(a, a)


def words(g):
    return g.q().view(np.int64)


@pytest.mark.gpu
def test_dplur_records_of_a_running_context(cuda_lib):
    import torch
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(24, 40, 48)
    out = []
    for queued in (False, True):
        g = Solver(ch)
        g.init()
        g.step(2)                       # the metrics are checked, nothing is left to wait for
        torch.cuda.synchronize()
        if queued:
            queue_work()
        g.set_inner_solver("dplur")     # allocates the records
        g.step(2)
        torch.cuda.synchronize()
        g.step(2)                       # a late fill would reach these
        out.append(words(g))
        g.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_general_metrics_of_a_running_context(cuda_lib, precision):
    import torch
    from cgli_fu_flow_b200.solver import Solver
    flat, wavy = Channel(24, 40, 48), Channel(24, 40, 48, wavy=True, wave=0.01)
    src = Solver(wavy, precision)
    names = ["J", "xidx", "xidy", "etdx", "etdy", "etdz", "ztdz"]
    metrics = {n: src.get(n) for n in names}
    src.close()
    out = []
    for queued in (False, True):
        g = Solver(flat, precision)
        g.init()
        g.step(2)
        torch.cuda.synchronize()
        if queued:
            queue_work()
        for n in names:
            g.set(n, metrics[n])
        g.step(2)                       # allocates the metric stream
        torch.cuda.synchronize()
        g.step(2)
        out.append(words(g))
        g.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
def test_statistics_and_filter_of_a_running_context(cuda_lib):
    import torch
    from cgli_fu_flow_b200.solver import Solver
    ch = Channel(24, 40, 48)
    y = np.broadcast_to(np.linspace(0.0, 1.0, ch.shape[1])[None, :, None], ch.shape)
    out = []
    for queued in (False, True):
        g = Solver(ch)
        g.init()
        g.step(2)
        torch.cuda.synchronize()
        if queued:
            queue_work()
        g.accumulate_statistics()
        ep = g.filter(y, 0.5, 1.0, 0.1)
        torch.cuda.synchronize()
        out.append(ep + [g.statistics()[0], g.get("Y_point")])
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
    assert np.array_equal(out[1][-1], y)


def test_network_fills_are_on_a_stream():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "cnn.cu")).read())
    assert not re.search(r"\bcudaMemset\(", text)


@pytest.mark.gpu
def test_network_made_behind_queued_work(cuda_lib):
    import torch
    from cgli_fu_flow_b200.cnn import Network
    from oracle import cnn_oracle as O
    dims = (12, 8, 32)
    rng = np.random.default_rng(5)
    theta = O.init_params(5)
    x0, target = rng.standard_normal((15,) + dims), rng.standard_normal((5,) + dims)
    torch.cuda.synchronize()
    out = []
    for queued in (False, True):
        if queued:
            queue_work()
        net = Network(*dims)
        net.set_params(theta)
        loss, grad = net.loss_grad(x0, target)   # allocates the training buffers
        torch.cuda.synchronize()
        out.append((loss, grad, net.get_params(), net.forward(x0)))
        net.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)
