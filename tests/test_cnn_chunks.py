"""Long x chunks of the convolutions, which wrap the planes' and the
accumulators' rings many times: with 148 columns of cells the grid is one CTA
per column over all 70 planes, with 37 it is four chunks per column (148 SMs).
An input that repeats four times along z (periodic) gives the same network the
same numbers in each repeat, word by word.  The loss is a mean over four times
as many cells, so the gradients at the output are a fourth, exactly, and the
parameters' gradients agree up to the order of FP32 sums of n = 7e5 terms: a few
6e-8 sqrt(n) = 5e-5 of their L2 norm; the bar is 3e-4."""
import numpy as np
import pytest

from oracle import cnn_oracle as O


@pytest.mark.gpu
def test_one_chunk_per_column_equals_several(cuda_lib):
    from cgli_fu_flow_b200.cnn import Network
    nx, ny, nz, rep = 70, 148, 32, 4
    rng = np.random.default_rng(3)
    W, b = O.unpack(O.init_params(3))
    W[-1] = rng.uniform(-0.05, 0.05, size=W[-1].shape)
    theta = O.pack(W, b)
    x0 = rng.standard_normal((15, nx, ny, nz)).astype(np.float32)
    target = rng.standard_normal((5, nx, ny, nz)).astype(np.float32)
    out = []
    for r in (1, rep):
        net = Network(nx, ny, nz * r)
        net.set_params(theta)
        x, t = np.tile(x0, (1, 1, 1, r)), np.tile(target, (1, 1, 1, r))
        out.append((net.forward(x), *net.loss_grad(x, t)))
        net.close()
    (f1, l1, g1), (f4, l4, g4) = out
    assert np.array_equal(np.tile(f1, (1, 1, 1, rep)), f4)
    assert abs(l1 - l4) <= 1e-6 * abs(l1)
    assert np.linalg.norm(g1 - g4) <= 3e-4 * np.linalg.norm(g1)
