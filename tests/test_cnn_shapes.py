"""The network's kernels where the work split changes: x chunks of the
convolutions chosen by the grid (one plane a CTA, several with a remainder),
chunks of the weight gradient with a remainder of one plane and its tap groups
spread over one or several CTAs.  The bars are those of the other network
tests: BF16 activations and weights (2^-9 relative each) through five layers,
1e-2 of the output's and 3e-2 of a gradient's L2 norm, 1e-3 of the loss."""
import numpy as np
import pytest

from oracle import cnn_oracle as O


def rel_l2(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-300))


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(2, 4, 32), (33, 4, 32), (37, 8, 64), (33, 32, 64)])
def test_forward_and_gradients_match_oracle(cuda_lib, dims):
    from cgli_fu_flow_b200.cnn import Network
    rng = np.random.default_rng(11)
    W, b = O.unpack(O.init_params(11))
    W[-1] = rng.uniform(-0.05, 0.05, size=W[-1].shape)
    b = [rng.uniform(-0.1, 0.1, size=bb.shape) for bb in b]
    theta = O.pack(W, b)
    x0, target = rng.standard_normal((15,) + dims), rng.standard_normal((5,) + dims)
    net = Network(*dims)
    net.set_params(theta)
    assert rel_l2(net.forward(x0), O.forward(theta.astype(np.float64), x0)) <= 1e-2
    loss, g = net.loss_grad(x0, target)
    lo, go, _ = O.loss_and_grad(theta.astype(np.float64), x0, target)
    assert abs(loss - lo) <= 1e-3 * lo
    off = 0
    for ci, co in zip(O.CIN, O.COUT):
        n = 27 * ci * co
        assert rel_l2(g[off:off + n], go[off:off + n]) <= 3e-2
        assert rel_l2(g[off + n:off + n + co], go[off + n:off + n + co]) <= 3e-2
        off += n + co
