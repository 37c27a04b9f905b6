"""The surrogate network where its parameters are more than 148 x 16 x 256 (606,208):
the optimiser and the BF16 copy of the weights reach every one of them. The first step
of Adam (Kingma & Ba 2015) moves a weight by -lr g / (|g| + eps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [544, 560, 768])  # 601,664, 637,344 and 1,190,480 parameters or so: both sides
def test_first_step_moves_every_weight(width):
    from pyqcm_b200 import surrogate as S
    net = S.MLP(n_in=4, width=width, seed=5)
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (64, 4)).astype(np.float32)
    t = np.sin(2 * x[:, 0] + x[:, 1]).astype(np.float32)
    before = net.get_params()
    g, _ = net.gradients(x, t)
    lr = 1e-3
    net.train(x, t, epochs=1, batch=64, lr=lr, seed=0)
    moved = net.get_params() - before
    # the training pass takes the rows in another order: its gradient differs by the
    # rounding of 64-term sums, less than 1e-3 of one that is above 1e-3 of the largest
    clear = np.abs(g) > 1e-3 * np.abs(g).max()
    assert np.count_nonzero(clear) > 0.1 * net.n_params
    assert np.max(np.abs(moved[clear] + lr * np.sign(g[clear]))) < 1e-2 * lr
    assert net.n_params - 1 - np.nonzero(clear)[0][-1] < 2 * width  # to the end of the vector


@pytest.mark.parametrize("width", [544, 768])
def test_forward_uses_every_weight_that_was_set(width):
    from oracle import mlp_port as port
    from pyqcm_b200 import surrogate as S
    net = S.MLP(n_in=4, width=width, seed=5)
    p = net.get_params()
    net.set_params(np.where(p != 0, p[::-1] * 0.5 + p, p).astype(np.float32))
    x = np.random.default_rng(0).uniform(-1, 1, (50, 4)).astype(np.float32)
    want, _ = port.forward(net.blocks(), x, 4)
    # BF16 activations: a rounding that lands differently moves an output by 2^-9 of a term
    assert np.max(np.abs(net(x) - want)) < 2e-3 * max(1.0, np.max(np.abs(want)))
