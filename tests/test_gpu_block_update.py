"""The block recurrence's kernels (csrc/block.cu, k_blhv, k_block_chol) at every
block size class, in sectors of even and of odd dimension, against the one-vector form
of the band recurrence. Both end at the same residual of the band (1e-5 of a weight's
root, second order in G): G agrees to 1e-7 well away from the real axis."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def block(qed):
    def form(min_p):
        qed.set_global_parameter("block_lanczos_min_p", min_p)
        qed.set_global_parameter("block_lanczos_min_dim", 64)

    yield form
    qed.set_global_parameter("block_lanczos_min_p", 4)
    qed.set_global_parameter("block_lanczos_min_dim", 200)


# sites (the block size), up, down
@pytest.mark.parametrize("n,up,dn", [(3, 1, 1), (4, 2, 2), (5, 2, 2), (7, 3, 3), (8, 2, 3), (9, 2, 2), (10, 3, 2),
                                     (11, 1, 2), (12, 2, 2), (13, 2, 1), (16, 1, 1)])
def test_block_form_matches_band_form(qed, fresh, block, n, up, dn):
    prob = W.hubbard_cluster(n, 1, U=4.0, mu=1.7, M=0.0)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    z = 1j * np.linspace(0.5, 8.0, 6) + 0.3
    G = []
    for min_p in (2, 99):
        block(min_p)
        suffix, label = fresh()
        qed.load_problem(prob, label, model_name="blk" + suffix, fmt="F")
        G.append(np.asarray(qed.Green_function(z, label=label)))
    assert np.isfinite(G[0]).all()
    assert np.abs(G[0] - G[1]).max() <= 1e-7 * np.abs(G[1]).max()
