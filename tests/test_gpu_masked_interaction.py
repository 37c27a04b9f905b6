"""One interaction on some of the sites only, through every form of H x: staged (which
takes the sites one by one), two-pass, tiled and the host entry, against each other and
at the diagonal. At most 60 terms per state in FP64: 60 eps sum |terms| stays below
1e-13 of the largest."""
import numpy as np
import pytest
import torch

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,up,dn,M", [(2, 6, 6, 6, None), (2, 6, 6, 5, 0.3), (3, 5, 4, 4, None)])
def test_masked_interaction_in_every_form(qed, fresh, nx, ny, up, dn, M):
    prob = W.hubbard_cluster(nx, ny, tp=0.3, U=5.0, mu=2.2, M=M)
    n, sites = prob.n_sites, [0, 2, 3, 7, 10]
    prob.operators["U"] = ("interaction", [(i, i + n, 1.0) for i in sites])
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="mask" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    x = torch.randn(H.dim, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    out = []
    try:
        for v in (10, 14, 2):  # staged where it applies; two passes; tiled or one launch
            qed.set_global_parameter("hv_variant", v)
            y = torch.full_like(x, float("nan"))
            H.apply_device(x.data_ptr(), y.data_ptr())
            torch.cuda.synchronize()
            out.append(y.cpu().numpy())
    finally:
        qed.set_global_parameter("hv_variant", 2)
    host = np.zeros(H.dim)
    H.mult_add(x.cpu().numpy(), host)
    scale = np.abs(out[0]).max()
    for y in out[1:] + [host]:
        assert np.abs(y - out[0]).max() <= 1e-13 * scale
    b_up, b_dn = qed.halfbasis(n, up).astype(np.int64), qed.halfbasis(n, dn).astype(np.int64)
    occ = lambda s: np.stack([(s >> i) & 1 for i in range(n)], 1).astype(float)
    U = np.zeros(n)
    U[sites] = 5.0
    field = np.array([0.0 if M is None else M * (1 if (i % nx + i // nx) % 2 == 0 else -1) for i in range(n)])
    want = (occ(b_dn) * U) @ occ(b_up).T + (occ(b_up) @ (field - 2.2))[None] + (occ(b_dn) @ (-field - 2.2))[:, None]
    assert np.abs(H.diag().reshape(want.shape) - want).max() < 1e-12
