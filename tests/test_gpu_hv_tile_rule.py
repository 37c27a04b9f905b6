"""Which sectors take the tiled H x: not those whose tiles leave the SMs uneven or, with
rows of odd length, whose vectors leave L2, where the two-pass and staged kernels are
faster. Those then give the bits of the kernels that hv_variant 8 leaves; the tiled form
adds in another order."""
import pytest
import torch

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,up,dn,tiled", [
    (3, 5, 4, 4, False), (3, 5, 5, 4, False), (3, 5, 4, 5, False), (14, 1, 6, 7, False),
    (14, 1, 6, 5, True), (14, 1, 5, 4, True), (14, 1, 4, 4, True), (2, 7, 7, 7, True), (13, 1, 6, 6, True)])
def test_form_of_the_product(qed, fresh, nx, ny, up, dn, tiled):
    prob = W.hubbard_cluster(nx, ny, tp=0.3 if ny > 1 else None, U=5.0, mu=2.2, M=0.2)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="rule" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    x = torch.randn(H.dim, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    out = []
    try:
        for v in (2, 10):
            qed.set_global_parameter("hv_variant", v)
            y = torch.full_like(x, float("nan"))
            H.apply_device(x.data_ptr(), y.data_ptr())
            torch.cuda.synchronize()
            out.append(y)
    finally:
        qed.set_global_parameter("hv_variant", 2)
    assert torch.equal(*out) != tiled
    assert float((out[0] - out[1]).abs().max()) <= 1e-13 * float(out[1].abs().max())
