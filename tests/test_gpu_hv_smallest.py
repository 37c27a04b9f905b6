"""The one-launch form of H x (csrc/hv_fused.cu) on the smallest sectors, against the
two-pass kernels (hv_variant bit 8 turns it off): one state, one string of either spin,
no hops, fewer strings than a warp has lanes. At most 40 terms per state in FP64: 40
eps sum |terms| stays below 1e-13 of the largest."""
import pytest
import torch

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (2, 1, 1, 1), (2, 1, 2, 1), (2, 2, 0, 0), (2, 2, 4, 4), (2, 2, 0, 2), (2, 2, 3, 4), (2, 2, 2, 2), (8, 1, 1, 0),
    (8, 1, 0, 3), (8, 1, 8, 4), (2, 3, 1, 2), (2, 4, 2, 1), (9, 1, 1, 4), (9, 1, 4, 1), (7, 1, 3, 2), (12, 1, 3, 0),
    (12, 1, 0, 3), (10, 1, 5, 0), (8, 1, 3, 1), (2, 5, 1, 2)])
@pytest.mark.parametrize("M", [None, 0.3])
def test_smallest_sectors_match_two_pass_kernels(qed, fresh, shape, M):
    nx, ny, up, dn = shape
    prob = W.hubbard_cluster(nx, ny, tp=0.3 if min(nx, ny) > 1 else None, U=5.0, mu=2.2, M=M)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="least" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    x = torch.randn(H.dim, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(9))
    out = []
    try:
        for v in (2, 10):
            qed.set_global_parameter("hv_variant", v)
            whole = torch.full((H.dim + 1,), float("nan"), dtype=torch.float64, device="cuda")
            d = torch.zeros(3, dtype=torch.float64, device="cuda")
            H.apply_dots_device(x.data_ptr(), whole.data_ptr(), d.data_ptr())
            torch.cuda.synchronize()
            assert torch.isnan(whole[-1])
            y = torch.full_like(x, float("nan"))
            H.apply_device(x.data_ptr(), y.data_ptr())
            torch.cuda.synchronize()
            assert torch.equal(y, whole[:-1])
            out.append((y, d))
    finally:
        qed.set_global_parameter("hv_variant", 2)
    (y, d), (r, e) = out
    scale = max(float(r.abs().max()), 1e-300)
    assert float((y - r).abs().max()) <= 1e-13 * scale
    assert float((d - e).abs().max()) <= 1e-12 * max(float(e.abs().max()), scale ** 2)
