"""H x on vectors that start between two 16-byte boundaries, with rows of even length:
the two-pass kernels' 16-byte accesses are for aligned vectors only (hv_variant bit 8
turns the other forms off; bit 1 has the gathers cached in L2 only). Both sides sum at
most 60 terms per state in FP64: 60 eps sum |terms| stays below 1e-13 of the largest."""
import pytest
import torch

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 1, 4, 4), (2, 5, 5, 4), (2, 6, 6, 6), (2, 7, 7, 7)])  # the last: staged when aligned
@pytest.mark.parametrize("variant", [2, 10, 11])
def test_misaligned_vectors_with_even_rows(qed, fresh, shape, variant):
    nx, ny, up, dn = shape
    prob = W.hubbard_cluster(nx, ny, tp=0.3 if ny > 1 else None, U=5.0, mu=2.2, M=0.2)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="align" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    base = torch.randn(H.dim, dtype=torch.float64, device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(2))
    out = {}
    qed.set_global_parameter("hv_variant", variant)
    try:
        for ox, oy in ((0, 0), (1, 0), (0, 1), (1, 1)):
            x = torch.empty(H.dim + 2, dtype=torch.float64, device="cuda")[ox:ox + H.dim]
            x.copy_(base)
            whole = torch.full((H.dim + 2,), float("nan"), dtype=torch.float64, device="cuda")
            y = whole[oy:oy + H.dim]
            d = torch.zeros(3, dtype=torch.float64, device="cuda")
            assert (x.data_ptr() % 16 == 0) == (ox == 0)
            H.apply_dots_device(x.data_ptr(), y.data_ptr(), d.data_ptr())
            torch.cuda.synchronize()
            assert int(torch.isnan(whole).sum()) == 2  # nothing written beside y
            out[ox, oy] = (y, d)
    finally:
        qed.set_global_parameter("hv_variant", 2)
    y0, d0 = out[0, 0]
    for y, d in out.values():
        assert float((y - y0).abs().max()) <= 1e-13 * float(y0.abs().max())
        assert float((d - d0).abs().max()) <= 1e-12 * float(d0.abs().max())
