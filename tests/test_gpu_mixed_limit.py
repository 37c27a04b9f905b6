"""mixed_csr_max_gb is the memory of the matrix as it is stored: a limit between the
packed form's 4 B per slot and CSR's 12 B per entry keeps the packed matrix, one below
both has every product recompute its entries."""
import pytest
import torch

from tests.test_gpu_mixed_packed import _apply, _ladder

pytestmark = pytest.mark.gpu


def test_limit_is_the_stored_size(qed, fresh):
    suffix, label = fresh()
    qed.load_problem(_ladder(2, 6), label, model_name="lim" + suffix)
    sec = "R0:N12:S0"

    def product(**options):
        old = {k: qed.get_global_double(k) if k == "mixed_csr_max_gb" else False for k in options}
        for k, v in options.items():
            qed.set_global_parameter(k, v)
        try:
            H = qed.MixedHamiltonian(label, sec)
        finally:
            for k, v in old.items():
                qed.set_global_parameter(k, v)
        x = torch.randn(H.dim, dtype=torch.float64, device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(3))
        return H.nnz, _apply(qed, H, x)

    nnz, stored = product()
    _, recomputed = product(mixed_on_the_fly=True)
    assert not torch.equal(stored, recomputed)  # the two forms add in another order
    assert torch.equal(product(mixed_csr_max_gb=8e-9 * nnz)[1], stored)  # rows padded by less than their length
    assert torch.equal(product(mixed_csr_max_gb=2e-9 * nnz)[1], recomputed)
