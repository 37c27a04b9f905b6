"""The packed matrix of the symmetry-adapted basis in the recurrences (k_packed, with
each of its epilogues) adds every row and every reduction in the order of the CSR
kernels: energy, ground-state vector and G are the same bits with the matrix as CSR
(mixed_variant bit 1) and with the codes apart from the columns (bit 2). Sectors on
both sides of the rule for the warps per slice (14,208 states), dimensions that are no
multiple of 32."""
import numpy as np
import pytest

from tests.helpers import c2v_golden, c2v_problem
from tests.test_gpu_mixed_packed import _chain, _ladder

pytestmark = pytest.mark.gpu
Z = 1j * np.array([0.1, 0.7, 3.0])


@pytest.mark.parametrize("case,sector,min_p", [
    ("record", None, None), ("2x4", "R0:N8:S0", None), ("2x5", "R0:N10:S0", None), ("2x5", "R2:N9:S1", 99),
    ("chain9", "R1:N9:S1", None), ("2x6", "R0:N11:S1", None)])
def test_recurrences_are_the_same_bits_in_every_form(qed, fresh, case, sector, min_p):
    prob = (c2v_problem(c2v_golden(), True) if case == "record" else _chain(9) if case == "chain9"
            else _ladder(*map(int, case.split("x"))))
    if sector:
        prob.sectors = sector
    res = []
    try:
        if min_p:  # the band recurrence instead of the block one
            qed.set_global_parameter("block_lanczos_min_p", min_p)
        for v in (0, 1, 2):
            qed.set_global_parameter("mixed_variant", v)
            suffix, label = fresh()
            qed.load_problem(prob, label, model_name="order" + suffix)
            e, _ = qed.ground_state_solve(label)
            psi = np.asarray(qed.ground_state_vector(label))
            res.append((e, psi, np.asarray(qed.Green_function(Z, label=label))))
    finally:
        qed.set_global_parameter("mixed_variant", 0)
        qed.set_global_parameter("block_lanczos_min_p", 4)
    for e, psi, g in res[1:]:
        assert e == res[0][0]
        assert np.array_equal(psi, res[0][1])
        assert np.array_equal(g, res[0][2])


def test_wide_codes_give_the_same_product(qed, fresh):
    """k_packed_free with both layouts: the same sums in the same order."""
    import torch

    from tests.test_gpu_mixed_packed import _apply
    for case, sec in (("2x4", "R1:N8:S0"), ("2x5", "R0:N9:S1"), ("2x6", "R0:N12:S0")):
        suffix, label = fresh()
        qed.load_problem(_ladder(*map(int, case.split("x"))), label, model_name="wide" + suffix)
        H = qed.MixedHamiltonian(label, sec)
        qed.set_global_parameter("mixed_variant", 2)
        try:
            V = qed.MixedHamiltonian(label, sec)
        finally:
            qed.set_global_parameter("mixed_variant", 0)
        x = torch.randn(H.dim, dtype=torch.float64, device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(5))
        assert H.nnz == V.nnz and torch.equal(_apply(qed, H, x), _apply(qed, V, x)), case
