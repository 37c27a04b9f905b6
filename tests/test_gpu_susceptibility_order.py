"""The start vector O psi of a susceptibility's recurrence keeps the order of its sums
(HvOperator::keep_order), as the recurrence itself does: the same poles, bit for bit,
with the one-launch form of H x on and off (hv_variant bit 8)."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(8, 1), (2, 4), (3, 3)])
def test_susceptibility_poles_do_not_depend_on_the_form(qed, fresh, nx, ny):
    prob = W.hubbard_cluster(nx, ny, tp=0.3 if ny > 1 else None, U=5.0, mu=2.2, M=0.2)
    n = prob.n_sites
    # hops over several distances, so that the sums have terms to exchange
    prob.operators["P"] = ("one-body", [(i, j, 0.1 + 0.17 * i + 0.05 * j) for i in range(n) for j in range(i + 1, n)]
                           + [(i + n, j + n, 0.2 + 0.11 * j) for i in range(n) for j in range(i + 1, n)])
    prob.params["P"] = 1e-3
    res = []
    try:
        for v in (2, 10):
            qed.set_global_parameter("hv_variant", v)
            suffix, label = fresh()
            qed.load_problem(prob, label, model_name="sus" + suffix, fmt="F")
            qed.ground_state_solve(label)
            w = np.linspace(0.1, 4.0, 9) + 0.1j
            res.append((np.asarray(qed.susceptibility_poles("P", label)), np.asarray(qed.susceptibility("P", w, label))))
    finally:
        qed.set_global_parameter("hv_variant", 2)
    assert np.array_equal(res[0][0], res[1][0])
    assert np.array_equal(res[0][1], res[1][1])
