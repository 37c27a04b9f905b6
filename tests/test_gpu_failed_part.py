"""A solve whose Q-matrix parts fail (here by the host's check of the projected
eigenvalues' gap) reports that error, as the parts taken one after the other do, and
leaves nothing that disturbs the solves after it."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu
Z = 1j * np.linspace(0.1, 5.0, 7)


def _load(qed, fresh, prob):
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="badpart" + suffix, fmt="F")
    return label


def test_error_of_a_part_and_the_solve_after_it(qed, fresh):
    rng = np.random.default_rng(6)
    prob = W.plaquette_bath(rng.uniform(-2, 2, 8), rng.uniform(0.1, 1, 8), U=6.0)
    ok = _load(qed, fresh, prob)
    qed.Green_function_solve_batch([ok])
    want = np.asarray(qed.Green_function(Z, label=ok))
    for _ in range(3):
        x = _load(qed, fresh, prob)
        qed.ground_state_solve(x)
        old = qed.get_global_double("band_lanczos_minimum_gap")
        qed.set_global_parameter("band_lanczos_minimum_gap", 1e3)
        qed.set_global_parameter("no_degenerate_BL", True)
        try:
            with pytest.raises(qed.QEDError, match="gap between the first two eigenvalues"):
                qed.Green_function_solve(x)
        finally:
            qed.set_global_parameter("no_degenerate_BL", False)
            qed.set_global_parameter("band_lanczos_minimum_gap", old)
        qed.Green_function_solve(x)  # the same instance, now without the check
        assert np.abs(np.asarray(qed.Green_function(Z, label=x)) - want).max() <= 1e-13 * np.abs(want).max()
        qed.erase_model_instance(x)
