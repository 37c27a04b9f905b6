"""The job table of the ground-state Lanczos (k_lanczos_jobs): sectors on both sides
of the wide form's limit against the whole-GPU recurrence, and a batch whose next
chunk is launched ahead of the tests against the same clusters one by one. Energies
are those of a Ritz value with a residual of 1e-9, quadratic in it: 1e-11 covers the
different orders of sums; the batch has the same arithmetic and the same bits."""
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,up,dn", [(9, 4, 4), (9, 4, 5), (10, 4, 3), (10, 3, 6), (10, 5, 4), (10, 5, 5), (13, 2, 6)])
def test_wide_form_matches_whole_gpu(qed, fresh, n, up, dn):
    prob = W.hubbard_cluster(n, 1, U=4.0, mu=1.9, M=0.1)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    E = []
    try:
        for limit in (1 << 18, 16):
            qed.set_global_parameter("lanczos_job_max_dim", limit)
            suffix, label = fresh()
            qed.load_problem(prob, label, model_name="job" + suffix, fmt="F")
            E.append(qed.ground_state_solve(label)[0])
    finally:
        qed.set_global_parameter("lanczos_job_max_dim", 65536)
    assert abs(E[0] - E[1]) <= 1e-11 * abs(E[1])


def test_batch_of_many_sectors_is_each_cluster_alone(qed, fresh):
    probs = W.random_batch(24, seed=5)
    E = []
    for batch in (True, False):
        labels = []
        for prob in probs:
            suffix, label = fresh()
            qed.load_problem(prob, label, model_name="jobs" + suffix, fmt="F")
            labels.append(label)
        if batch:
            E.append([float(e) for e in qed.ground_state_solve_batch(labels)])
        else:
            E.append([float(qed.ground_state_solve(x)[0]) for x in labels])
    assert E[0] == E[1]
