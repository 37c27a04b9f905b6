"""Calls leave no kernel behind that reads what the caller may free.

The job table of the ground-state Lanczos launches a chunk ahead of the tests of the
one before; equal clusters stop in the same chunk, so the one ahead is then of no use
and still under way. With a sector above the table's limit in the same batch the
table runs on another thread's stream than the one its sectors' arrays are freed on."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _uneven_u(nx, ny, seed):
    """A cluster with an interaction of its own on every site."""
    p = W.hubbard_cluster(nx, ny, U=4.0, mu=1.7, M=0.2)
    n = p.n_sites
    u = np.random.default_rng(seed).uniform(0.5, 1.5, n)
    p.operators["U"] = ("interaction", [(i, i + n, float(u[i])) for i in range(n)])
    return p


def test_equal_clusters_freed_after_their_batch(qed, fresh):
    small, large = _uneven_u(2, 2, 1), _uneven_u(2, 4, 2)

    def load(prob):
        suffix, label = fresh()
        qed.load_problem(prob, label, model_name="inflight" + suffix, fmt="F")
        return label

    qed.set_global_parameter("lanczos_job_max_dim", 64)  # 36 states each, 4900 the large one
    try:
        want = [float(qed.ground_state_solve(load(p))[0]) for p in (small, large)]
        for _ in range(4):
            labels = [load(small) for _ in range(300)] + [load(large)]
            got = [float(e) for e in qed.ground_state_solve_batch(labels)]
            for x in labels:
                qed.erase_model_instance(x)
            assert got[:-1] == [want[0]] * 300  # the same arithmetic, the same bits
            assert abs(got[-1] - want[1]) <= 1e-11 * abs(want[1])
    finally:
        qed.set_global_parameter("lanczos_job_max_dim", 65536)
