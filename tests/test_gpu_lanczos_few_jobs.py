"""The job table of the ground-state Lanczos takes its wide form from fewer states on
where each sector has an SM to itself: a sector's energy is the same bits alone (wide)
and in a table of many (narrow), on both sides of both limits."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,up,dn", [(2, 3, 3, 3), (7, 1, 2, 3), (7, 1, 3, 3), (2, 4, 3, 3), (3, 3, 4, 3), (3, 3, 5, 4),
                                         (16, 1, 2, 2), (10, 1, 4, 3)])
def test_one_sector_alone_and_among_many(qed, fresh, nx, ny, up, dn):
    prob = W.hubbard_cluster(nx, ny, tp=0.3 if min(nx, ny) > 1 else None, U=5.0, mu=2.1, M=0.1)
    prob.sectors = f"R0:N{up + dn}:S{up - dn}"
    small = W.hubbard_cluster(2, 2, U=4.0, mu=1.0)

    def load(p):
        suffix, label = fresh()
        qed.load_problem(p, label, model_name="few" + suffix, fmt="F")
        return label

    alone = float(qed.ground_state_solve(load(prob))[0])
    for many in (147, 148, 200):  # 148 jobs, 149, and more
        E = qed.ground_state_solve_batch([load(prob)] + [load(small) for _ in range(many)])
        assert float(E[0]) == alone
