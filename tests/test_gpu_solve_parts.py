"""A single solve forms the parts of its Q-matrices (hole and electron, irreps of a
point group) at the same time; a batch call takes them as tasks. Both have the same
arithmetic: energies and G agree to the last digits, also from several host threads
at once (where all but one solve form their parts one after the other)."""
import threading

import numpy as np
import pytest

from pyqcm_b200 import workloads as W
from tests.helpers import c2v_golden, c2v_problem

pytestmark = pytest.mark.gpu
Z = 1j * np.linspace(0.1, 5.0, 7)


def _ladder(n):
    p = W.hubbard_cluster(2, n, tp=0.3, U=5.0, mu=2.1)
    s = lambda x, y: 1 + x + 2 * y
    p.generators = [[s(1 - x, y) for y in range(n) for x in range(2)]]
    p.sectors = f"R0:N{2 * n}:S0/R1:N{2 * n}:S0"
    return p


def _problems():
    rng = np.random.default_rng(4)
    yield "bath", W.plaquette_bath(rng.uniform(-2, 2, 8), rng.uniform(0.1, 1, 8), U=6.0)
    yield "spins", W.hubbard_cluster(3, 2, U=5.0, mu=2.2, M=0.3)
    yield "ladder", _ladder(4)
    yield "c2v", c2v_problem(c2v_golden(), True)


def _load(qed, fresh, prob):
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="part" + suffix)
    return label


def _g(qed, label):
    return np.asarray(qed.Green_function(Z, label=label))


@pytest.mark.parametrize("name", ["bath", "spins", "ladder", "c2v"])
def test_parts_at_once_match_batch_and_threads(qed, fresh, name):
    prob = dict(_problems())[name]
    labels = [_load(qed, fresh, prob) for _ in range(6)]
    qed.Green_function_solve_batch(labels[:1])
    want = _g(qed, labels[0])
    qed.Green_function_solve(labels[1])
    assert np.abs(_g(qed, labels[1]) - want).max() <= 1e-13 * np.abs(want).max()
    out, err = {}, []

    def solve(x):
        try:
            qed.Green_function_solve(x)
            out[x] = _g(qed, x)
        except Exception as e:  # shown below
            err.append(e)

    ts = [threading.Thread(target=solve, args=(x,)) for x in labels[2:]]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not err
    for x in labels[2:]:
        assert np.abs(out[x] - want).max() <= 1e-13 * np.abs(want).max()
