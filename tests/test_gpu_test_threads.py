"""The dense convergence tests that run beside a recurrence after a deflation share the
host's cores: a batch of 48 clusters, whose hole halves (90 states, six start vectors)
all go on for hundreds of steps after they have deflated, starts no more threads than
the library's pools have and one per core. Energies and G are those of each alone."""
import os
import threading

import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _threads():
    return len(os.listdir("/proc/self/task"))


def test_threads_of_a_batch_are_bounded(qed, fresh):
    rng = np.random.default_rng(8)
    probs = []
    for _ in range(48):
        p = W.hubbard_cluster(2, 3, U=float(rng.uniform(2, 12)), mu=float(rng.uniform(0.1, 2)), M=0.1)
        p.sectors = "R0:N4:S0"
        probs.append(p)

    def load(p):
        suffix, label = fresh()
        qed.load_problem(p, label, model_name="thr" + suffix, fmt="F")
        return label

    z = np.array([0.1j, 0.9j])
    want = []
    for p in probs[:4]:
        x = load(p)
        qed.Green_function_solve(x)
        want.append(np.asarray(qed.Green_function(z, label=x)))
    before, most, done = _threads(), 0, threading.Event()

    def watch():
        nonlocal most
        while not done.is_set():
            most = max(most, _threads())

    w = threading.Thread(target=watch)
    w.start()
    labels = [load(p) for p in probs]
    qed.Green_function_solve_batch(labels, threads=64)
    done.set()
    w.join()
    cores = os.cpu_count()
    pools = 63 + min(64, cores) - 1  # batch tasks, Ritz tests
    assert most <= before + 1 + pools + cores
    for x, g in zip(labels, want):
        assert np.abs(np.asarray(qed.Green_function(z, label=x)) - g).max() <= 1e-12 * np.abs(g).max()
