"""The wavevector sums with many elements per entry of V(k) (long-range hops), which are
stored per wavevector beforehand (csrc/lattice.cu), and with few, on both sides of the
rule (three elements a row on average): against numpy. Entries of one and of many
elements, rows without any, grids whose directions come in any order and of more points
than the phase table holds."""
import numpy as np
import pytest

from tests.test_gpu_lattice_sums import TOL, _V, _loaded_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk,nel", [(1, (4, 3, 2), 3), (1, (4, 3, 2), 4), (2, (9, 1, 1), 40), (3, (5, 4, 3), 9),
                                      (3, (5, 4, 3), 10), (4, (1, 7, 5), 100), (5, (6, 6, 1), 200), (6, (400, 1, 1), 60),
                                      (10, (3, 5, 2), 400), (13, (2, 2, 2), 60), (16, (3, 2, 1), 600)])
def test_many_elements_match_numpy(qed, fresh, n, nk, nel):
    rng = np.random.default_rng(1000 * n + nel)
    label, G = _loaded_instance(qed, fresh, n, rng)
    rows = max(1, n - 1)  # the last row has none (n > 1)
    r = [int(x) for x in rng.integers(0, rows, nel)]
    c = [int(x) for x in rng.integers(0, n, nel)]
    R = [tuple(int(x) for x in rng.integers(-7, 8, 3)) for _ in range(nel)]
    v = [complex(*rng.standard_normal(2)) / np.sqrt(nel / n) for _ in range(nel)]
    w = np.array([0.2, 2.1])
    V0 = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    grid = [(i / nk[0], j / nk[1], l / nk[2]) for i in range(nk[0]) for j in range(nk[1]) for l in range(nk[2])]
    got = qed.sef_integrand_grid(V0[0], r, c, R, v, w, nk, label=label)
    for i in range(2):
        ref = np.mean([np.linalg.slogdet(_V(V0[0], (r, c, R, v), k) @ G(w[i]) - np.eye(n))[1] for k in grid])
        assert abs(got[i] - ref) <= TOL * max(1.0, abs(ref)), i
    got = qed.cpt_projected_green_function(V0, r, c, R, v, w, nk, offset=0.5, label=label)
    for i in range(2):
        half = [tuple(x + 0.5 / m for x, m in zip(k, nk)) for k in grid]
        ref = np.mean([G(w[i]) @ np.linalg.inv(np.eye(n) - _V(V0[i], (r, c, R, v), k) @ G(w[i])) for k in half], axis=0)
        assert np.max(np.abs(got[i] - ref)) <= TOL * max(1.0, np.max(np.abs(ref))), i
