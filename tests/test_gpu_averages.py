"""Operator averages from the strings in one launch against numpy on the
ground-state vector: hops of both spins, density terms, bath orbitals,
interactions on some sites only."""
import numpy as np
import pytest

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _matrix(el, typ, n, up, dn):
    """The operator on the basis up + len(up) * dn (as the oracle's rules state it)."""
    D = len(up) * len(dn)
    M = np.zeros((D, D))
    iu, idn = {int(s): i for i, s in enumerate(up)}, {int(s): i for i, s in enumerate(dn)}
    for b, d in enumerate(dn):
        for a, u in enumerate(up):
            I, word = a + len(up) * b, int(u) | int(d) << n
            for r, c, v in el:
                if typ == "interaction" or r == c:
                    if word >> r & 1 and word >> c & 1:
                        M[I, I] += v
                    continue
                for x, y in ((r, c), (c, r)):  # c+_x c_y
                    if not word >> y & 1 or word >> x & 1:
                        continue
                    lo, hi = min(x, y), max(x, y)
                    sign = (-1) ** bin(word >> (lo + 1) & (1 << (hi - lo - 1)) - 1).count("1")
                    nw = word ^ 1 << x ^ 1 << y
                    M[I, iu[nw & (1 << n) - 1] + len(up) * idn[nw >> n]] += v * sign
    return M


@pytest.mark.parametrize("case", ["2x2", "2x3", "bath"])
def test_averages_match_numpy(qed, fresh, case):
    if case == "bath":
        rng = np.random.default_rng(2)
        prob = W.plaquette_bath(rng.uniform(-2, 2, 8), rng.uniform(0.2, 1, 8), U=5.0)
        nu, nd = 2, 1
    else:
        prob = W.hubbard_cluster(2, int(case[2]), tp=0.3, U=5.0, mu=2.1, M=0.2)
        nu, nd = (2, 1) if case == "2x2" else (3, 2)
    prob.sectors = f"R0:N{nu + nd}:S{nu - nd}"
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="ave" + suffix, fmt="F")
    qed.ground_state_solve(label)
    psi = qed.ground_state_vector(label)
    n = prob.n_orb
    up, dn = qed.halfbasis(n, nu), qed.halfbasis(n, nd)
    got = {name: (a, v) for name, a, v in qed.cluster_averages(label)}
    for name, (typ, el) in prob.operators.items():
        if name not in prob.params:
            continue
        O = _matrix(el, typ, n, up, dn)
        ave, var = psi @ O @ psi, np.sum((O @ psi) ** 2) - (psi @ O @ psi) ** 2
        # operators on cluster orbitals only are per site, "mu" counts particles
        cluster = all((i % n) < prob.n_sites for r, c, _ in el for i in (r, c))
        norm = (-1.0 if name == "mu" else 1.0) / prob.n_sites if cluster else 1.0
        a, v = got[name]
        # sums of at most 1e4 products of entries below 1
        assert abs(a - ave * norm) < 1e-11, name
        assert abs(v - var * norm * norm) < 1e-11, name
