"""The wavevector sums on the GPU (csrc/lattice.cu) against numpy for every kind
of matrix dimension: matrices that fill a warp's lanes exactly (1, 2, 4, 8, 16)
and that leave some over, grids that end inside a warp's batch, several elements
in one row, none at all. Instances hold random Lehmann representations, so G is
known without a solve."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# |d log det A| and |dA^-1| / |A^-1| are at most about 10 n cond(A) 2^-53; the
# random matrices have cond(A) below 1e4, so 16 * 1e4 * 1.1e-15 = 2e-10, times a
# margin of 5.
TOL = 1e-9


def _loaded_instance(qed, fresh, n, rng, M=40):
    suffix, label = fresh()
    name = "latsum" + suffix
    qed.new_model(name, n)
    qed.new_operator(name, "mu", "one-body", [(i, i, -1.0) for i in range(2 * n)])
    qed.new_operator(name, "U", "interaction", [(i, i + n, 1.0) for i in range(n)])
    qed.new_model_instance(name, {"mu": 1.0, "U": 2.0}, f"R0:N{n}:S{n % 2}", label)
    e = np.concatenate([-rng.uniform(0.5, 5, M // 2), rng.uniform(0.5, 5, M // 2)])
    v = rng.standard_normal((n, M)) / np.sqrt(M)
    dp = C.POINTER(C.c_double)
    lib, i = qed.lib(), C.c_int()
    qed._check(lib.qed_instance_load_begin(label, -1.0, 0, 0))
    qed._check(lib.qed_instance_load_state(label, b"R0:N0:S0", -1.0, 1.0, C.byref(i)))
    vt = np.ascontiguousarray(v.T)
    qed._check(lib.qed_instance_load_qmatrix(label, 0, 0, n, M, e.ctypes.data_as(dp), vt.ctypes.data_as(dp)))
    qed._check(lib.qed_instance_load_end(label))
    return label, lambda w: np.einsum("am,m,bm->ab", v, 1.0 / (1j * w - e), v)


def _elements(n, rng, nel):
    r = [int(x) for x in rng.integers(0, n, nel)]
    c = [int(x) for x in rng.integers(0, n, nel)]
    R = [tuple(int(x) for x in rng.integers(-2, 3, 3)) for _ in range(nel)]
    v = [complex(*rng.standard_normal(2)) for _ in range(nel)]
    return r, c, R, v


def _V(V0, el, k):
    V = V0.copy()
    for r, c, R, v in zip(*el):
        V[r, c] += v * np.exp(2j * np.pi * np.dot(k, R))
    return V


@pytest.mark.parametrize("n,nk,nel", [(1, (3, 5, 1), 2), (2, (4, 4, 4), 5), (3, (7, 3, 1), 6), (4, (9, 11, 1), 9),
                                      (5, (33, 1, 1), 0), (7, (5, 5, 2), 30), (8, (6, 7, 1), 12), (9, (3, 3, 3), 20),
                                      (10, (13, 9, 1), 14), (11, (1, 1, 1), 5), (12, (2, 31, 1), 20),
                                      (13, (4, 3, 2), 17), (15, (5, 3, 1), 40), (16, (6, 5, 1), 33)])
def test_wavevector_sums_match_numpy(qed, fresh, n, nk, nel):
    rng = np.random.default_rng(100 * n + nel)
    label, G = _loaded_instance(qed, fresh, n, rng)
    el = _elements(n, rng, nel)
    w = np.array([0.1, 0.7, 3.0])
    V0 = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))
    grid = [(i / nk[0], j / nk[1], l / nk[2]) for i in range(nk[0]) for j in range(nk[1]) for l in range(nk[2])]
    got = qed.sef_integrand_grid(V0[0], *el, w, nk, label=label)
    for i in range(3):
        ref = np.mean([np.linalg.slogdet(_V(V0[0], el, k) @ G(w[i]) - np.eye(n))[1] for k in grid])
        assert abs(got[i] - ref) <= TOL * max(1.0, abs(ref)), (i, got[i], ref)
    got = qed.cpt_projected_green_function(V0, *el, w, nk, offset=0.5, label=label)
    for i in range(3):
        half = [tuple(x + 0.5 / m for x, m in zip(k, nk)) for k in grid]
        ref = np.mean([G(w[i]) @ np.linalg.inv(np.eye(n) - _V(V0[i], el, k) @ G(w[i])) for k in half], axis=0)
        assert np.max(np.abs(got[i] - ref)) <= TOL * max(1.0, np.max(np.abs(ref))), i


def test_singular_matrix_gives_minus_infinity(qed, fresh):
    """V G - 1 with a zero row (G = 1 / z for one site, V = z at one frequency):
    log 0, as the elimination of the previous kernel gave."""
    suffix, label = fresh()
    name = "latsing" + suffix
    qed.new_model(name, 1)
    qed.new_operator(name, "mu", "one-body", [(0, 0, -1.0), (1, 1, -1.0)])
    qed.new_operator(name, "U", "interaction", [(0, 1, 1.0)])
    qed.new_model_instance(name, {"mu": 1.0, "U": 2.0}, "R0:N1:S1", label)
    dp = C.POINTER(C.c_double)
    lib, i = qed.lib(), C.c_int()
    e, v = np.array([0.0]), np.array([1.0])
    qed._check(lib.qed_instance_load_begin(label, -1.0, 0, 0))
    qed._check(lib.qed_instance_load_state(label, b"R0:N0:S0", -1.0, 1.0, C.byref(i)))
    qed._check(lib.qed_instance_load_qmatrix(label, 0, 0, 1, 1, e.ctypes.data_as(dp), v.ctypes.data_as(dp)))
    qed._check(lib.qed_instance_load_end(label))
    out = qed.sef_integrand_grid(np.array([[2j]]), [], [], [], [], [2.0, 1.0], (2, 2), label=label)
    assert out[0] == -np.inf
    assert out[1] == 0.0  # |2i / i - 1| = 1


@pytest.mark.parametrize("n,M", [(1, 2), (1, 1), (2, 7), (4, 360), (10, 481), (16, 300), (31, 97), (32, 1)])
def test_green_function_of_poles(qed, fresh, n, M):
    """G(z) of a loaded Lehmann representation: one slice of poles and many, more
    pairs than threads (n = 32), several shared-memory chunks (n = 10, M = 481).
    Sums of at most 481 terms: error below 481 eps sum |terms| < 1e-12 here."""
    rng = np.random.default_rng(n + M)
    suffix, label = fresh()
    name = "gfp" + suffix
    qed.new_model(name, n)
    qed.new_operator(name, "mu", "one-body", [(i, i, -1.0) for i in range(2 * n)])
    qed.new_operator(name, "U", "interaction", [(i, i + n, 1.0) for i in range(n)])
    qed.new_model_instance(name, {"mu": 1.0, "U": 2.0}, f"R0:N{n}:S{n % 2}", label)
    e, v = rng.uniform(-4, 4, M), rng.standard_normal((n, M)) / np.sqrt(M)
    dp = C.POINTER(C.c_double)
    lib, i = qed.lib(), C.c_int()
    vt = np.ascontiguousarray(v.T)
    qed._check(lib.qed_instance_load_begin(label, -1.0, 0, 0))
    qed._check(lib.qed_instance_load_state(label, b"R0:N0:S0", -1.0, 1.0, C.byref(i)))
    qed._check(lib.qed_instance_load_qmatrix(label, 0, 0, n, M, e.ctypes.data_as(dp), vt.ctypes.data_as(dp)))
    qed._check(lib.qed_instance_load_end(label))
    z = np.array([0.3 + 0.4j, -2.0 + 0.5j, 0.9j])
    got = qed.Green_function(z, label=label)
    ref = np.einsum("am,zm,bm->zab", v, 1.0 / (z[:, None] - e[None, :]), v)
    assert np.max(np.abs(got - ref)) < 1e-12
