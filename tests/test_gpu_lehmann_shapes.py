"""G(z) of a Lehmann representation over the shapes that choose the CTAs' threads and the
poles' slices (launch_qmatrix_gf): few and many frequencies, one pole to several
shared-memory chunks, one orbital to more pairs than threads. Sums of at most 3000
terms: error below 3000 eps sum |terms| < 1e-11 here; random signs leave far less."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 15, 16, 31, 32])
@pytest.mark.parametrize("M,nz", [(1, 1), (15, 3), (16, 296), (33, 297), (1500, 40), (64, 1185), (3000, 2)])
def test_green_function_of_poles_over_shapes(qed, fresh, n, M, nz):
    rng = np.random.default_rng(100 * n + M)
    suffix, label = fresh()
    name = "gfs" + suffix
    qed.new_model(name, n)
    qed.new_operator(name, "mu", "one-body", [(i, i, -1.0) for i in range(2 * n)])
    qed.new_operator(name, "U", "interaction", [(i, i + n, 1.0) for i in range(n)])
    qed.new_model_instance(name, {"mu": 1.0, "U": 2.0}, f"R0:N{n}:S{n % 2}", label)
    e, v = rng.uniform(-4, 4, M), rng.standard_normal((n, M)) / np.sqrt(M)
    dp = C.POINTER(C.c_double)
    lib, i = qed.lib(), C.c_int()
    vt = np.ascontiguousarray(v.T)
    qed._check(lib.qed_instance_load_begin(label, -1.0, 0, 0))
    for w in (0.75, 0.25):  # two states: the second one's matrices are added
        qed._check(lib.qed_instance_load_state(label, b"R0:N0:S0", -1.0, w, C.byref(i)))
        qed._check(lib.qed_instance_load_qmatrix(label, i.value, 0, n, M, e.ctypes.data_as(dp), vt.ctypes.data_as(dp)))
    qed._check(lib.qed_instance_load_end(label))
    z = rng.uniform(-4, 4, nz) + 1j * rng.uniform(0.2, 2, nz)
    got = qed.Green_function(z, label=label)
    ref = 2 * np.einsum("am,zm,bm->zab", v, 1.0 / (z[:, None] - e[None, :]), v, optimize=True)
    assert np.max(np.abs(got - ref)) < 1e-11 * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("n,M", [(1, 40), (4, 360), (10, 480), (16, 130)])
def test_a_frequency_is_the_same_in_any_call(qed, fresh, n, M):
    from tests.test_gpu_lattice_sums import _loaded_instance
    label, _ = _loaded_instance(qed, fresh, n, np.random.default_rng(n), M=M)
    z = 1j * np.linspace(0.1, 30.0, 3000)
    G = qed.Green_function(z, label=label)
    for m in (1, 70, 500):
        assert np.array_equal(qed.Green_function(z[:m], label=label), G[:m]), m
