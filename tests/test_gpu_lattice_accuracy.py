"""Rounding of the self-energy functional's integrand (csrc/lattice.cu) in its mean over
the wavevectors, where V G is small against 1 (high frequencies): against sums in 80
bits from the same G."""
import numpy as np
import pytest

from tests.test_gpu_lattice_sums import _loaded_instance

pytestmark = pytest.mark.gpu


def _log_det(A):
    """log |det| of a stack of matrices, in the precision of its input."""
    A, ar = A.copy(), np.arange(len(A))
    out = np.zeros(len(A), np.longdouble)
    for j in range(A.shape[1]):
        p = j + np.abs(A[:, j:, j]).argmax(1)
        A[ar, p], A[ar, j] = A[ar, j].copy(), A[ar, p].copy()
        out += np.log(np.abs(A[:, j, j]))
        A[:, j + 1:, j + 1:] -= (A[:, j + 1:, j] / A[:, j, j][:, None])[:, :, None] * A[:, j, None, j + 1:]
    return out


@pytest.mark.parametrize("n", [4, 10, 16])
def test_rounding_averages_out_over_the_wavevectors(qed, fresh, n):
    rng = np.random.default_rng(n)
    label, _ = _loaded_instance(qed, fresh, n, rng)
    w = np.linspace(150.0, 400.0, 24)
    G = np.asarray(qed.Green_function(1j * w, label=label))  # the G that the sums use
    V0 = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    side = 64
    # every row has elements whose phases change with either direction
    r = [i for i in range(n) for _ in range(2)]
    c = [int(x) for x in rng.integers(0, n, 2 * n)]
    R = [(1, int(rng.integers(1, 4)), 0) if i % 2 else (int(rng.integers(1, 4)), -1, 0) for i in range(2 * n)]
    v = [complex(*rng.standard_normal(2)) for _ in range(2 * n)]
    got = qed.sef_integrand_grid(V0, r, c, R, v, w, (side, side), label=label)
    kx, ky = (a.ravel() for a in np.meshgrid(np.arange(side), np.arange(side), indexing="ij"))
    pi = 4 * np.arctan(np.longdouble(1))
    V = np.broadcast_to(V0.astype(np.clongdouble), (side * side, n, n)).copy()
    for a, b, x, f in zip(r, c, R, v):
        ph = 2 * pi * ((kx * x[0] + ky * x[1]) % side).astype(np.longdouble) / side
        V[:, a, b] += np.clongdouble(f) * (np.cos(ph) + 1j * np.sin(ph))
    err = []
    for i in range(len(w)):
        A = np.zeros_like(V)
        for m in range(n):
            A += V[:, :, m, None] * G[i].astype(np.clongdouble)[None, m, None, :]
        err.append(float(np.longdouble(got[i]) - _log_det(A - np.eye(n)).mean()))
    # a matrix's value carries a few roundings of numbers next to 1 per row, 4 eps
    # sqrt(n) in all (eps = 2^-53); independent from one wavevector to the next, their
    # mean is 4 eps sqrt(n / K). Twice that for the root mean square over frequencies.
    # What all wavevectors share is relative to V G, 1e-2 here: below 0.1 eps sqrt(n).
    bound = 2.0 ** -53 * np.sqrt(n) * (8 / side + 0.1)
    assert np.sqrt(np.mean(np.square(err))) < bound, (np.sqrt(np.mean(np.square(err))), bound)
