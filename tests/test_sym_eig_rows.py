"""Eigenvalues and first rows of the eigenvectors of a symmetric matrix (sym_eig_rows,
pyqcm_b200/csrc/eigen.cpp), the projected eigensystem of a band recurrence after a
deflation: moments sum_k w_k^q Z_rk Z_sk = (A^q)_rs, and the eigenvalues, against
numpy. Host code, compiled here. Backward errors of a few n eps of the norm."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyqcm_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <vector>
#include "eigen.hpp"
int main() {
  int n, m;
  if (scanf("%d %d", &n, &m) != 2) return 1;
  std::vector<double> A((size_t)n * n), w, Z;
  for (auto &v : A) if (scanf("%lf", &v) != 1) return 1;
  if (!qed::sym_eig_rows(n, A, m, w, Z)) return 2;
  for (double v : w) printf("%.17g\n", v);
  for (double v : Z) printf("%.17g\n", v);
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("eig_rows")
    (d / "drv.cpp").write_text(DRIVER)
    exe = str(d / "drv")
    subprocess.run(["g++", "-O3", "-std=c++17", "-I", CSRC, str(d / "drv.cpp"), os.path.join(CSRC, "eigen.cpp"), "-o",
                    exe], check=True)
    return exe


@pytest.mark.parametrize("n,m,kind", [(1, 1, "full"), (2, 2, "full"), (3, 5, "full"), (7, 3, "full"), (40, 4, "band"),
                                      (90, 6, "full"), (200, 6, "band"), (60, 2, "blocks"), (33, 3, "zero")])
def test_moments_and_eigenvalues(driver, n, m, kind):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    if kind == "band":  # with a few spikes, as a deflated recurrence leaves them
        A = np.triu(np.tril(A, m), -m)
        A[5, 12:] = A[12:, 5] = 1e-8
    elif kind == "blocks":
        A[:n // 2, n // 2:] = 0
        A[n // 2:, :n // 2] = 0
    elif kind == "zero":
        A[:] = 0
    out = subprocess.run([driver], input=f"{n} {m}\n" + " ".join(f"{v:.17g}" for v in A.ravel()), capture_output=True,
                         text=True, check=True).stdout.split()
    v = np.array([float(x) for x in out])
    mm = min(m, n)
    w, Z = v[:n], v[n:].reshape(n, mm).T
    norm = max(1.0, np.abs(A).sum(1).max())
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-14 * n * norm
    for q, Aq in enumerate((np.eye(n), A, A @ A)):
        assert np.abs((Z * w ** q) @ Z.T - Aq[:mm, :mm]).max() <= 1e-14 * n * norm ** q
