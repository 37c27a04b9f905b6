"""The packed form of the symmetry-adapted Hamiltonian (csrc/mixed.cu) against the
on-the-fly products, which evaluate the same matrix elements from the states:
every number of warps per slice, dimensions that are no multiple of 32, bath
orbitals with irrep phases, all irreps, more than 2^24 states (separate codes),
and infinities next to padded entries."""
import ctypes as C

import numpy as np
import pytest
import torch

from pyqcm_b200 import workloads as W
from tests.helpers import c2v_golden, c2v_problem

pytestmark = pytest.mark.gpu


def _ladder(nx, ny, tp=0.3):
    p = W.hubbard_cluster(nx, ny, tp=tp, U=5.0, mu=2.1)
    s = lambda x, y: 1 + x + nx * y
    p.generators = [[s(nx - 1 - x, y) for y in range(ny) for x in range(nx)],
                    [s(x, ny - 1 - y) for y in range(ny) for x in range(nx)]]
    return p


def _chain(n):
    p = W.hubbard_cluster(n, 1, U=5.0)
    p.generators = [list(range(n, 0, -1))]
    return p


def _apply(qed, H, x):
    y = torch.full_like(x, float("nan"))
    qed._check(qed.lib().qed_mixed_hamiltonian_apply_device(H.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                                                            C.c_void_p(0)))
    torch.cuda.synchronize()
    return y


def _pair(qed, fresh, prob, sector):
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="pack" + suffix)
    qed.set_global_parameter("mixed_on_the_fly", True)
    try:
        ref = qed.MixedHamiltonian(label, sector)
    finally:
        qed.set_global_parameter("mixed_on_the_fly", False)
    return qed.MixedHamiltonian(label, sector), ref


@pytest.mark.parametrize("case,sectors", [
    ("record", ["R0:N12:S0", "R1:N12:S0", "R2:N11:S1", "R3:N12:S0", "R1:N7:S1"]),
    ("2x4", ["R0:N8:S0", "R3:N7:S1"]), ("2x5", ["R1:N10:S0", "R2:N9:S1"]), ("2x6", ["R0:N12:S0"]),
    ("2x7", ["R2:N13:S1"]), ("chain9", ["R0:N9:S1", "R1:N8:S0"]), ("4x4", ["R0:N14:S0"])])
def test_packed_products_match_on_the_fly(qed, fresh, case, sectors):
    prob = (c2v_problem(c2v_golden(), True) if case == "record" else _chain(9) if case == "chain9"
            else _ladder(*map(int, case.split("x"))))
    for sec in sectors:
        H, R = _pair(qed, fresh, prob, sec)
        assert H.dim == R.dim and H.nnz == R.nnz, sec
        assert case != "4x4" or H.dim > 1 << 24
        x = torch.randn(H.dim, dtype=torch.float64, device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(3))
        y, r = _apply(qed, H, x), _apply(qed, R, x)
        # sums of at most 100 terms in another order: 100 eps sum |terms|
        assert float((y - r).abs().max()) <= 1e-12 * float(r.abs().max()), sec


def test_padding_reads_nothing(qed, fresh):
    """Rows shorter than their slice: an infinite entry of x reaches exactly the
    rows that have a matrix element on it."""
    H, R = _pair(qed, fresh, _ladder(2, 4), "R0:N7:S1")
    x = torch.randn(H.dim, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    x[H.dim // 3] = float("inf")
    y, r = _apply(qed, H, x), _apply(qed, R, x)
    assert torch.equal(torch.isfinite(y), torch.isfinite(r))
    assert 1 < int((~torch.isfinite(y)).sum()) < H.dim // 4
