"""The one-launch (csrc/hv_fused.cu) and tiled (csrc/hv_tile.cu) forms of H x
against the two-pass kernels (hv_variant bit 8 turns the new forms off): row
counts that leave part of a tile, odd dimensions, misaligned vectors, asymmetric
spins, every range of sector sizes. Both sides sum at most 60 terms per state in
FP64: 60 eps sum |terms| stays below 1e-13 of the largest."""
from math import comb

import numpy as np
import pytest
import torch

from pyqcm_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _problem(nx, ny, up, dn, tp=None, M=0.2, bath=False):
    if bath:
        rng = np.random.default_rng(3)
        p = W.plaquette_bath(rng.uniform(-2, 2, 8), rng.uniform(0.1, 1, 8), U=6.0)
    else:
        p = W.hubbard_cluster(nx, ny, tp=tp, U=5.0, mu=2.2, M=M)
    p.sectors = f"R0:N{up + dn}:S{up - dn}"
    return p


@pytest.fixture
def variant(qed):
    yield lambda v: qed.set_global_parameter("hv_variant", v)
    qed.set_global_parameter("hv_variant", 2)


@pytest.mark.parametrize("shape", [
    (8, 1, 4, 4), (7, 1, 3, 3), (7, 1, 2, 5), (2, 4, 3, 5), (9, 1, 4, 5), (10, 1, 5, 5), (2, 5, 5, 2),   # one launch
    (2, 6, 6, 3), (13, 1, 2, 6), (3, 4, 1, 6), (14, 1, 1, 7), (2, 7, 7, 2),
    (11, 1, 5, 6), (12, 1, 5, 4), (2, 6, 6, 5), (13, 1, 6, 4), (3, 5, 4, 4), (2, 7, 7, 6)])                # tiles
def test_new_forms_match_two_pass_kernels(qed, fresh, variant, shape):
    nx, ny, up, dn = shape
    # vectors off the 16-byte boundary where the rows are of odd length (the two-pass
    # kernels need 16-byte alignment for even ones)
    offset = comb(nx * ny, up) % 2
    prob = _problem(nx, ny, up, dn, tp=0.3 if ny > 1 else None)
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="form" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(H.dim + offset, dtype=torch.float64, device="cuda", generator=g)[offset:]
    out = []
    for v in (2, 10):
        variant(v)
        y = torch.full((H.dim + offset,), float("nan"), dtype=torch.float64, device="cuda")[offset:]
        d = torch.zeros(3, dtype=torch.float64, device="cuda")
        H.apply_dots_device(x.data_ptr(), y.data_ptr(), d.data_ptr())
        torch.cuda.synchronize()
        out.append((y, d))
    (y, d), (r, e) = out
    assert float((y - r).abs().max()) <= TOL * float(r.abs().max())
    assert float((d - e).abs().max()) <= 1e-12 * float(e.abs().max())


@pytest.mark.parametrize("case", ["bath", "2x4", "2x5", "12x1"])
def test_recurrences_do_not_take_the_new_forms(qed, fresh, variant, case):
    """Ground states and Green functions keep the order of their sums: the same
    bits with the new forms on and off."""
    prob = _problem(0, 0, 6, 6, bath=True) if case == "bath" else {
        "2x4": _problem(2, 4, 4, 4, tp=0.3), "2x5": _problem(2, 5, 5, 5, tp=0.3),
        "12x1": _problem(12, 1, 6, 6, M=None)}[case]
    z = W.matsubara(32)
    res = []
    for v in (2, 10):
        variant(v)
        suffix, label = fresh()
        qed.load_problem(prob, label, model_name="formsolve" + suffix, fmt="F")
        e, _ = qed.ground_state_solve(label)
        res.append((e, qed.Green_function(z, label=label)))
    assert res[0][0] == res[1][0]
    assert np.array_equal(res[0][1], res[1][1])


def test_interaction_on_some_sites(qed, fresh, variant):
    """U on the cluster and none on the bath: the masked interaction term against
    the diagonal, also through qed_hamiltonian_diag."""
    prob = _problem(0, 0, 2, 3, bath=True)
    suffix, label = fresh()
    qed.load_problem(prob, label, model_name="formmask" + suffix, fmt="F")
    H = qed.Hamiltonian(label, prob.sectors)
    n = prob.n_orb
    up, dn = qed.halfbasis(n, 2).astype(np.int64), qed.halfbasis(n, 3).astype(np.int64)
    occ = lambda s: np.stack([(s >> i) & 1 for i in range(n)], 1).astype(float)
    eps = np.array([-prob.params["mu"]] * 4 + [prob.params[f"eb{b}"] for b in range(8)])
    U = np.array([prob.params["U"]] * 4 + [0.0] * 8)
    ref = (occ(dn) * U) @ occ(up).T + (occ(up) @ eps)[None] + (occ(dn) @ eps)[:, None]
    assert np.max(np.abs(H.diag().reshape(len(dn), len(up)) - ref)) < 1e-12
