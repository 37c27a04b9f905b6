"""The wavevector sums (csrc/lattice.cu) on grids beyond their tables and CTAs: more
points along a direction than the phase table holds, and so many in all that a warp
takes more batches of them (the memory of the partial sums does not grow with the
grid). Where V depends on one direction only, the average over the whole grid is that
over this direction, which numpy forms."""
import numpy as np
import pytest
import torch

from tests.test_gpu_lattice_sums import TOL, _V, _loaded_instance

pytestmark = pytest.mark.gpu


def _along(axis, n, rng, nel):
    """Elements whose translations all lie along one direction."""
    R = [tuple(int(x) if i == axis else 0 for i in range(3)) for x in rng.integers(-3, 4, nel)]
    return ([int(x) for x in rng.integers(0, n, nel)], [int(x) for x in rng.integers(0, n, nel)], R,
            [complex(*rng.standard_normal(2)) for _ in range(nel)])


@pytest.mark.parametrize("n,nk,axis", [(3, (400, 1, 1), 0), (4, (1, 380, 7), 1), (2, (5, 3, 1000), 2),   # sincospi
                                       (6, (300, 40, 44), 0), (10, (128, 128, 1), 1),
                                       (16, (64, 64, 3), 2), (1, (128, 100, 128), 0)])                  # more batches
def test_large_grids_match_the_one_direction(qed, fresh, n, nk, axis):
    rng = np.random.default_rng(n + nk[axis])
    label, G = _loaded_instance(qed, fresh, n, rng)
    el = _along(axis, n, rng, 2 * n)
    w = np.array([0.2, 1.3])
    V0 = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    line = lambda off: [np.eye(3)[axis] * (i + off) / nk[axis] for i in range(nk[axis])]
    got = qed.sef_integrand_grid(V0[0], *el, w, nk, label=label)
    for i in range(2):
        ref = np.mean([np.linalg.slogdet(_V(V0[0], el, k) @ G(w[i]) - np.eye(n))[1] for k in line(0.0)])
        assert abs(got[i] - ref) <= TOL * max(1.0, abs(ref)), i
    got = qed.cpt_projected_green_function(V0, *el, w, nk, offset=0.5, label=label)
    for i in range(2):
        ref = np.mean([G(w[i]) @ np.linalg.inv(np.eye(n) - _V(V0[i], el, k) @ G(w[i])) for k in line(0.5)], axis=0)
        assert np.max(np.abs(got[i] - ref)) <= TOL * max(1.0, np.max(np.abs(ref))), i


def test_partial_sums_do_not_grow_with_the_grid(qed, fresh):
    """256 frequencies of dimension 4 on 128^3 wavevectors: 64 partial sums a frequency
    are 4 MB, one per CTA at a fixed number of wavevectors each would be 537 MB."""
    rng = np.random.default_rng(5)
    label, _ = _loaded_instance(qed, fresh, 4, rng)
    el = _along(0, 4, rng, 6)
    w = np.linspace(0.1, 9.0, 256)
    V0 = np.zeros((256, 4, 4), complex)
    ref = qed.cpt_projected_green_function(V0, *el, w, (128, 1, 1), offset=0.5, label=label)
    free = torch.cuda.mem_get_info()[0]
    got = qed.cpt_projected_green_function(V0, *el, w, (128, 128, 128), offset=0.5, label=label)
    assert free - torch.cuda.mem_get_info()[0] < 128 << 20
    assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))
