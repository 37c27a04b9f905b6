"""A call of the projected Green function whose input is too large for the pinned
staging (10 MB here) gives the numbers of the same frequencies in small calls, bit for
bit where the grid's CTAs are the same."""
import numpy as np
import pytest

from tests.test_gpu_lattice_sums import _elements, _loaded_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nw", [(4, 40000), (16, 300), (2, 16380), (2, 16390)])  # the last two: both sides of 1 MB
def test_large_inputs_match_small_calls(qed, fresh, n, nw):
    rng = np.random.default_rng(n)
    label, _ = _loaded_instance(qed, fresh, n, rng)
    el = _elements(n, rng, 5)
    w = np.linspace(0.1, 20.0, nw)
    V0 = rng.standard_normal((nw, n, n)) + 1j * rng.standard_normal((nw, n, n))
    call = lambda a, b: qed.cpt_projected_green_function(V0[a:b], *el, w[a:b], (3, 2, 1), offset=0.5, label=label)
    got = call(0, nw)
    for a in (0, nw // 2, nw - 7):  # six wavevectors fit one CTA whatever the frequencies
        assert np.array_equal(got[a:a + 7], call(a, a + 7)), a
    again = call(0, 5)  # the pinned buffer serves the next small call
    assert np.array_equal(again, got[:5])
