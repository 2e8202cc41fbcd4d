"""The optimality-criteria update at 32^3, where its block sums (two buffers of 152) once passed
the end of a handle's array, against the bisection in NumPy, and on the 2D grid of about as many
cells. Tolerance as in test_gpu_oc_forms: either ends with a bracket of half-width at most 1e-9
of the multiplier around the same root. (28^3, the other such size, has a dense coarsest level of
90160 unknowns, 260 GB, and is checked by test_oc_form_cpu alone.)
"""
import numpy as np
import pytest

from tests.test_gpu_oc_forms import bisect

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(3, 32), (2, 160)])
def test_oc_update_between_the_cluster_and_full_grids(stg, dim, n):
    rng = np.random.default_rng(n)
    x = 0.05 + 0.9 * rng.random((n,) * dim)
    dc = -rng.random((n,) * dim)
    s = stg.Solver(n, dim=dim)
    vw = s.filter(1.5, np.ones((n,) * dim), transpose=True)
    xn, lam = s.oc_update(1.5, x, dc, 0.4)
    again, lam2 = s.oc_update(1.5, x, dc, 0.4)
    s.close()
    ref, ref_lam = bisect(x.ravel(), dc.ravel(), vw.ravel(), 0.4, 0.2, 0.0, 1.0)
    assert abs(lam - ref_lam) <= 2e-9 * ref_lam
    assert np.max(np.abs(xn.ravel() - ref)) <= 1e-9
    assert lam2 == lam and np.array_equal(again, xn)


@pytest.mark.parametrize("dim,n", [(3, 8), (3, 32), (2, 160)])
def test_volume_that_cannot_be_compared_keeps_widening(stg, dim, n):
    """A NaN fraction: no volume undershoots it, so the bracket is widened to its end (60
    decades past 1e9) and bisected down to its lower one, and the design falls as far as it may."""
    x = 0.05 + 0.9 * np.random.default_rng(n).random((n,) * dim)
    s = stg.Solver(n, dim=dim)
    xn, lam = s.oc_update(1.5, x, -np.ones((n,) * dim), float("nan"))
    s.close()
    assert abs(lam / 1e68 - 1.0) < 1e-8
    assert np.max(np.abs(xn - np.maximum(0.0, x - 0.2))) <= 1e-30  # x sqrt(ncell / 1e68) at most
