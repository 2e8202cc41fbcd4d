"""Coarsest matrices without an inverse: a domain whose boundary faces are all fixed, set up without the
ones that `closed` adds, leaves the constant pressure undetermined, so the last cell's pivot is a
few units of the last place or exactly 0, by chance. (After an exact 0 the block elimination once
went on with NaN, where the lanes of its row search no longer agree, and could wait forever.) Every
set-up has to end, and the handle has to be as good as new for the closed problem.
"""
import numpy as np
import pytest

from tests.helpers import problem, problem2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(3, 4), (3, 8), (3, 16), (2, 8), (2, 32)])
def test_singular_setups_end(oracle, stg, dim, n):
    b, rho, phys, fp = (problem if dim == 3 else problem2)(oracle, n, seed=3)
    zero = np.zeros((n,) * dim)

    def solve(s):
        s.set_boundary(b.cell_vol, None, b.face_vol, b.face_fixed, True)
        s.set_penalty(zero, fp)
        s.set_rhs(b.cell_b, b.face_b)
        return s.solve()

    s = stg.Solver(n, dim=dim)
    s.set_boundary(b.cell_vol, None, b.face_vol, b.face_fixed, False)
    rng = np.random.default_rng(n)
    for _ in range(64):  # about one in ten meets an exact 0
        s.set_penalty(zero, [1e4 * rng.random(f.shape) for f in fp])
        s.update()
    s.set_penalty(zero, [np.zeros(f.shape) for f in fp])
    s.update()
    p, vel, st = solve(s)
    q, ref, _ = solve(stg.Solver(n, dim=dim))
    s.close()
    assert st["status"] == 0 and np.array_equal(p, q)
    assert all(np.array_equal(a, c) for a, c in zip(vel, ref))


@pytest.mark.parametrize("dim,n", [(3, 8), (3, 16), (2, 8), (2, 64)])  # (4^3 has no inlet)
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_handle_survives_penalties_that_are_no_numbers(oracle, stg, dim, n, value):
    """The pivot search of a column of NaN once pointed one row past the matrix. The solve reports
    the non-finite residual, and the next penalties are solved as on a new handle."""
    b, rho, phys, fp = (problem if dim == 3 else problem2)(oracle, n, seed=3)
    zero = np.zeros((n,) * dim)

    def solve(s, pen):
        s.set_boundary_from(b)
        s.set_penalty(zero, pen)
        s.set_rhs(b.cell_b, b.face_b)
        return s.solve()

    bad = [f.copy() for f in fp]
    for f in bad:
        f[(n // 2,) * dim] = value
    s = stg.Solver(n, dim=dim)
    with pytest.raises(stg.StgError) as e:
        solve(s, bad)
    assert e.value.code == stg.STG_E_NONFINITE
    p, vel, _ = solve(s, fp)
    q, ref, _ = solve(stg.Solver(n, dim=dim), fp)
    s.close()
    assert np.array_equal(p, q) and all(np.array_equal(a, c) for a, c in zip(vel, ref))
