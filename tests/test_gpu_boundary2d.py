"""Which 2D boundaries take the Laplacian-form V-cycle: every boundary face fixed, no cell fixed, one
vol on the free faces, wherever the exception lies (first and last cell or face of either axis).
The form shows in the launches: its V-cycle of 64^2 is one, the general one's over sixty. Either
way the solve reaches its tolerance; where the vols differ or boundary faces are free, its
residual is checked through the FP64 operator by the solve itself.
"""
import numpy as np
import pytest

from tests.helpers import problem2

pytestmark = pytest.mark.gpu


def launches_a_cycle(stg, s, b, fp):
    s.set_penalty(np.zeros(b.cell_b.shape), fp)
    s.set_rhs(b.cell_b, b.face_b)
    s.solve(want=False, allow_not_converged=True)
    before = stg.kernel_launches()
    st = s.solve(want=False, allow_not_converged=True)[2]
    return (stg.kernel_launches() - before) / st["inner_iters"]


@pytest.mark.parametrize("n", [64, 512])
def test_boundary_form(oracle, stg, n):
    b, rho, phys, fp = problem2(oracle, n, seed=2)
    s = stg.Solver(n, dim=2, max_outer=1)
    one = [np.ones(f.shape) for f in b.face_fixed]
    cycle = 12.0 if n == 64 else 30.0  # 512^2: a launch a pass of the two levels above the cluster's

    def form(cell_fixed=None, face_vol=one, face_fixed=b.face_fixed):
        s.set_boundary(b.cell_vol, cell_fixed, face_vol, face_fixed, True)
        return launches_a_cycle(stg, s, b, fp) < cycle

    assert form()
    assert form(np.zeros((n, n), np.int32))
    for at in ((0, 0), (n - 1, n - 1), (n // 2, 3)):
        c = np.zeros((n, n), np.int32)
        c[at] = 1
        assert not form(c)
    for d in range(2):
        for at in ((1, 1), (n - 1, n - 1)):  # free faces of either end
            v = [f.copy() for f in one]
            v[d][at] = 0.5
            assert not form(None, v)
            v[d][at] = np.nan
            fixed = [f.copy() for f in b.face_fixed]
            fixed[d][at] = 1
            assert form(None, v, fixed)  # a fixed face's vol does not count
        for end in (0, n):
            fixed = [f.copy() for f in b.face_fixed]
            fixed[d][(end, n - 1) if d == 0 else (n - 1, end)] = 0
            assert not form(None, one, fixed)
    assert form()
    s.close()
