"""The solver's sweep by cells (sweep.cu k_sweep_cell) at the sizes where its tiles end: part
tiles in k and j (12 of 16, 24 and 48 of 32 slots; levels 12 to 96), whole ones of both
widths, chunks of one plane, one sweep a colour (the first two in one launch) and two, and
fixed faces inside the domain. A sweep that
loses an unknown at an edge, or moves a fixed one, leaves a V-cycle that no longer
converges at the smooth densities' rate: the solve must reach its FP64 tolerance within 30
V-cycles (18 to 20 are usual), with the residual confirmed by the FP64 operator and
velocities of fixed faces exactly as the right-hand side has them.
"""
import numpy as np
import pytest

from tests.helpers import problem, relerr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def solve_and_check(oracle, stg, n, b, fp, limit, **opts):
    s = stg.Solver(n, tol=1e-8, **opts)
    s.set_boundary_from(b)
    s.set_penalty(np.zeros((n, n, n)), fp)
    s.set_rhs(b.cell_b, b.face_b)
    p, vel, st = s.solve()
    assert st["status"] == 0 and st["inner_iters"] <= limit, st
    x = torch.from_numpy(oracle.field_to_blocked(n, p, vel)).cuda()
    ax = torch.zeros_like(x)
    s.apply_A_device(s.levels - 1, ax.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    assert relerr(ax.cpu().numpy(), oracle.field_to_blocked(n, b.cell_b, b.face_b)) <= 2e-8
    for d in range(3):
        fixed = b.face_fixed[d] != 0
        assert np.array_equal(vel[d][fixed], b.face_b[d][fixed])
    s.close()


@pytest.mark.parametrize("n,sweeps,method", [(8, 1, 0), (16, 2, 0), (16, 1, 0), (16, 1, 1), (24, 1, 0), (32, 1, 1), (48, 2, 0), (64, 1, 0), (96, 1, 0),
                                             (96, 1, 1)])
def test_solve_at_tile_edges(oracle, stg, n, sweeps, method):
    b, rho, phys, fp = problem(oracle, n, seed=2)
    solve_and_check(oracle, stg, n, b, fp, 30, smooth_sweeps=sweeps, method=method)


@pytest.mark.parametrize("n", [16, 32, 64])
def test_solve_with_fixed_faces_inside(oracle, stg, n):
    """A baffle: the x-faces of half a cross-section are fixed, so the flow passes through the
    other half. (A fully closed-off block of cells is no test: its pressures are undetermined
    and the coarse levels, which fix a face when any child is, do not converge on it.)"""
    b, rho, phys, fp = problem(oracle, n, seed=2)
    b.face_fixed[0][n // 2, : n // 2, :] = 1
    solve_and_check(oracle, stg, n, b, fp, 120)
