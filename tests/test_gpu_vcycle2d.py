"""The 2D solver's Laplacian-form V-cycle (solver2d.cu vcycle2_lap) against the general one it
replaces on closed boundaries, over its launch forms: everything in one cluster (16 to 128),
one level only (8, 24), the coarsest solve outside the cluster (48, 96), levels above the
cluster's (192, 256).

A boundary whose face vols are one value but whose cell (0, 0) is fixed runs the general form,
so the pair cannot share a problem; instead each solve must reach the FP64 tolerance, confirmed
by the FP64 operator, in about as many V-cycles as the same problem at the sizes of the parity
tests takes (17 to 22 on smooth densities), and with a baffle of fixed faces inside.
"""
import numpy as np
import pytest

from tests.helpers import problem2, relerr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def solve_and_check(oracle, stg, n, b, fp, limit, vol=1.0):
    s = stg.Solver(n, dim=2, tol=1e-10)
    s.set_boundary(b.cell_vol, b.cell_fixed, [vol * f for f in b.face_vol], b.face_fixed, True)
    s.set_penalty(np.zeros((n, n)), [vol * f for f in fp])
    rhs = [vol * b.cell_b, [vol * f for f in b.face_b]]
    s.set_rhs(*rhs)
    p, vel, st = s.solve()
    assert st["status"] == 0 and st["inner_iters"] <= limit, st
    x = torch.from_numpy(oracle.field_to_blocked2(n, p, vel)).cuda()
    ax = torch.zeros_like(x)
    s.apply_A_device(s.levels - 1, ax.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    assert relerr(ax.cpu().numpy(), oracle.field_to_blocked2(n, rhs[0], rhs[1])) <= 2e-10
    for d in range(2):
        assert not np.any(vel[d][b.face_fixed[d] != 0])
    s.close()


@pytest.mark.parametrize("n,vol", [(8, 1.0), (16, 1.0), (24, 1.0), (48, 1.0), (64, 0.9), (96, 1.0), (128, 1.0), (192, 1.0), (256, 1.0)])
def test_solve_2d_launch_forms(oracle, stg, n, vol):
    b, rho, phys, fp = problem2(oracle, n, seed=2)
    solve_and_check(oracle, stg, n, b, fp, 40, vol)


@pytest.mark.parametrize("n", [32, 64, 256])
def test_solve_2d_with_baffle(oracle, stg, n):
    b, rho, phys, fp = problem2(oracle, n, seed=2)
    b.face_fixed[0][n // 2, : n // 2] = 1
    solve_and_check(oracle, stg, n, b, fp, 200)
