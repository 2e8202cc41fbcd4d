"""The coarsest inverse formed by blocks (dense.cu k_inv_blocks) against the oracle's pivoted
LU: both block sizes (304 and 320 unknowns in 16-wide blocks, 2112 in 32-wide ones), high
contrast, and the cases that leave the block elimination (negative penalties make a pivot's
sign wrong; fixed cells).

Tolerance 1e-9 as for the coarsest solve of the parity tests: two backward-stable FP64
inversions differ by about N eps cond; cond is at most 1e4 (contrast) times N.
"""
import numpy as np
import pytest

from tests.helpers import problem, problem2, relerr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def check(stg, o, s, tol=1e-9):
    assert o.coarse_info() == 0
    fixed = o.descr(0)[2]
    for seed in (7, 8):
        r = np.random.default_rng(seed).standard_normal(o.level_dof(0)) * (1 - fixed)
        out = torch.zeros(o.level_dof(0), dtype=torch.float64, device="cuda")
        rd = torch.from_numpy(r).cuda()
        s.apply_op_device(stg.STG_OP_COARSE, 0, out.data_ptr(), rd.data_ptr())
        torch.cuda.synchronize()
        assert relerr(out.cpu().numpy(), o.coarse_apply(r)) < tol


def pair2(po, stg, n, fp, b):
    o = po.Steady2D(n)
    o.init_boundary(b)
    o.update_penalty(np.zeros((n, n)), fp)
    o.update_b(b.cell_b, b.face_b)
    s = stg.Solver(n, dim=2)
    s.set_boundary_from(b)
    s.set_penalty(np.zeros((n, n)), fp)
    s.update()
    return o, s


@pytest.mark.parametrize("n,kind", [(8, "noise"), (16, "contrast"), (24, "noise"), (24, "contrast"), (48, "noise"), (16, "negative"),
                                    (16, "fixed_cell")])
def test_coarse_inverse_2d(oracle, stg, n, kind):
    b, rho, phys, fp = problem2(oracle, n, seed=3)
    rng = np.random.default_rng(5)
    if kind == "contrast":
        fp = [np.where(rng.random(f.shape) < 0.5, 1e4, 1e-3) for f in fp]
    if kind == "negative":
        fp = [f - 2.0 * f.max() * (rng.random(f.shape) < 0.3) for f in fp]
    if kind == "fixed_cell":
        b.cell_fixed[n // 2, n // 2] = 1
    check(stg, *pair2(oracle, stg, n, fp, b))


@pytest.mark.parametrize("n,kind", [(4, "noise"), (16, "noise"), (8, "contrast"), (8, "negative")])
def test_coarse_inverse_3d(oracle, stg, n, kind):
    b, rho, phys, fp = problem(oracle, n, seed=3)
    rng = np.random.default_rng(5)
    if kind == "contrast":
        fp = [np.where(rng.random(f.shape) < 0.5, 1e4, 1e-3) for f in fp]
    if kind == "negative":
        fp = [f - 2.0 * f.max() * (rng.random(f.shape) < 0.3) for f in fp]
    o = oracle.Steady3D(n)
    o.init_boundary(b)
    o.update_penalty(np.zeros((n, n, n)), fp)
    o.update_b(b.cell_b, b.face_b)
    o.setup()
    s = stg.Solver(n)
    s.set_boundary_from(b)
    s.set_penalty(np.zeros((n, n, n)), fp)
    s.update()
    check(stg, o, s)
