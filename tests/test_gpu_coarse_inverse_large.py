"""The coarsest inverse of the 12^3 level (7344 unknowns: grids of 12, 24, 48 and 96 cells), formed by
blocks of three axes in 32-wide tiles, which no smaller grid takes: A x = r through the FP64
operator, and that it is the block form that ran.

Residual: for a computed inverse X, |A X - I| is at most a few N eps |A| |X|, so |r - A x| is held
to N eps |A| |x|, |A| bounded by its largest row sum. Route: the pivoted form's 4 N^3 = 1.6e12 FP64
operations take 1.2 s at the GPU's peak rate (1.3e12 / s) at the least, and take 11; the block
form's set-up is 0.17 s.
"""
import time

import numpy as np
import pytest

from tests.helpers import problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,contrast", [(12, False), (24, False), (48, True)])
def test_inverse_of_the_12_cubed_level(oracle, stg, n, contrast):
    b, rho, phys, fp = problem(oracle, n, seed=3)
    if contrast:
        rng = np.random.default_rng(5)
        fp = [np.where(rng.random(f.shape) < 0.5, 1e4, 1e-3) for f in fp]
    s = stg.Solver(n)
    s.set_boundary_from(b)
    s.set_penalty(np.zeros((n, n, n)), fp)
    s.update()  # attributes and module loading
    torch.cuda.synchronize()
    t = time.perf_counter()
    s.update()
    torch.cuda.synchronize()
    assert time.perf_counter() - t < 1.2
    nd = s.level_dof(0)
    vol, pen = torch.zeros(nd, dtype=torch.float64, device="cuda"), torch.zeros(nd, dtype=torch.float64, device="cuda")
    fixed = torch.zeros(nd, dtype=torch.uint8, device="cuda")
    s.level_descr_device(0, vol.data_ptr(), pen.data_ptr(), fixed.data_ptr())
    v, cells = float(vol[12 ** 3:].max()), 12 ** 3
    row_sum = 14.0 * v + float(pen.max()) + cells
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(nd)).cuda() * (1 - fixed)
    x, ax = torch.zeros_like(r), torch.zeros_like(r)
    s.apply_op_device(stg.STG_OP_COARSE, 0, x.data_ptr(), r.data_ptr())
    s.apply_A_device(0, ax.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    ax[:cells] += x[:cells].sum()
    s.close()
    assert float((r - ax).norm()) <= 7344 * 2.0 ** -52 * row_sum * float(x.norm())
