"""The operators A and E in the blocked layout (kernels.cu k_op_blocked) against the slot form
that vectors sharing their memory take: any vector, fixed faces and the layout's padding
included, on grids that fill their 4 x 4 x 16 tiles and grids that do not, with fixed faces
inside. Both sum at most 13 terms of one size, so they agree to a few eps of the largest: 1e-14.
"""
import numpy as np
import pytest

from tests.helpers import problem, relerr, stable_vec

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [4, 8, 12, 16, 24, 32])
@pytest.mark.parametrize("inside", [False, True])
def test_blocked_operator_matches_slot_form(oracle, stg, n, inside):
    b, rho, phys, fp = problem(oracle, n, seed=6)
    if inside:
        b.face_fixed[1][:, n // 2, : n // 2] = 1
    s = stg.Solver(n)
    s.set_boundary_from(b)
    s.set_penalty(np.abs(stable_vec(3, n ** 3)).reshape(n, n, n), fp)
    lvl = s.levels - 1
    x = torch.from_numpy(stable_vec(9, s.level_dof(lvl))).cuda()
    for apply in (lambda o, i: s.apply_A_device(lvl, o.data_ptr(), i.data_ptr()),
                  lambda o, i: s.apply_E_device(o.data_ptr(), i.data_ptr())):
        out = torch.full_like(x, 7.0)
        apply(out, x)
        same = x.clone()
        apply(same, same)
        torch.cuda.synchronize()
        assert relerr(out.cpu().numpy(), same.cpu().numpy()) < 1e-14
    s.close()
