"""A handle whose boundary changes the faces' vol answers as one created for that vol: the captured
set-up and V-cycle hold the vol as a kernel argument and must not be replayed with the old one.
"""
import numpy as np
import pytest

from tests.helpers import problem, problem2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def answers(stg, s, b, fp, vol):
    s.set_boundary(b.cell_vol, None, [np.full(f.shape, vol) for f in b.face_vol], b.face_fixed, True)
    s.set_penalty(np.zeros(b.cell_b.shape), [vol * f for f in fp])
    s.set_rhs(vol * b.cell_b, [vol * f for f in b.face_b])
    p, vel, st = s.solve()
    s.update()
    nd = s.level_dof(0)
    fixed = torch.zeros(nd, dtype=torch.uint8, device="cuda")
    a, c = torch.zeros(nd, dtype=torch.float64, device="cuda"), torch.zeros(nd, dtype=torch.float64, device="cuda")
    s.level_descr_device(0, a.data_ptr(), c.data_ptr(), fixed.data_ptr())
    r = torch.from_numpy(np.random.default_rng(2).standard_normal(nd)).cuda() * (1 - fixed)
    s.apply_op_device(stg.STG_OP_COARSE, 0, c.data_ptr(), r.data_ptr())
    torch.cuda.synchronize()
    return [p] + list(vel) + [c.cpu().numpy(), np.array(st["inner_iters"])]


@pytest.mark.parametrize("dim,n", [(3, 16), (3, 32), (2, 64), (2, 256)])
def test_vol_change_reaches_the_captured_graphs(oracle, stg, dim, n):
    b, rho, phys, fp = (problem if dim == 3 else problem2)(oracle, n, seed=2)
    s = stg.Solver(n, dim=dim)
    for _ in range(3):  # run, capture, replay
        answers(stg, s, b, fp, 1.0)
    again = answers(stg, s, b, fp, 0.25)
    fresh = answers(stg, stg.Solver(n, dim=dim), b, fp, 0.25)
    s.close()
    for x, y in zip(again, fresh):
        assert np.array_equal(x, y)
