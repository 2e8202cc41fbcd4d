"""The first calls on a fresh handle find its memory cleared, not being cleared: the arrays are zeroed
on the handle's own stream (by the default stream, which the handle's does not wait for, a clearing could
land on what the first call had written). A boundary and penalties set right after creation read
back as they were given, and the first call of each entry point that allocates its buffers on
first use gives the bits of the second. The solve's own tables, too: a solve that needs its whole
basis several times over (a channel of contrast 1e4) gives the same bits on every fresh handle.
"""
import numpy as np
import pytest

from tests.helpers import stable_vec

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,n,times", [(2, 8, 20), (2, 64, 20), (2, 1024, 3), (3, 8, 20), (3, 32, 10), (3, 128, 3)])
def test_first_calls_on_a_fresh_handle(stg, dim, n, times):
    shapes = [tuple(n + (a == d) for a in range(dim)) for d in range(dim)]
    fixed = [np.zeros(s, np.int32) for s in shapes]
    for d in range(dim):
        np.moveaxis(fixed[d], d, 0)[[0, n]] = 1
    pen = [np.full(s, 2.0 + d) for d, s in enumerate(shapes)]
    vol = [np.ones(s) for s in shapes]
    free = [int((f == 0).sum()) for f in fixed]
    for _ in range(times):
        s = stg.Solver(n, dim=dim)
        s.set_boundary(np.ones((n,) * dim), None, vol, fixed, True)
        s.set_penalty(np.zeros((n,) * dim), pen)
        top = s.levels - 1
        nd = s.level_dof(top)
        v, p = torch.zeros(nd, dtype=torch.float64, device="cuda"), torch.zeros(nd, dtype=torch.float64, device="cuda")
        f = torch.zeros(nd, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        s.level_descr_device(top, v.data_ptr(), p.data_ptr(), f.data_ptr())
        assert [int((p == 2.0 + d).sum()) for d in range(dim)] == free
        assert int((f == 0).sum()) == n ** dim + sum(free)
        x = torch.from_numpy(stable_vec(3, nd)).cuda() * (1 - f)
        out = [torch.zeros(nd, dtype=torch.float64, device="cuda") for _ in range(6)]
        torch.cuda.synchronize()
        for k in range(2):
            s.vcycle_device(out[k].data_ptr(), x.data_ptr())
            s.apply_A_device(top, out[2 + k].data_ptr(), x.data_ptr())
            s.apply_E_device(out[4 + k].data_ptr(), x.data_ptr())
        torch.cuda.synchronize()
        assert all(torch.equal(out[k], out[k + 1]) and float(out[k].abs().max()) > 0 for k in (0, 2, 4))
        s.close()


@pytest.mark.parametrize("dim,n", [(2, 64), (3, 16), (3, 64), (3, 128)])
def test_first_solve_on_a_fresh_handle(stg, dim, n):
    g = np.indices((n,) * dim) / n
    x = np.where(np.abs(g[1] - 0.5) < 0.125, 1.0, 1e-8)
    shapes = [tuple(n + (a == d) for a in range(dim)) for d in range(dim)]
    fixed = [np.zeros(s, np.int32) for s in shapes]
    for d in range(dim):
        np.moveaxis(fixed[d], d, 0)[[0, n]] = 1
    cell = np.zeros((n,) * dim)
    cell[0, 3 * n // 8:5 * n // 8], cell[n - 1, 3 * n // 8:5 * n // 8] = 1.0, -1.0
    got = []
    for _ in range(3):
        s = stg.Solver(n, dim=dim, inner_max=12)
        s.set_boundary(np.ones((n,) * dim), None, [np.ones(q) for q in shapes], fixed, True)
        s.set_density(x, stg.alpha_bp(1e4))
        s.set_rhs(cell, [np.zeros(q) for q in shapes])
        p, vel, st = s.solve()
        got.append([p] + list(vel) + [np.array([st["inner_iters"], st["outer_iters"]])])
        s.close()
    for a in got[1:]:
        assert all(np.array_equal(u, v) for u, v in zip(a, got[0]))
    assert st["status"] == 0 and st["inner_iters"] < 300
