"""One application of the solver's own V-cycle against its FP64 restatement (vcycle_ref.py), over
every launch form: 3D levels in one cluster launch (8^3; 16^3 with one sweep a colour in shared
memory, with two through L2), the sweeps by cells in tiles of 16 and 32 slots, single and in pairs,
with part tiles (24, 48, 96), with the injection fused, apart, linear, and rounded to BF16; 2D from
one level (8, 24) over one cluster (16 to 128) to a launch a pass (192, 256); fixed faces inside, cell
penalties, another vol. A converged solve cannot show this: FGMRES and the FP64 refinement correct
whatever a preconditioner gets wrong, at the price of V-cycles only.

A solve of one refinement step that ends at its first column returns y z, z = M b the V-cycle of the
right-hand side, so z is compared up to a factor. Tolerance, relative to the largest entry of its
kind of unknown (pressure, velocity): a pass (4 sweeps a colour-sweep and level, residual, restriction,
prolongation) sums at most 20 terms in FP32, so passes x 20 x 2^-24. Corrections stored in BF16:
an entry within the FP32 error of a rounding tie goes the other way, 2^-8 of its size, about one in
2000, so 2^-7 at most and 5e-4 in the mean square.
"""
import numpy as np
import pytest

from tests import vcycle_ref
from tests.helpers import problem, problem2

pytestmark = pytest.mark.gpu


def check(stg, dim, n, b, fp, baffle, cell_pen, vol=1.0, **opts):
    rng = np.random.default_rng(n)
    if baffle:
        b.face_fixed[0][(n // 2, slice(0, n // 2))] = 1
        b.face_fixed[1][(slice(0, n // 4), n // 2)] = 1
    pen = rng.integers(0, 64, (n,) * dim) / 64.0 if cell_pen else np.zeros((n,) * dim)
    face_vol = [np.full(f.shape, vol) for f in b.face_vol]
    s = stg.Solver(n, dim=dim, max_outer=1, inner_tol=100.0, **opts)
    s.set_boundary(b.cell_vol, None, face_vol, b.face_fixed, True)
    s.set_penalty(pen, fp)
    cell_r = rng.standard_normal((n,) * dim)
    cell_r -= cell_r.mean()
    face_r = [np.where(f != 0, 0.0, rng.standard_normal(f.shape)) for f in b.face_fixed]
    s.set_rhs(cell_r, face_r)
    p, vel, st = s.solve(allow_not_converged=True)
    assert st["inner_iters"] == 1
    nlev = s.levels
    s.close()
    sweeps = opts.get("smooth_sweeps", 1) if dim == 3 else 1
    mixed = opts.get("method", 0) == stg.STG_METHOD_MIXED
    norm = np.sqrt(np.sum(cell_r ** 2) + sum(np.sum(f ** 2) for f in face_r))  # the basis vector (BF16's ties go with its scale)
    zp, zu = vcycle_ref.run(dim, n, nlev, vol, b.face_fixed, pen, fp, cell_r / norm, [f / norm for f in face_r], sweeps,
                            opts.get("prolong", 0) == 1, mixed)
    got, ref = [p] + list(vel), [zp] + list(zu)
    dot = lambda a, c: sum(float(np.vdot(x, y)) for x, y in zip(a, c))
    y = dot(got, ref) / dot(ref, ref)
    tol = (4 * sweeps + 3) * nlev * 20 * 2.0 ** -24
    for kind in ([0], range(1, dim + 1)):
        top = max(np.abs(y * ref[q]).max() for q in kind)
        err = max(np.abs(got[q] - y * ref[q]).max() for q in kind)
        assert err <= (2.0 ** -7 if mixed else tol) * top, (kind, err / top, tol)
        if mixed:
            rms = np.sqrt(sum(np.sum((got[q] - y * ref[q]) ** 2) for q in kind) / sum(np.sum((y * ref[q]) ** 2) for q in kind))
            assert rms <= 5e-4, rms
    for d in range(dim):
        assert not np.any(vel[d][b.face_fixed[d] != 0])


FORMS = [(n, s, m, p) for n, s, m, p in [
    (4, 1, 0, 0), (8, 1, 0, 0), (8, 2, 0, 0), (8, 1, 1, 0), (8, 1, 0, 1), (8, 2, 0, 1), (16, 1, 0, 0), (16, 2, 0, 0), (16, 1, 1, 0), (16, 2, 1, 0),
    (16, 1, 0, 1), (16, 2, 0, 1), (16, 1, 1, 1), (24, 1, 0, 0), (24, 2, 0, 0), (24, 1, 0, 1), (24, 1, 1, 0), (32, 1, 0, 0), (32, 2, 0, 0),
    (32, 1, 1, 0), (32, 1, 0, 1), (48, 1, 0, 0), (48, 2, 1, 0), (64, 1, 0, 0), (64, 2, 0, 0), (64, 1, 1, 0), (64, 1, 0, 1), (96, 1, 0, 0),
    (96, 1, 1, 0), (128, 1, 0, 0), (128, 2, 0, 0)]]


@pytest.mark.parametrize("n,sweeps,method,prolong", FORMS)
@pytest.mark.parametrize("inside", [False, True])
def test_vcycle_3d(oracle, stg, n, sweeps, method, prolong, inside):
    b, rho, phys, fp = problem(oracle, n, seed=4)
    check(stg, 3, n, b, fp, inside and n > 4, inside, smooth_sweeps=sweeps, method=method, prolong=prolong)


@pytest.mark.parametrize("n", [8, 16, 24, 32, 40, 48, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("inside,vol", [(False, 1.0), (True, 1.0), (True, 0.8)])
def test_vcycle_2d(oracle, stg, n, inside, vol):
    b, rho, phys, fp = problem2(oracle, n, seed=4)
    check(stg, 2, n, b, fp, inside, False, vol)
