"""The optimality-criteria update where its form changes (topo.cu oc_update_device): one cluster
up to 16384 cells, the whole device with a thread's cells in registers, and with the cells read
for each probe, against the bisection in NumPy. Either ends with a bracket of half-width at most
1e-9 of the multiplier around the same root, so the multipliers differ by at most 2e-9 and the
designs, which go with its root, by 1e-9 of the largest entry (1).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bisect(x, dc, vw, frac, move, lo, hi):
    n = x.size

    def new(lam):
        return np.minimum(np.minimum(hi, x + move), np.maximum(np.maximum(lo, x - move),
                                                              x * np.sqrt(np.maximum(0.0, -dc) / (vw / n * lam))))

    l1, l2 = 0.0, 1e9
    while np.sum(vw * new(l2)) > frac * n:
        l1, l2 = l2, 10 * l2
    for _ in range(200):
        if l2 - l1 <= 1e-9 * (l1 + l2):
            break
        mid = 0.5 * (l1 + l2)
        l1, l2 = (mid, l2) if np.sum(vw * new(mid)) > frac * n else (l1, mid)
    mid = 0.5 * (l1 + l2)
    return new(mid), mid


# cells: 64, 4096 and 16384 (all that the cluster holds), 25600 and 64^3 (registers), 96^3 (either), 128^3
# (more than 1216 blocks of 256 threads hold four a thread)
@pytest.mark.parametrize("dim,n", [(2, 8), (2, 64), (2, 128), (2, 160), (3, 24), (3, 64), (3, 96), (3, 128)])
@pytest.mark.parametrize("scale", [1.0, 1e14])
def test_oc_forms(stg, dim, n, scale):
    rng = np.random.default_rng(n)
    shape = (n,) * dim
    x = 0.05 + 0.9 * rng.random(shape)
    dc = -scale * rng.random(shape)
    dc[rng.random(shape) < 0.1] *= -1.0  # rising objective: the lower bound
    s = stg.Solver(n, dim=dim)
    vw = s.filter(1.5, np.ones(shape), transpose=True)
    xn, lam = s.oc_update(1.5, x, dc, 0.4)
    s.close()
    ref, ref_lam = bisect(x.ravel(), dc.ravel(), vw.ravel(), 0.4, 0.2, 0.0, 1.0)
    assert abs(lam - ref_lam) <= 2e-9 * ref_lam
    assert np.max(np.abs(xn.ravel() - ref)) <= 1e-9


@pytest.mark.parametrize("rmin", [1.5, 4.0])
def test_transposed_filter(stg, rmin):
    """H^T y over the weights written out: at most (2R+1)^3 = 343 positive terms a sum."""
    n, R = 8, int(np.ceil(rmin)) - 1
    y = np.random.default_rng(2).random((n, n, n))
    off = np.arange(-R, R + 1)
    g = np.stack(np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"), -1).reshape(-1, 3)
    w = np.maximum(0.0, rmin - np.sqrt(((g[:, None] - g[None]) ** 2).sum(-1)))
    ref = w.T @ (y.ravel() / w.sum(1))
    s = stg.Solver(n)
    out = s.filter(rmin, y, transpose=True).ravel()
    s.close()
    assert np.max(np.abs(out - ref)) <= (2 * off.size ** 3) * 2.3e-16 * np.max(ref)
