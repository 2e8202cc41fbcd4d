"""The solver's own V-cycle (uniform face vols, every boundary face fixed, no fixed cell) restated
in FP64 with NumPy, independently of the kernels: slot arrays of one component each with a
two-slot halo of zeros, absent unknowns marked fixed. `vcycle3` / `vcycle2` take the finest level's
fixed flags, penalties and right-hand side in Field order and return the correction likewise.
The penalties the 3D sweeps read are rounded as the library stores them (FP16 over a
power-of-two scale per level); everything else is FP64.
"""
import numpy as np
import scipy.sparse as sp
import scipy.sparse.linalg as spl

H = 2  # halo


def sh(a, d, s):
    """The value s slots on along axis d."""
    return np.roll(a, -s, axis=d)


class Level:
    def __init__(self, dim, n):
        self.dim, self.n = dim, n
        self.shape = (n + 2 * H + 1,) * dim
        self.core = (slice(H, H + n + 1),) * dim
        self.vol = self.lap = 1.0

    def box(self, d):
        """Where unknowns of kind d (-1: cells) exist."""
        return tuple(slice(H, H + self.n + (a == d)) for a in range(self.dim))

    def present(self, d):
        m = np.zeros(self.shape, bool)
        m[self.box(d)] = True
        return m

    def put(self, d, field):
        a = np.zeros(self.shape)
        a[self.box(d)] = field
        return a

    def children(self, a):
        """(2, n/2 + 1) pairs along every axis of the box, one slot of halo included."""
        c = self.n // 2 + 1
        a = a[(slice(H, H + 2 * c),) * self.dim]
        order = tuple(range(1, 2 * self.dim, 2)) + tuple(range(0, 2 * self.dim, 2))
        return a.reshape((c, 2) * self.dim).transpose(order).reshape((2 ** self.dim,) + (c,) * self.dim)

    def zeros(self):
        return [np.zeros(self.shape) for _ in range(self.dim + 1)]

    def parity(self, flag):
        s = sum(np.indices(self.shape)) - H * self.dim + flag
        return self.present(-1) & (s % 2 == 0)


def hierarchy(dim, n, nlev, vol, fixed, cell_pen, face_pen):
    F = Level(dim, n)
    F.vol = vol
    F.fix = [~F.present(d) for d in range(dim)]
    for d in range(dim):
        F.fix[d][F.box(d)] = np.asarray(fixed[d]) != 0
    F.P = [F.put(-1, cell_pen)] + [np.where(F.fix[d], 0.0, F.put(d, face_pen[d])) for d in range(dim)]
    levels = [F]
    for _ in range(nlev - 1):
        f = levels[0]
        C = Level(dim, f.n // 2)
        C.vol, C.lap = f.vol * 2 ** (dim - 1), f.lap * 2
        C.P = [np.zeros(C.shape)]
        C.P[0][C.core] = f.children(f.P[0]).sum(0)
        C.fix = []
        for d in range(dim):
            any_fixed = np.ones(C.shape, bool)
            any_fixed[C.core] = (f.children(f.fix[d]) & f.children(f.present(d))).any(0)
            C.fix.append(any_fixed | ~C.present(d))
            low = np.where(f.children(f.fix[d]), np.inf, f.children(f.P[d + 1])).min(0)
            p = np.zeros(C.shape)
            p[C.core] = 2.0 ** dim * low
            C.P.append(np.where(C.fix[d], 0.0, p))
        levels.insert(0, C)
    return levels


def laplace(a):
    return 2.0 * a.ndim * a - sum(sh(a, d, s) for d in range(a.ndim) for s in (-1, 1))


def residual(L, r, x, P):
    p, u = x[0], x[1:]
    rp = r[0] - (L.vol * sum(sh(u[d], d, 1) - u[d] for d in range(L.dim)) + P[0] * p)
    out = [np.where(L.present(-1), rp, 0.0)]
    for d in range(L.dim):
        ru = r[d + 1] - (L.vol * (laplace(u[d]) - (p - sh(p, d, -1))) + P[d + 1] * u[d])
        out.append(np.where(L.fix[d], 0.0, ru))
    return out


def sweep3(L, r, x, flag):
    res = residual(L, r, x, L.Ps)
    red = L.parity(flag)
    e = [np.where(L.fix[d], 0.0, 1.0 / (6.0 * L.vol + L.Ps[d + 1])) for d in range(3)]
    re = [res[d + 1] * e[d] for d in range(3)]
    num = res[0] + L.vol * sum(re[d] - sh(re[d], d, 1) for d in range(3))
    den = 2.0 * L.Ps[0] - L.vol ** 2 * sum(e[d] + sh(e[d], d, 1) for d in range(3))
    dp = np.where(red & (den != 0), num / np.where(den != 0, den, 1.0), 0.0)
    out = [x[0] + dp]
    for d in range(3):
        lo, hi = red, sh(red, d, -1)  # the face is the low or the high one of a cell of the colour
        out.append(x[d + 1] + re[d] * (lo | hi) + e[d] * L.vol * (dp - sh(dp, d, -1)))
    return out


def sweep2(L, r, x, flag):
    res = residual(L, r, x, L.P)
    red = L.parity(flag)
    out = [x[0].copy(), x[1].copy(), x[2].copy()]
    z, w, fixed = [], [], []
    schur, num = L.P[0].copy(), res[0].copy()
    for d in range(2):
        fa, fb = L.fix[d], sh(L.fix[d], d, 1)
        ra, rb = res[d + 1], sh(res[d + 1], d, 1)
        da, db = 4.0 * L.lap + L.P[d + 1], 4.0 * L.lap + sh(L.P[d + 1], d, 1)
        s = np.where(fa | fb, 0.0, L.lap)
        det = da * db - s * s
        ga, gb = np.where(fa, 0.0, -L.vol), np.where(fb, 0.0, L.vol)
        inv = lambda a, b: ((db * a + s * b) / det, (s * a + da * b) / det)
        z.append(inv(ra, rb))
        w.append(inv(ga, gb))
        schur = schur - (ga * w[d][0] + gb * w[d][1])
        num = num - (ga * z[d][0] + gb * z[d][1])
    dp = np.where(red & (schur != 0), num / np.where(schur != 0, schur, 1.0), 0.0)
    out[0] += dp
    for d in range(2):
        out[d + 1] += np.where(red, z[d][0] - dp * w[d][0], 0.0)
        out[d + 1] += sh(np.where(red, z[d][1] - dp * w[d][1], 0.0), d, -1)
    return out


def restrict(L, C, res):
    out = C.zeros()
    for q in range(L.dim + 1):
        out[q][C.core] = L.children(res[q]).sum(0)
        out[q] = np.where(C.present(-1) if q == 0 else ~C.fix[q - 1], out[q], 0.0)
    return out


def bf16(a):
    b = np.asarray(a, np.float32).view(np.uint32).astype(np.uint64)
    b = (b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000
    return b.astype(np.uint32).view(np.float32).astype(np.float64)


def prolong(L, C, x, xc, linear, mixed):
    if mixed:
        xc = [bf16(a) for a in xc]
    idx = np.arange(L.n + 1) >> 1
    out = [x[0].copy()] + [a.copy() for a in x[1:]]
    for q in range(L.dim + 1):
        box = xc[q][np.ix_(*[idx + H] * L.dim)]
        if linear and q:
            box = xc[q]
            for a in range(L.dim):
                i = np.arange(L.n + 1)
                c = i >> 1
                if a == q - 1:
                    box = 0.5 * (box.take(c + H, a) + box.take(np.where(i & 1, c + 1, c) + H, a))
                else:
                    box = 0.75 * box.take(c + H, a) + 0.25 * box.take(np.where(i & 1, c + 1, c - 1) + H, a)
        add = np.zeros(L.shape)
        add[L.core] = box
        out[q] = out[q] + np.where(L.present(-1) if q == 0 else ~L.fix[q - 1], add, 0.0)
    return out


def coarsest(L, r, visc):
    """(A + e e^T) x = r, e the cells' ones (closed domain). A is singular along e alone (the 3D matrix
    has no cell penalties, as the reference's, and the 2D one gets none here), so x is A's solution
    of zero mean pressure for r without its e part, found with the first cell's pressure held at 0,
    plus e (e r) / cells^2."""
    num, count = [], 0
    for q in list(range(1, L.dim + 1)) + [0]:  # the faces first, then the cells
        m = L.present(-1) if q == 0 else ~L.fix[q - 1]
        a = np.full(L.shape, -1)
        a[m] = np.arange(count, count + int(m.sum()))
        count += int(m.sum())
        num.insert(0, a) if q == 0 else num.append(a)
    assert L.dim == 3 or not np.any(L.P[0])
    ncell = int(L.present(-1).sum())
    R, Cc, V = [], [], []

    def add(row, col, v):
        ok = (row >= 0) & (col >= 0)
        R.append(row[ok])
        Cc.append(col[ok])
        V.append(np.broadcast_to(v, row.shape)[ok].astype(float))

    for d in range(L.dim):
        u = num[d + 1]
        add(u, u, 2.0 * L.dim * visc + L.P[d + 1])
        for a in range(L.dim):
            for s in (-1, 1):
                add(u, sh(u, a, s), -visc)
        for cell, v in ((num[0], -L.vol), (sh(num[0], d, -1), L.vol)):  # the cells above and below the face
            add(u, cell, v)
            add(cell, u, v)
    A = sp.csc_matrix((np.concatenate(V), (np.concatenate(R), np.concatenate(Cc))), shape=(count,) * 2)
    b = np.zeros(count)
    for q in range(L.dim + 1):
        b[num[q][num[q] >= 0]] = r[q][num[q] >= 0]
    total = b[-ncell:].sum()
    b[-ncell:] -= total / ncell
    hold = np.arange(count) != count - ncell
    x = np.zeros(count)
    x[hold] = spl.spsolve(A[hold][:, hold], b[hold])
    x[-ncell:] += total / ncell ** 2 - x[-ncell:].mean()
    out = L.zeros()
    for q in range(L.dim + 1):
        out[q][num[q] >= 0] = x[num[q][num[q] >= 0]]
    return out


def cycle(levels, i, r, sweep, sweeps, linear, mixed, visc):
    L = levels[i]
    if i == 0:
        return coarsest(L, r, visc(L))
    C = levels[i - 1]
    x = L.zeros()
    for s in range(2 * sweeps):
        x = sweep(L, r, x, s // sweeps)
    xc = cycle(levels, i - 1, restrict(L, C, residual(L, r, x, L.P)), sweep, sweeps, linear, mixed, visc)
    x = prolong(L, C, x, xc, linear, mixed)
    for s in range(2 * sweeps):
        x = sweep(L, r, x, 1 - s // sweeps)
    return x


def run(dim, n, nlev, vol, fixed, cell_pen, face_pen, cell_r, face_r, sweeps=1, linear=False, mixed=False):
    levels = hierarchy(dim, n, nlev, vol, fixed, cell_pen, face_pen)
    F = levels[-1]
    if dim == 3:
        scale, mx = np.float32(1.0), max(np.abs(p.astype(np.float32)).max() for p in F.P)
        while mx > np.float32(32768.0) * scale:
            scale *= np.float32(2.0)
        for L in levels[::-1]:
            L.Ps = [((p.astype(np.float32) / scale).astype(np.float16).astype(np.float32) * scale).astype(np.float64) for p in L.P]
            scale *= np.float32(8.0)
    r = [F.put(-1, cell_r)] + [np.where(F.fix[d], 0.0, F.put(d, face_r[d])) for d in range(dim)]
    x = cycle(levels, nlev - 1, r, sweep3 if dim == 3 else sweep2, sweeps, linear, mixed,
              (lambda L: L.vol) if dim == 3 else (lambda L: L.lap))
    return x[0][F.box(-1)], [x[d + 1][F.box(d)] for d in range(dim)]
