"""Performance cases of the Brinkman-Stokes topology-optimization path.

Each case is work a program has the library do through its public entry points (the C ABI
of include/stokes_gb300.h and its binding stokes_to_gb300.capi):

  solve     a whole solve as a caller of FluidSteadyState{,3D} runs it: penalties and
            right-hand side from pinned host Field arrays, set-up, Krylov solve to the
            FP64 tolerance, velocities and pressure back to pinned host arrays
  design    one iteration of the optimality-criteria design loop on a host design: filter,
            penalty law, forward solve, energy, adjoint solve and sensitivity, filter
            transpose, OC update
  operator  the LinearMapping plug-ins A and E on device vectors in the blocked layout
  net       one forward and backward pass of the learned preconditioner's network

Densities are seeded smoothed noise, standardised and pushed through a logistic curve
(`contrast` its steepness: 0.1 gives the nearly uniform medium of the solve benchmarks,
0.25 to 0.5 the uneven grey media of a design loop on its way), then filtered with radius
1.5; the penalty follows the Borrvall-Petersson law with amax 1e4, the boundary is the
parabolic inlet and outlet on N/4-wide patches. Tolerances are the library's own: 1e-8 in
3D, 1e-10 in 2D.
"""
import ctypes
import math

import numpy as np
import torch

from stokes_to_gb300 import capi

RMIN = 1.5
AMAX = 1e4
FRAC = 0.4
MOVE = 0.2


def listed():
    return [
        # the smallest 3D solve in use (the tests' and smoke's size): launches and set-up
        {"name": "solve3d_16", "kind": "solve", "dim": 3, "n": 16, "method": "plain", "sigma": 2.0, "contrast": 0.5},
        # an ordinary interactive size: the coarse levels weigh as much as the finest one
        {"name": "solve3d_64", "kind": "solve", "dim": 3, "n": 64, "method": "plain", "sigma": 4.0, "contrast": 0.5},
        # the batch of 128^3 solves of the benchmark configurations
        {"name": "solve3d_128", "kind": "solve", "dim": 3, "n": 128, "method": "plain", "sigma": 4.0, "contrast": 0.1},
        # the headline benchmark's solve, host to host
        {"name": "solve3d_256", "kind": "solve", "dim": 3, "n": 256, "method": "plain", "sigma": 4.0, "contrast": 0.1},
        # BF16 coarse corrections, the mixed option's solve
        {"name": "solve3d_128_mixed", "kind": "solve", "dim": 3, "n": 128, "method": "mixed", "sigma": 4.0, "contrast": 0.1},
        # a 3D design iteration: forward and adjoint solve on an uneven grey medium
        {"name": "design3d_64", "kind": "design", "dim": 3, "n": 64, "sigma": 4.0, "contrast": 0.25},
        # the 2D design loop's iteration at the benchmark's 64^2
        {"name": "design2d_64", "kind": "design", "dim": 2, "n": 64, "sigma": 3.0, "contrast": 0.5},
        # a ragged 2D size: its coarsest level has 24^2 cells (2112 unknowns)
        {"name": "solve2d_96", "kind": "solve", "dim": 2, "n": 96, "method": "plain", "sigma": 3.0, "contrast": 0.5},
        # a large 2D solve
        {"name": "solve2d_512", "kind": "solve", "dim": 2, "n": 512, "method": "plain", "sigma": 4.0, "contrast": 0.5},
        # A and E as a caller's own Krylov or energy code applies them, on a ragged grid
        {"name": "operator3d_96", "kind": "operator", "dim": 3, "n": 96, "sigma": 4.0, "contrast": 0.5},
        # a training step's network pass
        {"name": "net_32", "kind": "net", "n": 32},
    ]


def draw(rng):
    kind = rng.choice(["solve3", "solve3", "solve3", "design3", "solve2", "solve2", "design2", "operator", "net"])
    sigma = round(rng.uniform(1.5, 5.0), 3)
    contrast = round(math.exp(rng.uniform(math.log(0.1), math.log(0.5))), 3)
    if kind == "solve3":
        n = rng.choice([16, 32, 64, 128, 256])
        return {"kind": "solve", "dim": 3, "n": n, "method": rng.choice(["plain", "plain", "mixed"]) if n < 256 else "plain",
                "sigma": sigma, "contrast": contrast if n < 128 else min(contrast, 0.3)}
    if kind == "design3":
        return {"kind": "design", "dim": 3, "n": rng.choice([16, 32, 64]), "sigma": sigma,
                "contrast": min(contrast, 0.25)}
    if kind == "solve2":
        return {"kind": "solve", "dim": 2, "n": rng.choice([16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512]), "method": "plain",
                "sigma": sigma, "contrast": contrast}
    if kind == "design2":
        return {"kind": "design", "dim": 2, "n": rng.choice([16, 32, 48, 64, 128, 256]), "sigma": sigma, "contrast": contrast}
    if kind == "operator":
        return {"kind": "operator", "dim": 3, "n": rng.choice([16, 24, 32, 48, 64, 96, 128]), "sigma": sigma, "contrast": contrast}
    return {"kind": "net", "n": rng.choice([8, 12, 16, 20, 24, 28, 32])}


# ------------------------------------------------------------------ inputs
def _face_shape(n, d, dim):
    return tuple(n + (a == d) for a in range(dim))


def _blur(a, sigma):
    r = int(math.ceil(3 * sigma))
    w = [math.exp(-t * t / (2 * sigma * sigma)) for t in range(-r, r + 1)]
    s = sum(w)
    for ax in range(a.dim()):
        n = a.shape[ax]
        base = torch.arange(n, device=a.device)
        out = torch.zeros_like(a)
        for t in range(-r, r + 1):
            out += (w[t + r] / s) * a.index_select(ax, (base + t).clamp(0, n - 1))
        a = out
    return a


def _design(case, seed):
    """Seeded design on the GPU, FP64, values in (0, 1), mean about one half."""
    dim, n = case["dim"], case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = _blur(torch.rand((n,) * dim, generator=g, device="cuda", dtype=torch.float64), case["sigma"])
    z = (z - z.mean()) / z.std()
    return torch.sigmoid(case["contrast"] * z)


def _offsets(dim):
    r = int(math.ceil(RMIN)) - 1
    rng = range(-r, r + 1)
    for o in np.ndindex(*(len(rng),) * dim):
        o = tuple(rng[q] for q in o)
        w = RMIN - math.sqrt(sum(q * q for q in o))
        if w > 0:
            yield o, w


def _shift_add(dst, src, o, w):
    """dst[c] += w src[c + o] over the cells c whose neighbour c + o lies inside."""
    n = src.shape[0]
    a = tuple(slice(max(0, -q), n - max(0, q)) for q in o)
    b = tuple(slice(max(0, q), n - max(0, -q)) for q in o)
    dst[a] += w * src[b]


def _hat(a, transpose=False):
    """The linear hat filter H (rows normalised) or its transpose."""
    ws = torch.zeros_like(a)
    for o, w in _offsets(a.dim()):
        _shift_add(ws, torch.ones_like(a), o, w)
    src = a / ws if transpose else a
    out = torch.zeros_like(a)
    for o, w in _offsets(a.dim()):
        _shift_add(out, src, o, w)
    return out if transpose else out / ws


def _penalty(phys):
    """Face penalties of the Borrvall-Petersson law, half of alpha from each adjacent cell."""
    dim, n = phys.dim(), phys.shape[0]
    a = 0.5 * AMAX * 0.1 * (1.0 - phys) / (0.1 + phys)
    out = []
    for d in range(dim):
        f = torch.zeros(_face_shape(n, d, dim), dtype=a.dtype, device=a.device)
        f.narrow(d, 1, n).add_(a)
        f.narrow(d, 0, n).add_(a)
        out.append(f)
    return out


def _inlet(dim, n):
    """Cell and face sources of the parabolic inlet (x = 0) and outlet, as numpy arrays."""
    w = n // 4
    lo = n // 2 - w // 2
    s = np.arange(lo, lo + w) + 0.5 - n / 2.0
    g = 1.0 - (2.0 * s / w) ** 2
    if dim == 3:
        g = np.outer(g, g)
    cell = np.zeros((n,) * dim)
    face = [np.zeros(_face_shape(n, d, dim)) for d in range(dim)]
    at = (slice(lo, lo + w),) * (dim - 1)
    cell[(0,) + at], cell[(n - 1,) + at] = g, -g
    face[0][(1,) + at], face[0][(n - 1,) + at] = g, g
    return cell, face


def _solver(case):
    dim, n = case["dim"], case["n"]
    method = capi.STG_METHOD_MIXED if case.get("method") == "mixed" else capi.STG_METHOD_PLAIN
    s = capi.Solver(n, dim=dim, method=method, tol=1e-8 if dim == 3 else 1e-10)
    fixed = [np.zeros(_face_shape(n, d, dim), dtype=np.int32) for d in range(dim)]
    for d in range(dim):
        np.moveaxis(fixed[d], d, 0)[[0, n]] = 1
    s.set_boundary(np.ones((n,) * dim), None, [np.ones(f.shape) for f in fixed], fixed, True)
    return s


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    return h.copy_(t)


def _table(ts):
    return (capi.DP * len(ts))(*[ctypes.cast(t.data_ptr(), capi.DP) for t in ts])


def _dptr(t):
    return ctypes.cast(t.data_ptr(), capi.DP)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        n = case["n"]
        g = torch.Generator().manual_seed(seed)
        s = capi.Solver(8)
        s.net_init(seed)
        p = torch.from_numpy(s.net_params())
        p += 0.02 * torch.rand(p.shape, generator=g) * (p == 0)  # biases as after some training
        s.net_set_params(p.numpy())
        inp = torch.randn((n ** 3, 8), generator=g)
        inp[:, 0] = torch.rand(n ** 3, generator=g)
        inp[:, 5:] = torch.rand((n ** 3, 3), generator=g)
        return {"case": case, "s": s, "inp": inp.numpy(), "target": torch.randn((n ** 3, 4), generator=g).numpy()}
    dim, n = case["dim"], case["n"]
    s = _solver(case)
    cell_b, face_b = _inlet(dim, n)
    x = _design(case, seed)
    st = {"case": case, "s": s}
    if kind == "design":
        s.set_rhs(cell_b, face_b)
        st["x"] = x.cpu().numpy()
        st["law"] = capi.alpha_bp(AMAX)
    elif kind == "operator":
        pen = [f.cpu().numpy() for f in _penalty(_hat(x))]
        s.set_penalty(None, pen)
        st["level"] = s.levels - 1
        st["in"] = _krylov_vector(n, seed)
        st["A"], st["E"] = torch.empty_like(st["in"]), torch.empty_like(st["in"])
        torch.cuda.synchronize()
    else:
        st["pen"] = [_pinned(f) for f in _penalty(_hat(x))]
        st["cell_b"], st["face_b"] = _pinned(torch.from_numpy(cell_b)), [_pinned(torch.from_numpy(f)) for f in face_b]
        st["p"] = torch.empty((n,) * dim, dtype=torch.float64, pin_memory=True)
        st["vel"] = [torch.empty(_face_shape(n, d, dim), dtype=torch.float64, pin_memory=True) for d in range(dim)]
        st["stats"] = capi.Stats()
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    kind, s = st["case"]["kind"], st["s"]
    if kind == "net":
        out, loss, grad = s.net_forward_backward(st["case"]["n"], st["inp"], st["target"])
        return {"out": out, "loss": np.float32(loss), "grad": grad}
    if kind == "design":
        law = st["law"]
        s.filter(RMIN, st["x"], want=False)
        s.set_density(None, law)
        s.solve(want=False)
        J = s.energy()
        dJ, _ = s.adjoint_sensitivity(law)
        s.filter(RMIN, None, transpose=True, want=False)
        x_new, _ = s.oc_update(RMIN, st["x"], None, FRAC, move=MOVE)
        return {"J": J, "dJ": dJ, "x_new": x_new}
    if kind == "operator":
        s.apply_A_device(st["level"], st["A"].data_ptr(), st["in"].data_ptr())
        s.apply_E_device(st["E"].data_ptr(), st["in"].data_ptr())
        return {"A": st["A"], "E": st["E"]}
    L = capi.lib()
    capi.check(L.stg_set_penalty(s.h, None, _table(st["pen"])))
    capi.check(L.stg_set_rhs(s.h, _dptr(st["cell_b"]), _table(st["face_b"])))
    capi.check(L.stg_solve(s.h, _dptr(st["p"]), _table(st["vel"]), ctypes.byref(st["stats"])))
    # the boundary is closed, so the pressure is known up to a constant: its mean is set to 0
    st["p"].sub_(st["p"].mean())
    return {"p": st["p"], "vel": st["vel"]}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: host arrays and, for a solve, one reading of the operator and one writing of
    the solution a V-cycle; the V-cycle count is the least a solve to the tolerance has
    been seen to take. A slot is a cell's pressure and its `dim` low faces."""
    if case["kind"] == "net":
        n = case["n"]
        c = [(16, 16, 1), (16, 16, 1), (16, 32, 8), (32, 32, 8), (32, 64, 64), (64, 64, 64), (96, 32, 8), (32, 32, 8), (48, 16, 1),
             (16, 16, 1)]
        flops = sum(3 * 2 * 27 * a * b * n ** 3 / q for a, b, q in c)
        return {"bytes": n ** 3 * (8 + 4 + 4) * 4 + 359813 * 8, "flops": flops}
    dim, n = case["dim"], case["n"]
    unk = n ** dim + dim * n ** (dim - 1) * (n + 1)
    if case["kind"] == "operator":
        return {"bytes": unk * 8 * 6, "flops": unk * 2 * 20}
    if case["kind"] == "design":
        return {"bytes": 2 * 10 * unk * 4 * 4 + 6 * n ** dim * 8, "flops": 2 * 10 * unk * 100}
    its = 14 if dim == 3 else 12
    return {"bytes": its * unk * 4 * 4 + 3 * unk * 8, "flops": its * unk * 100}


# ------------------------------------------------------------------ 64-bit values
def _free(n, d, dim):
    f = torch.ones(_face_shape(n, d, dim), dtype=torch.bool)
    f.select(d, 0).fill_(False)
    f.select(d, n).fill_(False)
    return f


def _viscous(u):
    """2 dim u - sum of the 2 dim neighbours, values outside the array zero."""
    out = 2.0 * u.dim() * u
    for a in range(u.dim()):
        m = u.shape[a]
        out.narrow(a, 1, m - 1).sub_(u.narrow(a, 0, m - 1))
        out.narrow(a, 0, m - 1).sub_(u.narrow(a, 1, m - 1))
    return out


def _dense(pen, dim, n):
    """The free unknowns' matrix of A (faces, then cells; the pressure block gets 1 / cells,
    which fixes the constant), on the GPU, and the free-face masks."""
    dev = "cuda"
    free = [_free(n, d, dim) for d in range(dim)]
    num, count = [], 0
    for d in range(dim):
        q = torch.full(free[d].shape, -1, dtype=torch.long)
        q[free[d]] = torch.arange(count, count + int(free[d].sum()))
        count += int(free[d].sum())
        num.append(q)
    cell = torch.arange(count, count + n ** dim).reshape((n,) * dim)
    A = torch.zeros((count + n ** dim,) * 2, dtype=torch.float64, device=dev)

    def put(r, c, v):
        ok = (r >= 0) & (c >= 0)
        A[r[ok].to(dev), c[ok].to(dev)] = v[ok].to(dev) if isinstance(v, torch.Tensor) else v

    for d in range(dim):
        put(num[d], num[d], 2.0 * dim + pen[d].cpu())
        for a in range(dim):
            m = num[d].shape[a]
            put(num[d].narrow(a, 0, m - 1), num[d].narrow(a, 1, m - 1), -1.0)
            put(num[d].narrow(a, 1, m - 1), num[d].narrow(a, 0, m - 1), -1.0)
        lo, hi = num[d].narrow(d, 0, n), num[d].narrow(d, 1, n)  # the faces below and above each cell
        put(lo, cell, -1.0)
        put(hi, cell, 1.0)
        put(cell, lo, -1.0)
        put(cell, hi, 1.0)
    A[count:, count:] += 1.0 / n ** dim
    return A, free, count


def _solve_exact(lu, free, count, cell_b, face_b, dim, n):
    b = torch.cat([torch.cat([f[m.to(f.device)] for f, m in zip(face_b, free)]), cell_b.reshape(-1)])
    x = torch.linalg.lu_solve(*lu, b[:, None])[:, 0]
    vel, at = [], 0
    for d in range(dim):
        v = torch.zeros(_face_shape(n, d, dim), dtype=torch.float64, device=x.device)
        k = int(free[d].sum())
        v[free[d].to(x.device)] = x[at:at + k]
        at += k
        vel.append(v)
    p = x[count:].reshape((n,) * dim)
    return p - p.mean(), vel


def _oc(x, dc):
    nc = x.numel()
    vw = _hat(torch.ones_like(x), transpose=True)

    def new(lam):
        xn = x * torch.sqrt(torch.clamp(-dc, min=0.0) / (vw / nc * lam))
        return torch.minimum(torch.clamp(x + MOVE, max=1.0), torch.maximum(torch.clamp(x - MOVE, min=0.0), xn))

    l1, l2 = 0.0, 1e9
    for _ in range(200):
        mid = 0.5 * (l1 + l2)
        if float((vw * new(mid)).sum()) > FRAC * nc:
            l1 = mid
        else:
            l2 = mid
        if l2 - l1 <= 1e-12 * (l1 + l2):
            break
    return new(0.5 * (l1 + l2))


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        return _net_exact(prepare(case, seed))
    dim, n = case["dim"], case["n"]
    x = _design(case, seed)
    if kind == "operator":
        return _operator_exact(case, seed, x)
    if n > (64 if dim == 2 else 16):
        return None  # a dense solve would take too long
    phys = _hat(x)
    pen = _penalty(phys)
    cell_b, face_b = _inlet(dim, n)
    cell_b, face_b = torch.from_numpy(cell_b).cuda(), [torch.from_numpy(f).cuda() for f in face_b]
    A, free, count = _dense(pen, dim, n)
    lu = torch.linalg.lu_factor(A)
    del A
    p, u = _solve_exact(lu, free, count, cell_b, face_b, dim, n)
    if kind == "solve":
        return {"p": p, "vel": u}
    ex = [torch.where(m.cuda(), _viscous(v) + f * v, torch.zeros_like(v)) for v, f, m in zip(u, pen, free)]
    J = 0.5 * sum(float((a * b).sum()) for a, b in zip(u, ex))
    _, lam = _solve_exact(lu, free, count, torch.zeros_like(p), ex, dim, n)
    dJ = torch.zeros_like(x)
    for d in range(dim):
        g = -u[d] * lam[d] + 0.5 * u[d] * u[d]
        dJ += g.narrow(d, 0, n) + g.narrow(d, 1, n)
    dJ *= 0.5 * (-AMAX * 0.1 * 1.1 / (0.1 + phys) ** 2)
    return {"J": J, "dJ": dJ, "x_new": _oc(x, _hat(dJ, transpose=True))}


# the blocked solver layout: cells in 4^3 blocks, then each axis's faces in blocks padded by
# one block along the axis
def _blocked(n):
    """Per kind (cells, x-, y-, z-faces): the stored indices of its Field-order entries, and
    the vector's length."""
    maps, off = [], 0
    idx = np.arange(n ** 3)
    nb = n // 4
    b = idx >> 6
    x, y, z = (b % nb) * 4 + (idx & 3), (b // nb % nb) * 4 + (idx >> 2 & 3), (b // nb // nb) * 4 + (idx >> 4 & 3)
    m = np.zeros((n, n, n), dtype=np.int64)
    m[x, y, z] = idx
    maps.append(torch.from_numpy(m))
    off += n ** 3
    for d in range(3):
        idx = np.arange((n + 4) * n * n)
        nbx, nby = nb + (d == 0), nb + (d == 1)
        b, q = idx >> 6, (idx & 3, idx >> 2 & 3, idx >> 4 & 3)
        x = (b % nbx) * 4 + q[2 if d == 0 else 0]
        y = (b // nbx % nby) * 4 + q[(0, 2, 1)[d]]
        z = (b // nbx // nby) * 4 + q[2 if d == 2 else 1]
        ok = (x, y, z)[d] <= n
        m = np.zeros(_face_shape(n, d, 3), dtype=np.int64)
        m[x[ok], y[ok], z[ok]] = idx[ok] + off
        maps.append(torch.from_numpy(m))
        off += len(idx)
    return maps, off


def _krylov_vector(n, seed):
    """A vector as the Krylov method of a caller holds it: zero on fixed and absent unknowns."""
    maps, size = _blocked(n)
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.zeros(size, dtype=torch.float64, device="cuda")
    for d, m in enumerate([maps[0]] + [m[_free(n, d, 3)] for d, m in enumerate(maps[1:])]):
        m = m.reshape(-1).cuda()
        v[m] = torch.randn(m.shape, generator=g, device="cuda", dtype=torch.float64)
    return v


def _operator_exact(case, seed, x):
    n = case["n"]
    maps, size = _blocked(n)
    maps = [m.cuda() for m in maps]
    v = _krylov_vector(n, seed)
    pen = _penalty(_hat(x))
    p, u = v[maps[0]], [v[m] for m in maps[1:]]
    A, E = torch.zeros_like(v), torch.zeros_like(v)
    div = torch.zeros_like(p)
    for d in range(3):
        div += u[d].narrow(d, 1, n) - u[d].narrow(d, 0, n)
        grad = torch.zeros_like(u[d])
        grad.narrow(d, 1, n - 1).copy_(p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1))
        e = _viscous(u[d]) + pen[d] * u[d]
        m = _free(n, d, 3).cuda()
        A[maps[d + 1][m]] = (e - grad)[m]
        E[maps[d + 1][m]] = e[m]
    A[maps[0].reshape(-1)] = div.reshape(-1)
    return {"A": A, "E": E}


def _net_exact(st):
    n = st["case"]["n"]
    conv = torch.nn.functional.conv3d
    cin = [16, 16, 16, 32, 32, 64, 96, 32, 48, 16]
    cout = [16, 16, 32, 32, 64, 64, 32, 32, 16, 16]
    P = torch.from_numpy(st["s"].net_params()).double().requires_grad_(True)
    at, W, B = 0, [], []
    for a, b in zip(cin, cout):
        W.append(P[at:at + 27 * a * b].reshape(3, 3, 3, b, a).permute(3, 4, 0, 1, 2))
        B.append(P[at + 27 * a * b:at + 27 * a * b + b])
        at += 27 * a * b + b
    hw, hb = P[at:at + 64].reshape(4, 16), P[at + 64:at + 68]
    x = torch.zeros(1, 16, n, n, n, dtype=torch.float64)
    x[0, :8] = torch.from_numpy(st["inp"]).double().reshape(n, n, n, 8).permute(3, 0, 1, 2)

    def layer(l, a):
        return torch.relu(conv(a, W[l], B[l], padding=1))

    def up(a):
        return torch.nn.functional.interpolate(a, scale_factor=2, mode="nearest")

    pool = torch.nn.functional.avg_pool3d
    s0 = layer(1, layer(0, x))
    s1 = layer(3, layer(2, pool(s0, 2)))
    b2 = layer(5, layer(4, pool(s1, 2)))
    b1 = layer(7, layer(6, torch.cat([up(b2), s1], 1)))
    b0 = layer(9, layer(8, torch.cat([up(b1), s0], 1)))
    out = torch.einsum("bcijk,oc->bijko", b0, hw) + hb
    t = torch.from_numpy(st["target"]).double().reshape(1, n, n, n, 4)
    loss = ((out - t) ** 2).sum() / (t ** 2).sum()
    loss.backward()
    return {"out": out.detach().reshape(-1, 4), "loss": loss.detach(), "grad": P.grad}
