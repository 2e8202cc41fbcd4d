// 2D path (dim = 2) of libstokes_gb300.
//
// The 2D configuration is small (64^2: 13,312 unknowns) and latency-bound, so its
// vectors stay in the reference's own 8x8-blocked solver layout
// [cells | x-faces | y-faces] (common_cpx/form01mapping.cu:10-57) and every kernel is a
// thread per unknown. The algorithm is the reference's 2D one:
//   A          stoke/StokeFlowMapping.cu:30-139 (grad-div, node-based curl-curl on the raw
//              velocity, -grad p, div, penalty; no definite fix: fixed rows are zero)
//   E          fluid_topo/FluidEnergyGrad.cu:30-61 (5-point face Laplacian + P x)
//   coarsening stoke/StokeFlowSubSystem.cu:100-160 (lap_coeff doubles per level)
//   smoother   stoke/StokeFlowSmoothing.cu:8-209 (5-unknown box with two 2x2 velocity
//              blocks, colours (x + y + flag) even, r-form with a residual update per colour)
//   coarsest   stoke/StokeFlowDirectSolve.cpp:6-133 (analytic dense matrix), inverted on
//              the GPU by blocks (dense.cu; pivoted where cells are fixed), applied as a GEMV
//   V-cycle    common_cpx/MultigridSolve.cpp:73-106 in FP32; Krylov as in 3D (solve_core).
#include <cooperative_groups.h>

#include <cmath>
#include <vector>

#include "alpha.cuh"
#include "ctx.h"
#include "rowdot.cuh"

namespace stg {

namespace {

constexpr int TPB = 256;

// common_cpx/form01mapping.cu:10-57 (faces padded by 8 along their normal)
struct G2d {
    int n = 0;
    __host__ __device__ int nc() const { return n * n; }
    __host__ __device__ int fs(int d) const { return (n + 8 * (d == 0)) * (n + 8 * (d == 1)); }
    __host__ __device__ int size() const { return nc() + fs(0) + fs(1); }
    __host__ __device__ int off(int d) const { return nc() + (d == 1 ? fs(0) : 0); }
    __host__ __device__ int cell(int x, int y) const { return ((y >> 3) * (n >> 3) + (x >> 3)) * 64 + ((y & 7) * 8 + (x & 7)); }
    __host__ __device__ int face(int x, int y, int d) const {
        int b = (y >> 3) * ((n >> 3) + (d == 0)) + (x >> 3);
        int ix = x & 7, iy = y & 7;
        return off(d) + b * 64 + (d == 0 ? ix * 8 + iy : iy * 8 + ix);
    }
    __host__ __device__ bool cell_ok(int x, int y) const { return x >= 0 && y >= 0 && x < n && y < n; }
    __host__ __device__ bool face_ok(int x, int y, int d) const {
        return x >= 0 && y >= 0 && (d == 0 ? (x <= n && y < n) : (x < n && y <= n));
    }
    // stored index -> kind (-1 cell, 0/1 face axis) and coordinates
    __host__ __device__ void decode(int t, int& kind, int& x, int& y) const {
        if (t < nc()) {
            kind = -1;
            int b = t >> 6, ix = t & 7, iy = (t >> 3) & 7;
            x = (b % (n >> 3)) * 8 + ix;
            y = (b / (n >> 3)) * 8 + iy;
            return;
        }
        t -= nc();
        int d = t < fs(0) ? 0 : 1;
        if (d == 1) t -= fs(0);
        int b = t >> 6, i = t & 63;
        int nbx = (n >> 3) + (d == 0);
        int ix = d == 0 ? i >> 3 : i & 7, iy = d == 0 ? i & 7 : i >> 3;
        kind = d;
        x = (b % nbx) * 8 + ix;
        y = (b / nbx) * 8 + iy;
    }
};

// ------------------------------------------------------------------ operator rows
template <class T>
struct Coef2 {
    const T* vol;
    const T* pen;
    const uint8_t* fixed;
};

template <class T>
__device__ __forceinline__ T fval(const G2d& g, const T* v, int x, int y, int d) {
    return g.face_ok(x, y, d) ? v[g.face(x, y, d)] : T(0);
}
template <class T>
__device__ __forceinline__ T vval(const G2d& g, const Coef2<T>& C, const T* v, int x, int y, int d) {
    if (!g.face_ok(x, y, d)) return T(0);
    int i = g.face(x, y, d);
    return C.vol[i] * v[i];
}
// fix_c D (V u) of cell (x, y); 0 outside the grid
template <class T>
__device__ __forceinline__ T divp(const G2d& g, const Coef2<T>& C, const T* v, int x, int y) {
    if (!g.cell_ok(x, y) || C.fixed[g.cell(x, y)]) return T(0);
    return (vval(g, C, v, x + 1, y, 0) - vval(g, C, v, x, y, 0)) + (vval(g, C, v, x, y + 1, 1) - vval(g, C, v, x, y, 1));
}
// node(x,y) = u(x,y-1) - u(x,y) - v(x-1,y) + v(x,y) on the raw velocity (form01mapping.cu:256-300)
template <class T>
__device__ __forceinline__ T node(const G2d& g, const T* v, int x, int y) {
    return fval(g, v, x, y - 1, 0) - fval(g, v, x, y, 0) - fval(g, v, x - 1, y, 1) + fval(g, v, x, y, 1);
}
template <class T>
__device__ __forceinline__ T cval(const G2d& g, const T* v, int x, int y) {
    return g.cell_ok(x, y) ? v[g.cell(x, y)] : T(0);
}

// one row of A (MODE 0), b - A x (MODE 1) or E (MODE 2, lap = lap_coeff of the energy)
template <class T, int MODE>
__device__ __forceinline__ T row(const G2d& g, const Coef2<T>& C, T lap, const T* v, int t) {
    int kind, x, y;
    g.decode(t, kind, x, y);
    const T pen = C.pen[t];
    if (kind < 0) {
        T out = pen * v[t];
        if (MODE != 2) out += divp(g, C, v, x, y);
        return out;
    }
    const int d = kind;
    if (!g.face_ok(x, y, d) || C.fixed[t]) return pen * v[t];  // zero rows (pen is 0 there)
    if (MODE == 2) {
        // 5-point Laplacian over the stored face array (faceLapMapping, form01mapping.cu:430-525)
        const int X = d == 0 ? g.n + 8 : g.n, Y = d == 0 ? g.n : g.n + 8;
        auto F = [&](int a, int b) { return (a >= 0 && b >= 0 && a < X && b < Y) ? v[g.face(a, b, d)] : T(0); };
        T l = T(4) * v[t] - F(x - 1, y) - F(x + 1, y) - F(x, y - 1) - F(x, y + 1);
        return lap * l + pen * v[t];
    }
    const T vol = C.vol[t];
    T gd, cc, gp;
    if (d == 0) {
        gd = -(divp(g, C, v, x, y) - divp(g, C, v, x - 1, y));
        cc = vol * (node(g, v, x, y + 1) - node(g, v, x, y));
        gp = vol * (cval(g, v, x, y) - cval(g, v, x - 1, y));
    } else {
        gd = -(divp(g, C, v, x, y) - divp(g, C, v, x, y - 1));
        cc = vol * (-(node(g, v, x + 1, y) - node(g, v, x, y)));
        gp = vol * (cval(g, v, x, y) - cval(g, v, x, y - 1));
    }
    return gd + cc - gp + pen * v[t];
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <class T, int MODE>
__global__ void k2_apply(G2d g, Coef2<T> C, T lap, const T* __restrict__ v, const T* __restrict__ b, T* __restrict__ out,
                         double* __restrict__ part) {
    __shared__ double sh[TPB / 32];
    int t = blockIdx.x * TPB + threadIdx.x;
    double acc = 0;
    if (t < g.size()) {
        T o = row<T, MODE == 1 ? 0 : MODE>(g, C, lap, v, t);
        if (MODE == 1) {
            o = b[t] - o;
            acc = (double)o * o;
        } else if (MODE == 2) {
            acc = (double)v[t] * o;
        }
        out[t] = o;
    }
    if (part) {
        acc = warp_sum(acc);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0;
            for (int w = 0; w < TPB / 32; w++) s += sh[w];
            part[blockIdx.x] = s;
        }
    }
}

// ------------------------------------------------------------------ smoother colour
// One colour of the 2D box smoother (the operator of stoke/StokeFlowSmoothing.cu:74-140):
// every cell of the colour solves for its 5 unknowns - the x-faces a (low) and b (high),
// the y-faces c (low) and d (high), the pressure p - with the box matrix
//
//     | K    g  |  | u |   | r_u |       K = diag(K_x, K_y),  K_x = | 4L+P_a   -s_x |
//     | g^T  P_p|  | p | = | r_p |                                  | -s_x   4L+P_b |
//
// where L is the level's Laplacian coefficient, s_x = L unless face a or b is fixed (0
// then), K_y likewise, and g = (-vol_a, vol_b, -vol_c, vol_d) holds the divergence
// weights. Block elimination: z = K^-1 r_u, w = K^-1 g, p = (r_p - g.z) / (P_p - g.w),
// u = z - p w; a fixed cell keeps p = 0. Each 2x2 block of K is inverted once and applied
// to both right-hand sides.
struct SymInv2 {
    float i00, i01, i11;  // inverse of [[d0, -s], [-s, d1]]
    __device__ __forceinline__ SymInv2(float d0, float d1, float s) {
        const float rdet = 1.f / (d0 * d1 - s * s);
        i00 = d1 * rdet;
        i11 = d0 * rdet;
        i01 = s * rdet;
    }
    __device__ __forceinline__ void apply(float v0, float v1, float& o0, float& o1) const {
        o0 = i00 * v0 + i01 * v1;
        o1 = i01 * v0 + i11 * v1;
    }
};

__global__ void k2_smooth(G2d g, Coef2<float> C, float lap, int flag, const float* __restrict__ r, float* __restrict__ dout) {
    const int c = blockIdx.x * TPB + threadIdx.x;
    if (c >= g.nc()) return;
    const int x = (c / 64 % (g.n >> 3)) * 8 + (c & 7), y = (c / 64 / (g.n >> 3)) * 8 + ((c >> 3) & 7);
    if ((((x & 1) ^ (y & 1) ^ flag)) != 0) return;
    const int fa = g.face(x, y, 0), fb = g.face(x + 1, y, 0), fc = g.face(x, y, 1), fd = g.face(x, y + 1, 1);
    const int cp = g.cell(x, y);
    const float sx = (C.fixed[fa] || C.fixed[fb]) ? 0.f : lap;
    const float sy = (C.fixed[fc] || C.fixed[fd]) ? 0.f : lap;
    const SymInv2 Kx(4.f * lap + C.pen[fa], 4.f * lap + C.pen[fb], sx);
    const SymInv2 Ky(4.f * lap + C.pen[fc], 4.f * lap + C.pen[fd], sy);
    const float ga = -C.vol[fa], gb = C.vol[fb], gc = -C.vol[fc], gd = C.vol[fd];
    float za, zb, zc, zd, wa, wb, wc, wd;
    Kx.apply(r[fa], r[fb], za, zb);
    Ky.apply(r[fc], r[fd], zc, zd);
    Kx.apply(ga, gb, wa, wb);
    Ky.apply(gc, gd, wc, wd);
    const float schur = C.pen[cp] - (ga * wa + gb * wb + gc * wc + gd * wd);
    const float rhs_p = r[cp] - (ga * za + gb * zb + gc * zc + gd * zd);
    const float p = C.fixed[cp] ? 0.f : rhs_p / schur;
    dout[fa] = za - p * wa;
    dout[fb] = zb - p * wb;
    dout[fc] = zc - p * wc;
    dout[fd] = zd - p * wd;
    dout[cp] = p;
}

// ------------------------------------------------------------------ transfers and coarsening
// children of a coarse unknown: (2X + a, 2Y + b), order (0,0), (1,0), (0,1), (1,1)
template <class T>
__global__ void k2_restrict(G2d gc, G2d gf, const T* __restrict__ rf, const uint8_t* __restrict__ cfixed, T* __restrict__ rc) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= gc.size()) return;
    int kind, X, Y;
    gc.decode(t, kind, X, Y);
    T s = 0;
    for (int q = 0; q < 4; q++) {
        int x = 2 * X + (q & 1), y = 2 * Y + (q >> 1);
        if (kind < 0)
            s += rf[gf.cell(x, y)];
        else if (gf.face_ok(x, y, kind))
            s += rf[gf.face(x, y, kind)];
    }
    rc[t] = cfixed[t] ? T(0) : s;
}

template <class T>
__global__ void k2_prolong(G2d gf, G2d gc, const T* __restrict__ xc, const uint8_t* __restrict__ ffixed, T* __restrict__ xf) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= gf.size()) return;
    int kind, x, y;
    gf.decode(t, kind, x, y);
    T v = 0;
    if (kind < 0)
        v = xc[gc.cell(x >> 1, y >> 1)];
    else if (gf.face_ok(x, y, kind))
        v = xc[gc.face(x >> 1, y >> 1, kind)];
    xf[t] = ffixed[t] ? T(0) : v;
}

// finish(): padded faces fixed, vol and penalty zero on fixed (stoke/StokeFlowDescriptor.cpp:40-46)
__device__ __forceinline__ bool padded2(const G2d& g, int kind, int x, int y) {
    return kind >= 0 && !g.face_ok(x, y, kind);
}

// FLOW (the solver's own hierarchy): a coarse face takes 4 x the smallest penalty of its
// children instead of the sum, so channels narrower than a coarse cell stay open on the
// coarse levels (the 3D k_coarsen gives the reason; oracle/oracle2d.cpp flow_penalties
// restates the rule).
template <bool FLOW>
__global__ void k2_coarsen(G2d gc, G2d gf, const uint8_t* __restrict__ ff, const double* __restrict__ fvol,
                           const double* __restrict__ fpen, uint8_t* __restrict__ cf, double* __restrict__ cvol,
                           double* __restrict__ cpen, float* __restrict__ cvol32, float* __restrict__ cpen32) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= gc.size()) return;
    int kind, X, Y;
    gc.decode(t, kind, X, Y);
    uint8_t fx = 0;
    double v = 0, p = 0, lo = INFINITY;
    for (int q = 0; q < 4; q++) {
        int x = 2 * X + (q & 1), y = 2 * Y + (q >> 1);
        int i;
        if (kind < 0)
            i = gf.cell(x, y);
        else if (gf.face_ok(x, y, kind))
            i = gf.face(x, y, kind);
        else
            continue;
        fx |= ff[i];
        p += fpen[i];
        lo = fmin(lo, fpen[i]);
        // cells: sum of 4; faces: the 2 coincident children (zero offset along the normal)
        bool coincident = kind < 0 || (kind == 0 ? (q & 1) == 0 : (q >> 1) == 0);
        if (coincident) v += fvol[i];
    }
    if (FLOW && kind >= 0 && lo < INFINITY) p = 4.0 * lo;
    if (padded2(gc, kind, X, Y)) fx = 1;
    if (fx) v = p = 0;
    cf[t] = fx;
    cvol[t] = v;
    cpen[t] = p;
    cvol32[t] = (float)v;
    cpen32[t] = (float)p;
}

// fine descriptor from Field-order host inputs (staged on the device). flags (pinned host memory):
// flags[0] becomes 1 when a cell is fixed, flags[1] when a face on the domain boundary is free or a
// free face's vol is not fv
__global__ void k2_fine_descr(G2d g, const double* __restrict__ cvol, const int* __restrict__ cfix, const double* __restrict__ fv0,
                              const double* __restrict__ fv1, const int* __restrict__ ff0, const int* __restrict__ ff1, double fv,
                              uint8_t* __restrict__ fixed, double* __restrict__ vol, int* __restrict__ flags) {
    int t = blockIdx.x * TPB + threadIdx.x;
    bool cell_fixed = false, uneven = false;
    if (t < g.size()) {
        int kind, x, y;
        g.decode(t, kind, x, y);
        const int n = g.n;
        uint8_t f = 0;
        double v = 0;
        if (kind < 0) {
            f = cfix ? (cfix[x * n + y] != 0) : 0;
            v = cvol ? cvol[x * n + y] : 0.0;
            cell_fixed = f;
        } else if (g.face_ok(x, y, kind)) {
            int idx = kind == 0 ? x * n + y : x * (n + 1) + y;
            f = (kind == 0 ? ff0 : ff1)[idx] != 0;
            v = (kind == 0 ? fv0 : fv1)[idx];
            const int c = kind == 0 ? x : y;
            uneven = !f && (c == 0 || c == n || !(v == fv));
        } else {
            f = 1;
        }
        fixed[t] = f;
        vol[t] = f ? 0.0 : v;
    }
    const int any_fixed = __syncthreads_or(cell_fixed), any_uneven = __syncthreads_or(uneven);
    if (threadIdx.x == 0) {
        if (any_fixed) flags[0] = 1;
        if (any_uneven) flags[1] = 1;
    }
}

__global__ void k2_penalty_from_field(G2d g, const double* __restrict__ cp, const double* __restrict__ f0,
                                      const double* __restrict__ f1, const uint8_t* __restrict__ fixed,
                                      double* __restrict__ pen, float* __restrict__ pen32) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= g.size()) return;
    int kind, x, y;
    g.decode(t, kind, x, y);
    const int n = g.n;
    double v = 0;
    if (kind < 0)
        v = cp ? cp[x * n + y] : 0.0;
    else if (g.face_ok(x, y, kind))
        v = (kind == 0 ? f0 : f1) ? (kind == 0 ? f0 : f1)[kind == 0 ? x * n + y : x * (n + 1) + y] : 0.0;
    if (fixed[t]) v = 0;
    pen[t] = v;
    pen32[t] = (float)v;
}

__global__ void k2_field_to_blocked(G2d g, const double* __restrict__ cell, const double* __restrict__ f0,
                                    const double* __restrict__ f1, double* __restrict__ out) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= g.size()) return;
    int kind, x, y;
    g.decode(t, kind, x, y);
    const int n = g.n;
    double v = 0;
    if (kind < 0)
        v = cell ? cell[x * n + y] : 0.0;
    else if (g.face_ok(x, y, kind)) {
        const double* f = kind == 0 ? f0 : f1;
        v = f ? f[kind == 0 ? x * n + y : x * (n + 1) + y] : 0.0;
    }
    out[t] = v;
}

__global__ void k2_blocked_to_field(G2d g, const double* __restrict__ in, double* __restrict__ cell, double* __restrict__ f0,
                                    double* __restrict__ f1) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= g.size()) return;
    int kind, x, y;
    g.decode(t, kind, x, y);
    const int n = g.n;
    if (kind < 0) {
        if (cell) cell[x * n + y] = in[t];
    } else if (g.face_ok(x, y, kind)) {
        double* f = kind == 0 ? f0 : f1;
        if (f) f[kind == 0 ? x * n + y : x * (n + 1) + y] = in[t];
    }
}

// face penalty = 1/2 alpha(left cell) + 1/2 alpha(right cell), zero on fixed
// (fluid_topo/FluidTopoOpt.cpp:143-160)
__global__ void k2_face_penalty(G2d g, const double* __restrict__ rho, stg_alpha L, const uint8_t* __restrict__ fixed,
                                double* __restrict__ pen, float* __restrict__ pen32) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= g.size()) return;
    int kind, x, y;
    g.decode(t, kind, x, y);
    const int n = g.n;
    double v = 0;
    if (kind >= 0 && g.face_ok(x, y, kind)) {
        int lx = x - (kind == 0), ly = y - (kind == 1);
        double lo = g.cell_ok(lx, ly) ? 0.5 * alpha_of(rho[lx * n + ly], L) : 0.0;
        double hi = g.cell_ok(x, y) ? 0.5 * alpha_of(rho[x * n + y], L) : 0.0;
        v = lo + hi;
    }
    if (fixed[t]) v = 0;
    pen[t] = v;
    pen32[t] = (float)v;
}

// dJ/drho = 1/2 alpha'(rho) sum over the 4 faces of (-u lambda + 1/2 u^2)
// (fluid_topo/FluidTopoOpt.cpp:166-190)
__global__ void k2_sensitivity(G2d g, const double* __restrict__ rho, stg_alpha L, const double* __restrict__ u,
                               const double* __restrict__ lam, double* __restrict__ grad) {
    int t = blockIdx.x * TPB + threadIdx.x;
    const int n = g.n;
    if (t >= n * n) return;
    int x = t / n, y = t % n;
    const int fi[4] = {g.face(x, y, 0), g.face(x + 1, y, 0), g.face(x, y, 1), g.face(x, y + 1, 1)};
    double s = 0;
    for (int q = 0; q < 4; q++) s += -(u[fi[q]] * lam[fi[q]]) + (0.5 * u[fi[q]]) * u[fi[q]];
    grad[t] = s * (0.5 * dalpha_of(rho[t], L));
}

// calcA (stoke/StokeFlowDirectSolve.cpp:6-133) as a function of the entry (row i, col j),
// written into row i of the row-major augmented matrix [A | I] (ld = 2 nd)
__global__ void k2_calcA(G2d g, const double* __restrict__ vol, const double* __restrict__ pen,
                         const uint8_t* __restrict__ fixed, double lap, int closed, double* __restrict__ aug) {
    const int nd = g.size();
    long long e = (long long)blockIdx.x * TPB + threadIdx.x;
    if (e >= (long long)nd * nd) return;
    int i = (int)(e / nd), j = (int)(e % nd);
    double a = 0;
    if (fixed[i] || fixed[j]) {
        a = i == j ? 1.0 : 0.0;
    } else {
        int ki, xi, yi, kj, xj, yj;
        g.decode(i, ki, xi, yi);
        g.decode(j, kj, xj, yj);
        if (ki < 0 && kj < 0) {
            a = closed ? 1.0 : 0.0;
        } else if (ki < 0 || kj < 0) {
            // cell-face coupling: -vol (left / bottom face), +vol (right / top face)
            int cx = ki < 0 ? xi : xj, cy = ki < 0 ? yi : yj;
            int fk = ki < 0 ? kj : ki, fxx = ki < 0 ? xj : xi, fyy = ki < 0 ? yj : yi;
            int fidx = ki < 0 ? j : i;
            if (g.face_ok(fxx, fyy, fk)) {
                if (fk == 0 && fyy == cy && fxx == cx) a = -vol[fidx];
                if (fk == 0 && fyy == cy && fxx == cx + 1) a = vol[fidx];
                if (fk == 1 && fxx == cx && fyy == cy) a = -vol[fidx];
                if (fk == 1 && fxx == cx && fyy == cy + 1) a = vol[fidx];
            }
        } else if (ki == kj && g.face_ok(xi, yi, ki) && g.face_ok(xj, yj, kj)) {
            int dx = xj - xi, dy = yj - yi;
            const int d = ki;
            if (dx == 0 && dy == 0) {
                a = 4.0 * lap;
            } else if (abs(dx) + abs(dy) == 1) {
                // the column face's neighbour list (its x / y range limits) decides the entry
                bool ok;
                if (d == 0)
                    ok = (dx == 1 && xj != 0) || (dx == -1 && xj != g.n) || (dy == 1 && yj != 0) || (dy == -1 && yj != g.n - 1);
                else
                    ok = (dy == 1 && yj != 0) || (dy == -1 && yj != g.n) || (dx == 1 && xj != 0) || (dx == -1 && xj != g.n - 1);
                if (ok) a = -lap;
            }
        }
        if (i == j) a += pen[i];
    }
    aug[(long long)i * 2 * nd + j] = a;
    aug[(long long)i * 2 * nd + nd + j] = i == j ? 1.0 : 0.0;
}

// x = Ainv r (warp per row), FP32 in/out
__global__ void k2_gemv(int nd, const double* __restrict__ inv, int ld, const float* __restrict__ r, float* __restrict__ x) {
    int row = (blockIdx.x * TPB + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= nd) return;
    double s = 0;
    for (int c = lane; c < nd; c += 32) s += inv[(long long)row * ld + c] * (double)r[c];
    s = warp_sum(s);
    if (lane == 0) x[row] = (float)s;
}
__global__ void k2_gemv64(int nd, const double* __restrict__ inv, int ld, const double* __restrict__ r, double* __restrict__ x) {
    int row = (blockIdx.x * TPB + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= nd) return;
    double s = 0;
    for (int c = lane; c < nd; c += 32) s += inv[(long long)row * ld + c] * r[c];
    s = warp_sum(s);
    if (lane == 0) x[row] = s;
}

// x += p; r -= Ap
__global__ void k2_update(int n, const float* __restrict__ p, const float* __restrict__ Ap, float* __restrict__ x,
                          float* __restrict__ r) {
    int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= n) return;
    x[t] += p[t];
    r[t] -= Ap[t];
}

unsigned g1(long long n) { return (unsigned)((n + TPB - 1) / TPB); }

// ------------------------------------------------------------------ Laplacian-form V-cycle
// Where every boundary face is fixed, no cell is and the free faces share one vol, A is vol x
// (the 5-point face Laplacian - grad p) + penalty on vectors that are zero on fixed faces (the
// edge-diagonal terms of grad-div and curl-curl cancel, as in 3D), so the solver's own V-cycle
// runs the smoother in correction form, x <- x + P_c (r - A x), one thread per cell of the
// colour: its pressure and four faces are exactly the unknowns the box solve changes. A level
// takes five passes (two sweeps, the restricted residual, two sweeps of which the first adds
// the prolonged correction on reading) instead of 28 kernels, copies and memsets.
//
// Vectors are row-major with a zero halo, by component (p, u, v), so neighbours lie at fixed
// offsets: value (x, y) of a component at (y + 1) S + x + 1. The finest right-hand side and
// result are converted on the way in and out.
struct Lv2 {
    int n, S, NS;  // cells per axis, row stride, component stride
    float vol, lap;
    const float* P;    // penalties (3 NS; 0 on fixed faces)
    const uint8_t* m;  // NS: bit 0 u fixed, bit 1 v fixed
    float *r, *xa, *xb;  // 3 NS each
    __device__ int at(int x, int y) const { return (y + 1) * S + x + 1; }
};
constexpr int MAXL2 = 12;
struct V2 {
    Lv2 lv[MAXL2];
    G2d fine;
    int L;
    const double* inv;  // coarsest inverse, row stride ld, blocked coarse order
    float2* inv2;       // its entries as sums of two floats, nd x nd (k2v_cycle; null: not used)
    int nd, ld;
    const int* map;     // blocked coarse index -> padded offset (-1: padding)
};

// padded offset (component included) of blocked index t, or -1
__device__ __forceinline__ int pad_index(const G2d& g, const Lv2& L, int t) {
    int kind, x, y;
    g.decode(t, kind, x, y);
    if (kind >= 0 && !g.face_ok(x, y, kind)) return -1;
    return (kind + 1) * L.NS + L.at(x, y);
}
__global__ void k2_pad_index(G2d g, Lv2 L, int* __restrict__ map) {
    const int t = blockIdx.x * TPB + threadIdx.x;
    if (t < g.size()) map[t] = pad_index(g, L, t);
}
__global__ void k2_pad_coef(G2d g, Lv2 L, const float* __restrict__ pen, const uint8_t* __restrict__ fixed, float* __restrict__ P,
                            uint8_t* __restrict__ m) {
    const int t = blockIdx.x * TPB + threadIdx.x;
    if (t >= L.n * L.n) return;  // the faces at x, y = n are fixed: 0 penalty (as allocated), never updated
    const int x = t % L.n, y = t / L.n, a = L.at(x, y);
    const int f0 = g.face(x, y, 0), f1 = g.face(x, y, 1);
    P[a] = pen[g.cell(x, y)];
    P[L.NS + a] = pen[f0];
    P[2 * L.NS + a] = pen[f1];
    m[a] = (uint8_t)((fixed[f0] ? 1 : 0) | (fixed[f1] ? 2 : 0));
}

// x and r change while the one-launch V-cycle runs: read through L2
__device__ __forceinline__ float ldv2(const float* p) { return __ldcg(p); }

// One colour of the smoother, cells t0, t0 + step, ...: xo = x + P_c (r - A x); HX false: x = 0.
// PRO: x is first corrected by the parent values of xc on level C (a fixed face's parent is
// fixed, so its value is 0). The other colour's pressures are copied. SM: the level's vectors and
// coefficients are in shared memory; CS: xc is. IN (red, x = 0): r comes from the blocked vector
// of g instead, and goes to L.r on the way; OUT (red): the result goes to the blocked vector xo.
// Either leaves out the faces on the domain boundary that lie at black cells (fixed: r is 0 there
// and so is x; out_border).
template <bool HX, bool PRO, bool SM = false, bool CS = SM, bool IN = false, bool OUT = false>
__device__ __forceinline__ void sweep2(const Lv2& L, int flag, const float* x, const Lv2& C, const float* xc, float* xo, int t0,
                                       int step, const G2d g = G2d(), const float* blocked = nullptr) {
    const int h = L.n >> 1, S = L.S, NS = L.NS;
    auto var = [](const float* p) { return SM ? *p : ldv2(p); };
    auto coef = [](const float* p) { return SM ? *p : __ldg(p); };
    auto mask = [](const uint8_t* p) { return SM ? *p : __ldg(p); };
    for (int t = t0; t < L.n * h; t += step) {
        const int y = t / h, xx = 2 * (t - y * h) + ((y + flag) & 1);
        const int i = L.at(xx, y);
        const int ob = (xx & 1) ? i - 1 : i + 1;  // the pair's other cell
        auto V = [&](int c, int a, int b) {
            float v = var(x + c * NS + i + b * S + a);
            if (PRO) {
                const float* e = xc + c * C.NS + C.at((xx + a) >> 1, (y + b) >> 1);
                v += CS ? *e : ldv2(e);
            }
            return v;
        };
        const uint8_t m0 = mask(L.m + i), m1 = mask(L.m + i + 1), m2 = mask(L.m + i + S);
        const bool fa = m0 & 1, fb = (m1 & 1) || xx + 1 == L.n, fc = m0 & 2, fd = (m2 & 2) || y + 1 == L.n;
        const float Pp = coef(L.P + i), Pa = coef(L.P + NS + i), Pb = coef(L.P + NS + i + 1), Pc = coef(L.P + 2 * NS + i),
                    Pd = coef(L.P + 2 * NS + i + S);
        float rp, ra, rb, rc, rd;
        if (IN) {
            rp = __ldg(blocked + g.cell(xx, y));
            ra = __ldg(blocked + g.face(xx, y, 0));
            rb = __ldg(blocked + g.face(xx + 1, y, 0));
            rc = __ldg(blocked + g.face(xx, y, 1));
            rd = __ldg(blocked + g.face(xx, y + 1, 1));
            L.r[i] = rp;
            L.r[ob] = __ldg(blocked + g.cell(xx ^ 1, y));
            L.r[NS + i] = ra;
            L.r[NS + i + 1] = rb;
            L.r[2 * NS + i] = rc;
            L.r[2 * NS + i + S] = rd;
        } else {
            rp = var(L.r + i);
            ra = var(L.r + NS + i);
            rb = var(L.r + NS + i + 1);
            rc = var(L.r + 2 * NS + i);
            rd = var(L.r + 2 * NS + i + S);
        }
        float p = 0.f, ua = 0.f, ub = 0.f, vc = 0.f, vd = 0.f, pb = 0.f;
        if (HX) {
            p = V(0, 0, 0);
            const float pl = V(0, -1, 0), pr = V(0, 1, 0), pd = V(0, 0, -1), pu = V(0, 0, 1);
            pb = (xx & 1) ? pl : pr;
            ua = V(1, 0, 0);
            ub = V(1, 1, 0);
            vc = V(2, 0, 0);
            vd = V(2, 0, 1);
            const float la = 4.f * ua - (V(1, -1, 0) + ub) - (V(1, 0, -1) + V(1, 0, 1));
            const float lb = 4.f * ub - (ua + V(1, 2, 0)) - (V(1, 1, -1) + V(1, 1, 1));
            const float lc = 4.f * vc - (V(2, -1, 0) + V(2, 1, 0)) - (V(2, 0, -1) + vd);
            const float ld = 4.f * vd - (V(2, -1, 1) + V(2, 1, 1)) - (vc + V(2, 0, 2));
            rp -= L.vol * ((ub - ua) + (vd - vc)) + Pp * p;
            ra -= L.vol * (la - (p - pl)) + Pa * ua;
            rb -= L.vol * (lb - (pr - p)) + Pb * ub;
            rc -= L.vol * (lc - (p - pd)) + Pc * vc;
            rd -= L.vol * (ld - (pu - p)) + Pd * vd;
        }
        if (fa) ra = 0.f;
        if (fb) rb = 0.f;
        if (fc) rc = 0.f;
        if (fd) rd = 0.f;
        // the box solve of k2_smooth
        const SymInv2 Kx(4.f * L.lap + Pa, 4.f * L.lap + Pb, (fa || fb) ? 0.f : L.lap);
        const SymInv2 Ky(4.f * L.lap + Pc, 4.f * L.lap + Pd, (fc || fd) ? 0.f : L.lap);
        const float ga = fa ? 0.f : -L.vol, gb = fb ? 0.f : L.vol, gc = fc ? 0.f : -L.vol, gd = fd ? 0.f : L.vol;
        float za, zb, zc, zd, wa, wb, wc, wd;
        Kx.apply(ra, rb, za, zb);
        Ky.apply(rc, rd, zc, zd);
        Kx.apply(ga, gb, wa, wb);
        Ky.apply(gc, gd, wc, wd);
        const float schur = Pp - (ga * wa + gb * wb + gc * wc + gd * wd);
        const float num = rp - (ga * za + gb * zb + gc * zc + gd * zd);
        const float dp = schur != 0.f ? num / schur : 0.f;  // a cell between four fixed faces keeps its pressure
        xo[OUT ? g.cell(xx, y) : i] = p + dp;
        xo[OUT ? g.cell(xx ^ 1, y) : ob] = pb;
        xo[OUT ? g.face(xx, y, 0) : NS + i] = ua + (za - dp * wa);
        xo[OUT ? g.face(xx + 1, y, 0) : NS + i + 1] = ub + (zb - dp * wb);
        xo[OUT ? g.face(xx, y, 1) : 2 * NS + i] = vc + (zc - dp * wc);
        xo[OUT ? g.face(xx, y + 1, 1) : 2 * NS + i + S] = vd + (zd - dp * wd);
    }
}

// 0 in the blocked vector's padding and on the faces of the domain boundary (fixed)
__device__ __forceinline__ void out_border(const G2d& g, float* out, int t0, int step) {
    for (int t = t0; t < 18 * g.n; t += step) {
        const int q = t % g.n, c = t / g.n % 9, d = t / (9 * g.n), a = c ? g.n + c - 1 : 0;
        out[d ? g.face(q, a, 1) : g.face(a, q, 0)] = 0.f;
    }
}

// C.r = the 4-child sums of r - A x, 0 on fixed coarse faces (the faces at X, Y = n are fixed: 0,
// as allocated). A lane per fine cell and its two low faces, the children of a coarse cell in
// neighbouring lanes (levels have n^2 a multiple of 32): bound by latency, so the loads of one
// child in a chain, not of four (512^2 children 6.7 us, 256^2 4.4; a thread a coarse cell took 10.9
// and 10.6).
template <bool SM = false>
__device__ __forceinline__ void restrict2(const Lv2& L, const float* x, const Lv2& C, int t0, int step) {
    const int S = L.S, NS = L.NS;
    auto var = [](const float* p) { return SM ? *p : ldv2(p); };
    auto coef = [](const float* p) { return SM ? *p : __ldg(p); };
    auto mask = [](const uint8_t* p) { return SM ? *p : __ldg(p); };
    for (int t = t0; t < L.n * L.n; t += step) {
        const int ch = t & 3, c = t >> 2, Y = c / C.n, X = c - Y * C.n, o = C.at(X, Y);
        const int i = L.at(2 * X + (ch & 1), 2 * Y + (ch >> 1));
        const uint8_t m = mask(L.m + i), mc = mask(C.m + o);
        const float *xp = x + i, *xu = x + NS + i, *xv = x + 2 * NS + i;
        const float p = var(xp), u = var(xu), v = var(xv), ub = var(xu + 1), vd = var(xv + S);
        const float lu = 4.f * u - (var(xu - 1) + ub) - (var(xu - S) + var(xu + S));
        const float lv = 4.f * v - (var(xv - 1) + var(xv + 1)) - (var(xv - S) + vd);
        float sp = var(L.r + i) - (L.vol * ((ub - u) + (vd - v)) + coef(L.P + i) * p);
        float su = var(L.r + NS + i) - (L.vol * (lu - (p - var(xp - 1))) + coef(L.P + NS + i) * u);
        float sw = var(L.r + 2 * NS + i) - (L.vol * (lv - (p - var(xp - S))) + coef(L.P + 2 * NS + i) * v);
        if (m & 1) su = 0.f;
        if (m & 2) sw = 0.f;
#pragma unroll
        for (int d = 1; d <= 2; d <<= 1) {
            sp += __shfl_xor_sync(0xffffffffu, sp, d);
            su += __shfl_xor_sync(0xffffffffu, su, d);
            sw += __shfl_xor_sync(0xffffffffu, sw, d);
        }
        if (ch == 0) {
            C.r[o] = sp;
            C.r[C.NS + o] = (mc & 1) ? 0.f : su;
            C.r[2 * C.NS + o] = (mc & 2) ? 0.f : sw;
        }
    }
}

__device__ __forceinline__ void pad_in(const V2& v, const Lv2& L, const float* rhs, int t0, int step) {
    for (int t = t0; t < v.fine.size(); t += step) {
        const int a = pad_index(v.fine, L, t);
        if (a >= 0) L.r[a] = __ldg(rhs + t);
    }
}
template <bool SM = false>
__device__ __forceinline__ void pad_out(const V2& v, const Lv2& L, const float* x, float* out, int t0, int step) {
    for (int t = t0; t < v.fine.size(); t += step) {
        const int a = pad_index(v.fine, L, t);
        out[t] = a < 0 ? 0.f : SM ? x[a] : ldv2(x + a);
    }
}

// levels too large for the one-launch part, a pass per launch
template <bool HX, bool PRO>
__global__ void __launch_bounds__(TPB) k2v_sweep(Lv2 L, int flag, const float* x, Lv2 C, const float* xc, float* xo) {
    sweep2<HX, PRO>(L, flag, x, C, xc, xo, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}
// the finest level's first sweep, from the blocked right-hand side, and its last, to the blocked
// result (512^2: 5.3 and 7.3 us; the sweeps 4.5 and 5.9 with a pass of its own for either
// conversion, 5.6 and 5.9)
__global__ void __launch_bounds__(TPB) k2v_sweep_in(const __grid_constant__ V2 v, const float* __restrict__ rhs) {
    const Lv2& L = v.lv[v.L - 1];
    sweep2<false, false, false, false, true>(L, 0, nullptr, L, nullptr, L.xa, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB, v.fine, rhs);
}
__global__ void __launch_bounds__(TPB) k2v_sweep_out(const __grid_constant__ V2 v, float* __restrict__ out) {
    const Lv2& L = v.lv[v.L - 1];
    const int t0 = blockIdx.x * TPB + threadIdx.x, step = gridDim.x * TPB;
    sweep2<true, false, false, false, false, true>(L, 0, L.xa, L, nullptr, out, t0, step, v.fine);
    out_border(v.fine, out, t0, step);
}
__global__ void __launch_bounds__(TPB) k2v_restrict(Lv2 L, const float* x, Lv2 C) {
    restrict2(L, x, C, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}
__global__ void __launch_bounds__(TPB) k2v_in(const __grid_constant__ V2 v, const float* __restrict__ rhs) {
    pad_in(v, v.lv[v.L - 1], rhs, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
}
__global__ void __launch_bounds__(TPB) k2v_out(const __grid_constant__ V2 v, float* __restrict__ out) {
    pad_out(v, v.lv[0], v.lv[0].xa, out, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);  // (one level)
}
// The coarsest solve, a warp a row, the right-hand side gathered into shared memory (as FP64: a
// conversion costs the FP64 unit as much as the multiply-add) and four loads of the row in flight.
// Bound: the FP64 unit, 64 clocks a warp instruction and quarter of an SM. 24^2 (2112 unknowns):
// 19.1 us, with the gather in the loop 43.5.
__global__ void __launch_bounds__(TPB) k2v_gemv(const __grid_constant__ V2 v) {
    extern __shared__ double gv_r[];
    const Lv2& L = v.lv[0];
    for (int c = threadIdx.x; c < v.nd; c += TPB) {
        const int a = __ldg(v.map + c);
        gv_r[c] = a >= 0 ? (double)ldv2(L.r + a) : 0.0;
    }
    __syncthreads();
    const int row = (blockIdx.x * TPB + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= v.nd) return;
    const double* in = v.inv + (long long)row * v.ld;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int c = lane;
    for (; c + 96 < v.nd; c += 128)
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] += __ldg(in + c + 32 * q) * gv_r[c + 32 * q];
    for (; c < v.nd; c += 32) s[0] += __ldg(in + c) * gv_r[c];
    const double x = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
    const int a = __ldg(v.map + row);
    if (lane == 0 && a >= 0) L.xa[a] = (float)x;
}

// The V-cycle of levels top .. 0 by one thread-block cluster, a cluster barrier between the
// passes: parts 1 the way down, 4 the way up, with the coarsest solve (a larger inverse than
// k2v_cycle takes) between them. rhs / out: blocked finest vectors when top is the finest.
// A level's passes are a few loads deep for each thread, so latency bounds it: 2.25 us a pass
// (96^2: two launches of 18 us a V-cycle).
constexpr int VT = 512;  // threads of a cluster's block
__global__ void __launch_bounds__(VT) k2v_cluster(const __grid_constant__ V2 v, int top, int parts, const float* rhs, float* out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    // consecutive warps in different blocks: the small levels then use every SM of the cluster
    const int t0 = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31), step = gridDim.x * VT;
    if (parts & 1) {
        for (int i = top; i >= 1; i--) {
            const Lv2 &L = v.lv[i], &C = v.lv[i - 1];
            if (i == top && rhs)
                sweep2<false, false, false, false, true>(L, 0, nullptr, C, nullptr, L.xa, t0, step, v.fine, rhs);
            else
                sweep2<false, false>(L, 0, nullptr, C, nullptr, L.xa, t0, step);
            cl.sync();
            sweep2<true, false>(L, 1, L.xa, C, nullptr, L.xb, t0, step);
            cl.sync();
            restrict2(L, L.xb, C, t0, step);
            if (i > 1) cl.sync();
        }
    }
    if (parts & 4) {
        for (int i = 1; i <= top; i++) {
            const Lv2 &L = v.lv[i], &C = v.lv[i - 1];
            sweep2<true, true>(L, 1, L.xb, C, i == 1 ? C.xa : C.xb, L.xa, t0, step);
            cl.sync();
            if (i == top && out) {
                sweep2<true, false, false, false, false, true>(L, 0, L.xa, C, nullptr, out, t0, step, v.fine);
                out_border(v.fine, out, t0, step);
            } else {
                sweep2<true, false>(L, 0, L.xa, C, nullptr, L.xb, t0, step);
            }
            if (i < top) cl.sync();
        }
    }
}

// The same with the coarsest solve, for an 8^2 coarsest level. Every block has the levels of at
// most 32 cells an axis to itself, in shared memory, so that their passes meet at block barriers;
// only the levels above, the coarsest right-hand side's sixteenth of rows a block and its solution
// cross the cluster. Bound: latency, 2.2 us for a pass through L2 and 0.5 for one in shared memory.
// 64^2 (levels to 8^2): 25.9 us a cycle; with all passes through L2, the coarsest product on the
// FP64 pipe and passes of their own for the blocked vectors 39.7; 128^2 below larger levels: 39.8
// and 48.7.
constexpr int CYCLE_ND = 320, CYCLE_BLOCKS = 16, CYCLE_LEVELS = 3;  // coarsest unknowns; levels of 8, 16 and 32
__host__ __device__ constexpr int cycle_mask(int NS) { return (NS + 15) / 16 * 16; }  // bytes of a level's mask: the next vectors lie on 16
constexpr int cycle_smem() {
    int s = 0;
    for (int n = 8; n <= 32; n *= 2) s += (n + 4) * (n + 3) * 12 * 4 + cycle_mask((n + 4) * (n + 3));
    return s;
}
__global__ void __launch_bounds__(VT) k2v_cycle(const __grid_constant__ V2 v, int top, const float* rhs, float* out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char cycle_window[];
    __shared__ Lv2 lv[CYCLE_LEVELS];
    __shared__ float rd[CYCLE_ND];
    const int tid = threadIdx.x, b = blockIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = (warp * CYCLE_BLOCKS + b) * 32 + lane, step = CYCLE_BLOCKS * VT;
    const int in = min(top, CYCLE_LEVELS - 1);  // levels in .. 0 are the block's own
    {
        unsigned char* at = cycle_window;
        for (int i = 0; i <= in; i++) {
            const Lv2& G = v.lv[i];
            float* f = reinterpret_cast<float*>(at);
            uint8_t* m = at + 12 * 4 * G.NS;
            if (tid == 0) {
                lv[i] = G;
                lv[i].r = f;
                lv[i].xa = f + 3 * G.NS;
                lv[i].xb = f + 6 * G.NS;
                lv[i].P = f + 9 * G.NS;
                lv[i].m = m;
            }
            // (NS is a multiple of 4)
            for (int t = tid; t < 9 * G.NS / 4; t += VT) reinterpret_cast<float4*>(f)[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int t = tid; t < 3 * G.NS / 4; t += VT) copy16(f + 9 * G.NS + 4 * t, G.P + 4 * t);
            for (int t = tid; t < G.NS / 4; t += VT) copy4(m + 4 * t, G.m + 4 * t);
            at = m + cycle_mask(G.NS);
        }
    }
    // the block's rows of the coarsest inverse, a warp a row
    constexpr int ROWS = CYCLE_ND / CYCLE_BLOCKS, Q = CYCLE_ND / 32, H = (ROWS + VT / 32 - 1) / (VT / 32);
    static_assert(CYCLE_ND % 32 == 0 && CYCLE_ND <= VT, "whole rows a warp, an entry a thread");
    float2 a[H][Q];
#pragma unroll
    for (int k = 0; k < H; k++)
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int r = warp + k * (VT / 32);
            a[k][q] = r < ROWS ? __ldg(v.inv2 + (b + CYCLE_BLOCKS * r) * CYCLE_ND + lane + 32 * q) : make_float2(0.f, 0.f);
        }
    const int at = tid < CYCLE_ND ? __ldg(v.map + tid) : -1;
    __syncthreads();
    auto started = cl.barrier_arrive();  // (cleared: other blocks may write here)
    if (top > in) {
        cl.barrier_wait(std::move(started));
        for (int i = top; i > in; i--) {
            const Lv2 &L = v.lv[i], &C = v.lv[i - 1];
            if (i == top && rhs)
                sweep2<false, false, false, false, true>(L, 0, nullptr, C, nullptr, L.xa, t0, step, v.fine, rhs);
            else
                sweep2<false, false>(L, 0, nullptr, C, nullptr, L.xa, t0, step);
            cl.sync();
            sweep2<true, false>(L, 1, L.xa, C, nullptr, L.xb, t0, step);
            cl.sync();
            restrict2(L, L.xb, C, t0, step);
            cl.sync();
        }
        const float4* r = reinterpret_cast<const float4*>(v.lv[in].r);
        for (int t = tid; t < 3 * v.lv[in].NS / 4; t += VT) reinterpret_cast<float4*>(lv[in].r)[t] = __ldcg(r + t);
    } else {
        pad_in(v, lv[top], rhs, tid, VT);
        cl.barrier_wait(std::move(started));
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    for (int i = in; i >= 1; i--) {
        const Lv2 &L = lv[i], &C = lv[i - 1];
        sweep2<false, false, true>(L, 0, nullptr, C, nullptr, L.xa, tid, VT);
        __syncthreads();
        sweep2<true, false, true>(L, 1, L.xa, C, nullptr, L.xb, tid, VT);
        __syncthreads();
        restrict2<true>(L, L.xb, C, tid, VT);
        __syncthreads();
    }
    if (tid < CYCLE_ND) rd[tid] = at >= 0 ? lv[0].r[at] : 0.f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < H; k++) {
        const int r = warp + k * (VT / 32);
        if (r >= ROWS) break;
        DfSum sum;
#pragma unroll
        for (int q = 0; q < Q; q++) sum.fma(a[k][q], rd[lane + 32 * q]);
        const float x = sum.warp_total();
        const int o = __ldg(v.map + b + CYCLE_BLOCKS * r);
        if (lane < CYCLE_BLOCKS && o >= 0) cl.map_shared_rank(lv[0].xa, lane)[o] = x;
    }
    cl.sync();
    for (int i = 1; i <= in; i++) {
        const Lv2 &L = lv[i], &C = lv[i - 1];
        sweep2<true, true, true>(L, 1, L.xb, C, i == 1 ? C.xa : C.xb, L.xa, tid, VT);
        __syncthreads();
        sweep2<true, false, true>(L, 0, L.xa, C, nullptr, L.xb, tid, VT);
        __syncthreads();
    }
    for (int i = in + 1; i <= top; i++) {
        const Lv2& L = v.lv[i];
        if (i == in + 1)
            sweep2<true, true, false, true>(L, 1, L.xb, lv[in], lv[in].xb, L.xa, t0, step);
        else
            sweep2<true, true>(L, 1, L.xb, v.lv[i - 1], v.lv[i - 1].xb, L.xa, t0, step);
        cl.sync();
        if (i == top && out) {
            sweep2<true, false, false, false, false, true>(L, 0, L.xa, v.lv[i - 1], nullptr, out, t0, step, v.fine);
            out_border(v.fine, out, t0, step);
        } else {
            sweep2<true, false>(L, 0, L.xa, v.lv[i - 1], nullptr, L.xb, t0, step);
        }
        if (i < top) cl.sync();
    }
    if (top == in && out) pad_out<true>(v, lv[top], top == 0 ? lv[0].xa : lv[top].xb, out, t0, step);
}

}  // namespace

// ====================================================================== 2D handle state
struct Level2 {
    G2d g;
    double lap = 1.0;
    uint8_t* fixed = nullptr;
    double *vol = nullptr, *pen = nullptr;
    float *vol32 = nullptr, *pen32 = nullptr;
    float *r = nullptr, *x = nullptr, *p = nullptr, *Ap = nullptr, *rs = nullptr, *d = nullptr, *Ad = nullptr;
    double *t0 = nullptr, *t1 = nullptr;
};

}  // namespace stg

struct Ctx2 {
    std::vector<stg::Level2> lv;
    double *aug0 = nullptr, *aug1 = nullptr;
    const double* inv = nullptr;
    int* info = nullptr;
    stg::InvOrder order;
    // Laplacian-form V-cycle: padded vectors, coefficients and the coarsest index map (one
    // allocation each, created with the handle); clusters: blocks of a cluster that can run
    stg::V2 v{};
    float* pad = nullptr;
    uint8_t* padm = nullptr;
    int* map = nullptr;
    int cluster = 0;
};

namespace stg {

namespace {

Level2& fine2(stg_t* h) { return h->c2->lv.back(); }

Coef2<double> coef64(const Level2& L) { return Coef2<double>{L.vol, L.pen, L.fixed}; }
Coef2<float> coef32(const Level2& L) { return Coef2<float>{L.vol32, L.pen32, L.fixed}; }

int apply2_32(stg_t* h, Level2& L, const float* x, float* y) {
    k2_apply<float, 0><<<g1(L.g.size()), TPB, 0, h->st>>>(L.g, coef32(L), (float)L.lap, x, nullptr, y, nullptr);
    STG_LAUNCH_CK();
    return STG_OK;
}

// StokeFlowSmoothing::applyMapping, iter_num 1, alpha 1: out = sum of the two colour
// corrections, each followed by r -= A d
int smoother2(stg_t* h, Level2& L, int order, const float* r, float* out) {
    const int n = L.g.size();
    STG_CK(cudaMemcpyAsync(L.rs, r, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->st));
    STG_CK(cudaMemsetAsync(out, 0, sizeof(float) * n, h->st));
    for (int i = 0; i < 2; i++) {
        int flag = order ? 1 - i : i;
        STG_CK(cudaMemsetAsync(L.d, 0, sizeof(float) * n, h->st));
        PROF(h, 1, 0.0, ([&] {
                 k2_smooth<<<g1(L.g.nc()), TPB, 0, h->st>>>(L.g, coef32(L), (float)L.lap, flag, L.rs, L.d);
                 STG_LAUNCH_CK();
                 return STG_OK;
             })());
        STG_TRY(apply2_32(h, L, L.d, L.Ad));
        k2_update<<<g1(n), TPB, 0, h->st>>>(n, L.d, L.Ad, out, L.rs);
        STG_LAUNCH_CK();
    }
    return STG_OK;
}

int coarse2(stg_t* h, const float* r, float* x) {
    Level2& C = h->c2->lv[0];
    const int nd = C.g.size();
    k2_gemv<<<g1(32ll * nd), TPB, 0, h->st>>>(nd, h->c2->inv, 2 * nd, r, x);
    STG_LAUNCH_CK();
    return STG_OK;
}

// MultigridSolve::Vcycle (common_cpx/MultigridSolve.cpp:73-106) in FP32
int vcycle2(stg_t* h) {
    auto& lv = h->c2->lv;
    const int L = (int)lv.size();
    for (int i = L - 1; i >= 0; i--) {
        Level2& F = lv[i];
        const int n = F.g.size();
        if (i > 0)
            STG_TRY(smoother2(h, F, 0, F.r, F.p));
        else
            STG_TRY(coarse2(h, F.r, F.p));
        STG_TRY(apply2_32(h, F, F.p, F.Ap));
        k2_update<<<g1(n), TPB, 0, h->st>>>(n, F.p, F.Ap, F.x, F.r);
        STG_LAUNCH_CK();
        if (i != 0) {
            Level2& C = lv[i - 1];
            k2_restrict<float><<<g1(C.g.size()), TPB, 0, h->st>>>(C.g, F.g, F.r, C.fixed, C.r);
            STG_LAUNCH_CK();
            STG_CK(cudaMemsetAsync(C.x, 0, sizeof(float) * C.g.size(), h->st));
        }
    }
    for (int i = 0; i < L; i++) {
        Level2& F = lv[i];
        const int n = F.g.size();
        if (i != 0) {
            Level2& C = lv[i - 1];
            k2_prolong<float><<<g1(n), TPB, 0, h->st>>>(F.g, C.g, C.x, F.fixed, F.p);
            STG_LAUNCH_CK();
            STG_TRY(apply2_32(h, F, F.p, F.Ap));
            k2_update<<<g1(n), TPB, 0, h->st>>>(n, F.p, F.Ap, F.x, F.r);
            STG_LAUNCH_CK();
        }
        if (i > 0) {
            STG_TRY(smoother2(h, F, 1, F.r, F.p));
            STG_TRY(apply2_32(h, F, F.p, F.Ap));
            k2_update<<<g1(n), TPB, 0, h->st>>>(n, F.p, F.Ap, F.x, F.r);
            STG_LAUNCH_CK();
        }
    }
    return STG_OK;
}

// ---------------------------------------------------------------- solve_core hooks
// FluidSteadyState::update_penalty set-up half (stoke/FluidSteadyState.cpp:122-140)
int setup2(stg_t* h) {
    if (!h->have_boundary || !h->have_penalty) {
        set_error("boundary and penalty must be set before the solver set-up");
        return STG_E_INVALID;
    }
    auto& lv = h->c2->lv;
    // coarsening and the analytic coarsest matrix touch fixed buffers only: replayed as a
    // CUDA graph; the inverse follows as one cooperative launch
    auto body = [&]() -> int {
        for (int i = (int)lv.size() - 2; i >= 0; i--) {
            Level2 &c = lv[i], &f = lv[i + 1];
            if (h->hier_flow)
                k2_coarsen<true><<<g1(c.g.size()), TPB, 0, h->st>>>(c.g, f.g, f.fixed, f.vol, f.pen, c.fixed, c.vol, c.pen, c.vol32,
                                                                      c.pen32);
            else
                k2_coarsen<false><<<g1(c.g.size()), TPB, 0, h->st>>>(c.g, f.g, f.fixed, f.vol, f.pen, c.fixed, c.vol, c.pen, c.vol32,
                                                                       c.pen32);
            STG_LAUNCH_CK();
        }
        V2& v = h->c2->v;
        for (int i = 0; i < v.L && h->lap2d; i++) {
            k2_pad_coef<<<g1((long long)v.lv[i].n * v.lv[i].n), TPB, 0, h->st>>>(lv[i].g, v.lv[i], lv[i].pen32, lv[i].fixed,
                                                                                const_cast<float*>(v.lv[i].P),
                                                                                const_cast<uint8_t*>(v.lv[i].m));
            STG_LAUNCH_CK();
        }
        Level2& C = lv[0];
        const int nd = C.g.size();
        k2_calcA<<<g1((long long)nd * nd), TPB, 0, h->st>>>(C.g, C.vol, C.pen, C.fixed, C.lap, h->closed ? 1 : 0, h->c2->aug0);
        STG_LAUNCH_CK();
        return STG_OK;
    };
    GraphCache& G = h->sgraph;
    STG_TRY(graphed(h, G, (h->closed ? 2 : 1) | (h->hier_flow ? 4 : 0) | (h->lap2d ? 8 : 0), body, [](bool) {}));
    // the inversion: one cooperative launch, outside the graph
    // fixed cells are identity rows among the pressures, which the block elimination's sign
    // rule does not cover: the pivoted elimination takes them
    if (h->fixed_cells2d)
        STG_TRY(gj_invert(h->st, lv[0].g.size(), h->c2->aug0, h->c2->aug1, h->c2->info, &h->c2->inv, true));
    else
        STG_TRY(inv_blocks(h->st, lv[0].g.size(), h->c2->order, h->closed ? 1 : 0, h->c2->aug0, h->c2->aug1, h->c2->info, &h->c2->inv));
    V2& v = h->c2->v;
    v.inv = h->c2->inv;
    if (v.inv2) STG_TRY(split_inverse(h->st, v.nd, v.inv, v.ld, v.inv2));
    for (int i = 0; i < v.L; i++) {  // a face's vol doubles a level down, as lap does
        v.lv[i].lap = (float)lv[i].lap;
        v.lv[i].vol = (float)std::ldexp(h->vol2d, v.L - 1 - i);
    }
    h->updated = true;
    return STG_OK;
}

// The solver's V-cycle in the Laplacian form. Levels of at most 128 cells an axis run in one
// cluster launch, with the coarsest solve when that level is 8^2 (128^2: 8192 cells a colour, one
// for each thread of 16 blocks; at 256^2 a pass of one cluster would take longer than a launch
// of the whole GPU); larger ones a launch a pass, replayed as a CUDA graph.
constexpr int CLUSTER_N = 128;

cudaLaunchConfig_t config2(cudaStream_t st, int blocks, bool cycle, cudaLaunchAttribute (&at)[1]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(VT);
    cfg.dynamicSmemBytes = cycle ? cycle_smem() : 0;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
// parts 7: the whole cycle of levels top .. 0 (k2v_cycle)
int launch_cluster2(stg_t* h, int top, int parts, const float* rhs, float* out) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config2(h->st, parts == 7 ? CYCLE_BLOCKS : h->c2->cluster, parts == 7, at);
    if (parts == 7)
        STG_CK(cudaLaunchKernelEx(&cfg, k2v_cycle, h->c2->v, top, rhs, out));
    else
        STG_CK(cudaLaunchKernelEx(&cfg, k2v_cluster, h->c2->v, top, parts, rhs, out));
    count_launch();
    return STG_OK;
}

int vcycle2_lap(stg_t* h, const float* rhs, float* out) {
    const V2& v = h->c2->v;
    const int fine = v.L - 1;
    const unsigned gs = g1(v.fine.size());
    int top = fine;  // finest level of the cluster part
    while (top > 0 && v.lv[top].n > CLUSTER_N) top--;
    const bool whole = top == fine, small = v.inv2 != nullptr;
    if (whole && small) return launch_cluster2(h, top, 7, rhs, out);
    // the finest level's first and last pass take the caller's vectors and stay outside the graph
    const unsigned gf = g1((long long)v.lv[fine].n * v.lv[fine].n / 2);
    if (!whole) {
        k2v_sweep_in<<<gf, TPB, 0, h->st>>>(v, rhs);
        STG_LAUNCH_CK();
    } else if (top == 0) {
        k2v_in<<<gs, TPB, 0, h->st>>>(v, rhs);
        STG_LAUNCH_CK();
    }
    auto body = [&]() -> int {
        for (int i = fine; i > top; i--) {
            const Lv2 &L = v.lv[i], &C = v.lv[i - 1];
            const unsigned gb = g1((long long)L.n * L.n / 2);
            if (i < fine) {
                k2v_sweep<false, false><<<gb, TPB, 0, h->st>>>(L, 0, nullptr, C, nullptr, L.xa);
                STG_LAUNCH_CK();
            }
            k2v_sweep<true, false><<<gb, TPB, 0, h->st>>>(L, 1, L.xa, C, nullptr, L.xb);
            STG_LAUNCH_CK();
            k2v_restrict<<<g1((long long)L.n * L.n), TPB, 0, h->st>>>(L, L.xb, C);
            STG_LAUNCH_CK();
        }
        if (small) {
            STG_TRY(launch_cluster2(h, top, 7, nullptr, nullptr));
        } else {
            if (top > 0) STG_TRY(launch_cluster2(h, top, 1, nullptr, nullptr));
            k2v_gemv<<<g1(32ll * v.nd), TPB, sizeof(double) * v.nd, h->st>>>(v);
            STG_LAUNCH_CK();
            if (top > 0) STG_TRY(launch_cluster2(h, top, 4, nullptr, nullptr));
        }
        for (int i = top + 1; i <= fine; i++) {
            const Lv2 &L = v.lv[i], &C = v.lv[i - 1];
            const unsigned gb = g1((long long)L.n * L.n / 2);
            k2v_sweep<true, true><<<gb, TPB, 0, h->st>>>(L, 1, L.xb, C, i == 1 ? C.xa : C.xb, L.xa);
            STG_LAUNCH_CK();
            if (i < fine) {
                k2v_sweep<true, false><<<gb, TPB, 0, h->st>>>(L, 0, L.xa, C, nullptr, L.xb);
                STG_LAUNCH_CK();
            }
        }
        return STG_OK;
    };
    if (whole && top > 0) {  // the levels fit a cluster, the coarsest inverse does not
        STG_TRY(launch_cluster2(h, top, 1, rhs, nullptr));
        k2v_gemv<<<g1(32ll * v.nd), TPB, sizeof(double) * v.nd, h->st>>>(v);
        STG_LAUNCH_CK();
        return launch_cluster2(h, top, 4, nullptr, out);
    }
    // the vol of the levels is a kernel argument: part of the key through a counter of changes
    STG_TRY(graphed(h, h->vgraph, 2 + 2 * (long long)h->vol_changes + (v.inv == h->c2->aug0 + v.nd), body, [](bool) {}));
    if (!whole)
        k2v_sweep_out<<<gf, TPB, 0, h->st>>>(v, out);
    else
        k2v_out<<<gs, TPB, 0, h->st>>>(v, out);
    STG_LAUNCH_CK();
    return STG_OK;
}

int resid2(stg_t* h, const d4* b, const d4* x, d4* r, double* nrm2_host) {
    Level2& F = fine2(h);
    unsigned nb = g1(F.g.size());
    k2_apply<double, 1><<<nb, TPB, 0, h->st>>>(F.g, coef64(F), F.lap, reinterpret_cast<const double*>(x),
                                               reinterpret_cast<const double*>(b), reinterpret_cast<double*>(r), h->d_parts);
    STG_LAUNCH_CK();
    STG_TRY(reduce_parts(h->st, h->d_parts, (int)nb, h->dnrm));
    STG_CK(cudaMemcpyAsync(nrm2_host, h->dnrm, sizeof(double), cudaMemcpyDeviceToHost, h->st));
    STG_CK(cudaStreamSynchronize(h->st));
    return STG_OK;
}

int precond2(stg_t* h, const float4* rhs, float4* out) {
    if (h->lap2d && h->c2->cluster) {
        PROF(h, 1, 0.0, vcycle2_lap(h, reinterpret_cast<const float*>(rhs), reinterpret_cast<float*>(out)));
        return STG_OK;
    }
    Level2& F = fine2(h);
    const int n = F.g.size();
    STG_CK(cudaMemcpyAsync(F.r, rhs, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->st));
    STG_CK(cudaMemsetAsync(F.x, 0, sizeof(float) * n, h->st));
    // the V-cycle works on the level buffers only: replayed as a CUDA graph
    STG_TRY(graphed(h, h->vgraph, 1, [&] { return vcycle2(h); }, [](bool) {}));
    STG_CK(cudaMemcpyAsync(out, F.x, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->st));
    return STG_OK;
}

int shift2(stg_t* h, const float4* v, const float4* z, float4* out) {
    Level2& L = fine2(h);
    k2_apply<float, 1><<<g1(L.g.size()), TPB, 0, h->st>>>(L.g, coef32(L), (float)L.lap, reinterpret_cast<const float*>(z),
                                                           reinterpret_cast<const float*>(v), reinterpret_cast<float*>(out), nullptr);
    STG_LAUNCH_CK();
    return STG_OK;
}

int apply2(stg_t* h, const float4* x, float4* y) {
    return apply2_32(h, fine2(h), reinterpret_cast<const float*>(x), reinterpret_cast<float*>(y));
}

}  // namespace

// ====================================================================== 2D entry points
// (called by the C ABI in solver.cu when the handle has dim == 2)
int create2d(stg_t* h) {
    const int n = h->n;
    h->c2 = new Ctx2();
    auto& lv = h->c2->lv;
    int low = n & -n;
    int L = (int)std::lround(std::log2((double)low)) - 2;  // FluidSteadyState::init (:12)
    if (L < 1) L = 1;
    lv.resize(L);
    for (int i = L - 1, m = n; i >= 0; i--, m /= 2) lv[i].g.n = m;
    lv[L - 1].lap = 1.0;
    for (int i = L - 2; i >= 0; i--) lv[i].lap = 2.0 * lv[i + 1].lap;  // createSubSystem (StokeFlowSubSystem.cu:155)
    for (auto& V : lv) {
        size_t s = V.g.size();
        STG_TRY(dalloc(h->st, &V.fixed, s));
        STG_TRY(dalloc(h->st, &V.vol, s));
        STG_TRY(dalloc(h->st, &V.pen, s));
        STG_TRY(dalloc(h->st, &V.vol32, s));
        STG_TRY(dalloc(h->st, &V.pen32, s));
        for (float** q : {&V.r, &V.x, &V.p, &V.Ap, &V.rs, &V.d, &V.Ad}) STG_TRY(dalloc(h->st, q, s));
    }
    const int nd = lv[0].g.size();
    if (nd > 8192) {
        set_error("N = %d leaves a %d-unknown coarsest level (N / 8 must have a larger power-of-two factor)", n, nd);
        return STG_E_UNSUPPORTED;
    }
    h->coarsest = nd;
    STG_TRY(dalloc(h->st, &h->c2->aug0, 2ull * nd * nd));
    STG_TRY(dalloc(h->st, &h->c2->aug1, 2ull * nd * nd));
    STG_TRY(dalloc(h->st, &h->c2->info, 1));
    std::vector<std::vector<int>> faces(2);
    std::vector<int> cells;
    for (int q = 0; q < nd; q++) (q < lv[0].g.off(0) ? cells : faces[q >= lv[0].g.off(1)]).push_back(q);
    STG_TRY(inv_order(h->c2->order, faces, cells));
    if (L <= MAXL2) {
        V2& v = h->c2->v;
        size_t nf = 0, nm = 0;
        for (auto& q : lv) nf += 12ull * (q.g.n + 4) * (q.g.n + 3), nm += (size_t)(q.g.n + 4) * (q.g.n + 3);
        STG_TRY(dalloc(h->st, &h->c2->pad, nf));
        STG_TRY(dalloc(h->st, &h->c2->padm, nm));
        STG_TRY(dalloc(h->st, &h->c2->map, (size_t)nd));
        v.L = L;
        v.fine = lv[L - 1].g;
        v.nd = nd;
        v.ld = 2 * nd;
        v.map = h->c2->map;
        float* f = h->c2->pad;
        uint8_t* m = h->c2->padm;
        for (int i = 0; i < L; i++) {
            Lv2& q = v.lv[i];
            q.n = lv[i].g.n;
            q.S = q.n + 4;
            q.NS = q.S * (q.n + 3);
            float** to[4] = {const_cast<float**>(&q.P), &q.r, &q.xa, &q.xb};
            for (auto t : to) *t = f, f += 3 * q.NS;
            q.m = m;
            m += q.NS;
        }
        k2_pad_index<<<g1(nd), TPB, 0, h->st>>>(lv[0].g, v.lv[0], h->c2->map);
        STG_LAUNCH_CK();
        // blocks of one cluster: 16 where the device grants it, else the portable 8
        STG_CK(cudaFuncSetAttribute(k2v_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        STG_CK(cudaFuncSetAttribute(k2v_gemv, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * (int)sizeof(double)));
        int can = 0;
        cudaLaunchAttribute at[1];
        for (int c = 16; c >= 8 && !h->c2->cluster; c /= 2) {
            const cudaLaunchConfig_t cfg = config2(nullptr, c, false, at);
            if (cudaOccupancyMaxActiveClusters(&can, k2v_cluster, &cfg) == cudaSuccess && can > 0) h->c2->cluster = c;
            cudaGetLastError();
        }
        if (nd == CYCLE_ND) {
            STG_CK(cudaFuncSetAttribute(k2v_cycle, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            STG_CK(cudaFuncSetAttribute(k2v_cycle, cudaFuncAttributeMaxDynamicSharedMemorySize, cycle_smem()));
            const cudaLaunchConfig_t cfg = config2(nullptr, CYCLE_BLOCKS, true, at);
            if (h->c2->cluster && cudaOccupancyMaxActiveClusters(&can, k2v_cycle, &cfg) == cudaSuccess && can > 0)
                STG_TRY(dalloc(h->st, &v.inv2, (size_t)nd * nd));
            cudaGetLastError();
        }
    }
    Level2& F = lv.back();
    h->L = L;
    h->n4 = F.g.size() / 4;
    h->ncell = (size_t)n * n;
    h->nface = (size_t)n * (n + 1);
    h->setup = setup2;
    h->resid64 = resid2;
    h->precond = precond2;
    h->apply32 = apply2;
    h->shift32 = shift2;
    return STG_OK;
}

void destroy2d(stg_t* h) {
    if (!h->c2) return;
    for (auto& V : h->c2->lv) {
        cudaFree(V.fixed);
        cudaFree(V.vol);
        cudaFree(V.pen);
        cudaFree(V.vol32);
        cudaFree(V.pen32);
        for (float* q : {V.r, V.x, V.p, V.Ap, V.rs, V.d, V.Ad}) cudaFree(q);
        cudaFree(V.t0);
        cudaFree(V.t1);
    }
    cudaFree(h->c2->aug0);
    cudaFree(h->c2->aug1);
    cudaFree(h->c2->info);
    inv_order_free(h->c2->order);
    cudaFree(h->c2->pad);
    cudaFree(h->c2->padm);
    cudaFree(h->c2->map);
    cudaFree(h->c2->v.inv2);
    delete h->c2;
    h->c2 = nullptr;
}

long long dof2d(const stg_t* h, int level) { return h->c2->lv[level].g.size(); }
int level_n2d(const stg_t* h, int level) { return h->c2->lv[level].g.n; }

// inputs are device staging copies of the Field-order host arrays
int set_boundary2d(stg_t* h, const double* cvol, const int* cfix, const double* fv0, const double* fv1, const int* ff0,
                   const int* ff1, double fv, bool* fixed_cells, bool* uniform) {
    Level2& F = fine2(h);
    h->hflags[0] = h->hflags[1] = 0;
    k2_fine_descr<<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, cvol, cfix, fv0, fv1, ff0, ff1, fv, F.fixed, F.vol, h->hflags);
    STG_LAUNCH_CK();
    STG_TRY(f64_to_f32(h->st, F.g.size() / 4, reinterpret_cast<const d4*>(F.vol), 1.0, reinterpret_cast<float4*>(F.vol32)));
    STG_CK(cudaStreamSynchronize(h->st));
    *fixed_cells = h->hflags[0] != 0;
    *uniform = h->hflags[1] == 0;
    return STG_OK;
}

int set_penalty2d(stg_t* h, const double* cp, const double* f0, const double* f1) {
    Level2& F = fine2(h);
    k2_penalty_from_field<<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, cp, f0, f1, F.fixed, F.pen, F.pen32);
    STG_LAUNCH_CK();
    return STG_OK;
}

int set_density2d(stg_t* h, const double* rho, const stg_alpha& law) {
    Level2& F = fine2(h);
    k2_face_penalty<<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, rho, law, F.fixed, F.pen, F.pen32);
    STG_LAUNCH_CK();
    return STG_OK;
}

int field_to_vec2d(stg_t* h, const double* cell, const double* f0, const double* f1, d4* out) {
    Level2& F = fine2(h);
    k2_field_to_blocked<<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, cell, f0, f1, reinterpret_cast<double*>(out));
    STG_LAUNCH_CK();
    return STG_OK;
}

int vec_to_field2d(stg_t* h, const d4* in, double* cell, double* f0, double* f1) {
    Level2& F = fine2(h);
    k2_blocked_to_field<<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, reinterpret_cast<const double*>(in), cell, f0, f1);
    STG_LAUNCH_CK();
    return STG_OK;
}

// E x (FluidEnergyGrad, lap_coeff 1 on the energy descriptor = fine coefficients)
int energy2d(stg_t* h, const d4* x, d4* out, double* part, int* nb) {
    Level2& F = fine2(h);
    *nb = (int)g1(F.g.size());
    k2_apply<double, 2><<<*nb, TPB, 0, h->st>>>(F.g, coef64(F), 1.0, reinterpret_cast<const double*>(x), nullptr,
                                                reinterpret_cast<double*>(out), part);
    STG_LAUNCH_CK();
    return STG_OK;
}

int sensitivity2d(stg_t* h, const double* rho, const stg_alpha& law, const d4* x, const d4* lam, double* grad) {
    Level2& F = fine2(h);
    k2_sensitivity<<<g1((long long)F.g.n * F.g.n), TPB, 0, h->st>>>(F.g, rho, law, reinterpret_cast<const double*>(x),
                                                                     reinterpret_cast<const double*>(lam), grad);
    STG_LAUNCH_CK();
    return STG_OK;
}

// ---------------------------------------------------------------- LinearMapping adapters (blocked layout = native)
int apply_A2d(stg_t* h, int level, double* out, const double* in) {
    Level2& L = h->c2->lv[level];
    k2_apply<double, 0><<<g1(L.g.size()), TPB, 0, h->st>>>(L.g, coef64(L), L.lap, in, nullptr, out, nullptr);
    STG_LAUNCH_CK();
    return STG_OK;
}

int apply_E2d(stg_t* h, double* out, const double* in) {
    int nb;
    return energy2d(h, reinterpret_cast<const d4*>(in), reinterpret_cast<d4*>(out), nullptr, &nb);
}

int vcycle2d(stg_t* h, double* out, const double* in) {
    Level2& F = fine2(h);
    const long long n4 = F.g.size() / 4;
    STG_TRY(f64_to_f32(h->st, n4, reinterpret_cast<const d4*>(in), 1.0, reinterpret_cast<float4*>(F.r)));
    STG_CK(cudaMemsetAsync(F.x, 0, sizeof(float) * F.g.size(), h->st));
    STG_TRY(vcycle2(h));
    STG_TRY(f32_to_f64(h->st, n4, reinterpret_cast<const float4*>(F.x), reinterpret_cast<d4*>(out)));
    return STG_OK;
}

int apply_op2d(stg_t* h, int op, int level, double* out, const double* in) {
    auto& lv = h->c2->lv;
    Level2& L = lv[level];
    switch (op) {
        case STG_OP_RESTRICT:
            if (level >= (int)lv.size() - 1) break;
            k2_restrict<double><<<g1(L.g.size()), TPB, 0, h->st>>>(L.g, lv[level + 1].g, in, L.fixed, out);
            STG_LAUNCH_CK();
            return STG_OK;
        case STG_OP_PROLONG: {
            if (level >= (int)lv.size() - 1) break;
            Level2& F = lv[level + 1];
            k2_prolong<double><<<g1(F.g.size()), TPB, 0, h->st>>>(F.g, L.g, in, F.fixed, out);
            STG_LAUNCH_CK();
            return STG_OK;
        }
        case STG_OP_SMOOTH_PRE:
        case STG_OP_SMOOTH_POST:
        case STG_OP_VANKA_RED:
        case STG_OP_VANKA_BLACK: {
            if (level == 0) break;
            const long long n4 = L.g.size() / 4;
            STG_TRY(f64_to_f32(h->st, n4, reinterpret_cast<const d4*>(in), 1.0, reinterpret_cast<float4*>(L.r)));
            if (op == STG_OP_SMOOTH_PRE || op == STG_OP_SMOOTH_POST) {
                STG_TRY(smoother2(h, L, op == STG_OP_SMOOTH_POST ? 1 : 0, L.r, L.x));
            } else {
                STG_CK(cudaMemsetAsync(L.x, 0, sizeof(float) * L.g.size(), h->st));
                k2_smooth<<<g1(L.g.nc()), TPB, 0, h->st>>>(L.g, coef32(L), (float)L.lap, op == STG_OP_VANKA_BLACK ? 1 : 0,
                                                             L.r, L.x);
                STG_LAUNCH_CK();
            }
            STG_TRY(f32_to_f64(h->st, n4, reinterpret_cast<const float4*>(L.x), reinterpret_cast<d4*>(out)));
            return STG_OK;
        }
        case STG_OP_COARSE: {
            if (level != 0) break;
            const int nd = L.g.size();
            k2_gemv64<<<g1(32ll * nd), TPB, 0, h->st>>>(nd, h->c2->inv, 2 * nd, in, out);
            STG_LAUNCH_CK();
            return STG_OK;
        }
        default: break;
    }
    set_error("operator %d not defined at level %d", op, level);
    return STG_E_INVALID;
}

int level_descr2d(stg_t* h, int level, double* vol, double* pen, uint8_t* fixed) {
    Level2& L = h->c2->lv[level];
    const size_t s = L.g.size();
    if (vol) STG_CK(cudaMemcpyAsync(vol, L.vol, sizeof(double) * s, cudaMemcpyDeviceToDevice, h->st));
    if (pen) STG_CK(cudaMemcpyAsync(pen, L.pen, sizeof(double) * s, cudaMemcpyDeviceToDevice, h->st));
    if (fixed) STG_CK(cudaMemcpyAsync(fixed, L.fixed, s, cudaMemcpyDeviceToDevice, h->st));
    return STG_OK;
}

}  // namespace stg
