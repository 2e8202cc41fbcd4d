// One cell of the box-Vanka smoother in the Laplacian form (sweep.cu k_sweep_cell, smallcycle.cu):
// its pressure and its six faces, numbered p, low u v w, high u v w.
#pragma once
#include <cuda_fp16.h>

#include "internal.cuh"

namespace stg {

// The penalties of a cell's unknowns p, u, v, w and of its high faces from FP16
// planes in shared memory (Q: the cell's slot, Qn: the next plane's).
template <int RW>
__device__ __forceinline__ void cell_penalty(const uint2* Q, const uint2* Qn, float psc, float raw[7]) {
    const uint2 po = *Q;
    const __half* Hn = reinterpret_cast<const __half*>(Qn);
    const __half* Hh = reinterpret_cast<const __half*>(Q);
    const float2 pa = __half22float2(*reinterpret_cast<const __half2*>(&po.x)),
                 pz = __half22float2(*reinterpret_cast<const __half2*>(&po.y));
    // a fixed face's copy is infinite: its e in cell_solve is 0, and x is 0 there, so any finite
    // penalty gives the same residual
    raw[0] = pa.x * psc;
    raw[1] = pa.y * psc;
    raw[2] = pz.x * psc;
    raw[3] = pz.y * psc;
    raw[4] = __half2float(Hn[1]) * psc;
    raw[5] = __half2float(Hh[4 * RW + 2]) * psc;
    raw[6] = __half2float(Hh[4 + 3]) * psc;
}

// res -= A x of the cell's rows. lap_lo, lap_hi: the faces' Laplacians, p_lo, p_hi: the pressures
// beyond them; raw: penalties, infinite on fixed faces, where x is 0.
__device__ __forceinline__ void cell_residual(float vol, const float raw[7], float p0, const float lap_lo[3], const float lap_hi[3],
                                              const float p_lo[3], const float p_hi[3], const float lo[3], const float hi[3],
                                              float res[7]) {
    float pen[7];
#pragma unroll
    for (int d = 0; d < 7; d++) pen[d] = fminf(raw[d], 1e38f);
    res[0] -= vol * ((hi[0] - lo[0]) + (hi[1] - lo[1]) + (hi[2] - lo[2])) + pen[0] * p0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        res[1 + d] -= vol * (lap_lo[d] - (p0 - p_lo[d])) + pen[1 + d] * lo[d];
        res[4 + d] -= vol * (lap_hi[d] - (p_hi[d] - p0)) + pen[4 + d] * hi[d];
    }
}

// The same with x in slot order (the rows of stencil.cuh lap_core, low face at the cell's slot, high
// face one on): A, B, D, E the cell's slot in planes i - 1 .. i + 2, XW the pitch of a row.
template <int XW>
__device__ __forceinline__ void slot_residual(const float4* A, const float4* B, const float4* D, const float4* E, float vol,
                                              const float raw[7], float& p0, float lo[3], float hi[3], float res[7]) {
    const float4 c = B[0], xm = A[0], xp = D[0], ym = B[-XW], yp = B[XW], zm = B[-1], zp = B[1];
    const float4 xy = D[XW], xz = D[1], yz = B[XW + 1];
    p0 = c.x;
    lo[0] = c.y;
    lo[1] = c.z;
    lo[2] = c.w;
    hi[0] = xp.y;
    hi[1] = yp.z;
    hi[2] = zp.w;
    const float lap_lo[3] = {6.f * c.y - (xm.y + xp.y) - (ym.y + yp.y) - (zm.y + zp.y),
                             6.f * c.z - (xm.z + xp.z) - (ym.z + yp.z) - (zm.z + zp.z),
                             6.f * c.w - (xm.w + xp.w) - (ym.w + yp.w) - (zm.w + zp.w)};
    const float lap_hi[3] = {6.f * xp.y - (c.y + E[0].y) - (D[-XW].y + xy.y) - (D[-1].y + xz.y),
                             6.f * yp.z - (A[XW].z + xy.z) - (c.z + B[2 * XW].z) - (B[XW - 1].z + yz.z),
                             6.f * zp.w - (A[1].w + xz.w) - (B[1 - XW].w + yz.w) - (c.w + B[2].w)};
    const float p_lo[3] = {xm.x, ym.x, zm.x}, p_hi[3] = {xp.x, yp.x, zp.x};
    cell_residual(vol, raw, p0, lap_lo, lap_hi, p_lo, p_hi, lo, hi, res);
}

// The same with x as the cells of the other colour have it: each by row and pair as (p, low faces)
// and, FH further on, (high faces). W, F, E: the cell's pair in planes i - 1 .. i + 1, FW the pitch
// of a row, q: the cell's place in its pair. pb: the pressure of the pair's other cell.
template <int FW, int FH>
__device__ __forceinline__ void neighbour_residual(const float4* W, const float4* F, const float4* E, int q, float vol,
                                                   const float raw[7], float p0, float lo[3], float hi[3], float res[7], float& pb) {
    const float4 wl = W[0], wh = W[FH], el = E[0], eh = E[FH], sl = F[-FW], sh = F[FH - FW], nl = F[FW], nh = F[FH + FW],
                 dl = F[q - 1], dh = F[FH + q - 1], ul = F[q], uh = F[FH + q];
    pb = q ? dl.x : ul.x;
    lo[0] = wh.x;
    lo[1] = sh.y;
    lo[2] = dh.z;
    hi[0] = el.y;
    hi[1] = nl.z;
    hi[2] = ul.w;
    const float lap_lo[3] = {6.f * wh.x - (wl.y + el.y) - (sl.y + nl.y) - (dl.y + ul.y),
                             6.f * sh.y - (wl.z + el.z) - (sl.z + nl.z) - (dl.z + ul.z),
                             6.f * dh.z - (wl.w + el.w) - (sl.w + nl.w) - (dl.w + ul.w)};
    const float lap_hi[3] = {6.f * el.y - (wh.x + eh.x) - (sh.x + nh.x) - (dh.x + uh.x),
                             6.f * nl.z - (wh.y + eh.y) - (sh.y + nh.y) - (dh.y + uh.y),
                             6.f * ul.w - (wh.z + eh.z) - (sh.z + nh.z) - (dh.z + uh.z)};
    const float p_lo[3] = {wl.x, sl.x, dl.x}, p_hi[3] = {el.x, nl.x, ul.x};
    cell_residual(vol, raw, p0, lap_lo, lap_hi, p_lo, p_hi, lo, hi, res);
}

// Block solve of a cell with the residuals res: adds the step to its faces and returns the
// pressure's. e = 1 / diagonal of the free faces (6 vol + P), 0 on fixed ones.
__device__ __forceinline__ float cell_solve(float vol, float v6, const float raw[7], const float res[7], float lo[3], float hi[3]) {
    float el[3], eh[3], num = res[0], den = 2.f * raw[0];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        el[d] = __fdividef(1.f, v6 + raw[1 + d]);
        eh[d] = __fdividef(1.f, v6 + raw[4 + d]);
        num += vol * (res[1 + d] * el[d] - res[4 + d] * eh[d]);
        den -= vol * vol * (el[d] + eh[d]);
    }
    const float dp = den != 0.f ? __fdividef(num, den) : 0.f, vdp = vol * dp;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] += (res[1 + d] + vdp) * el[d];
        hi[d] += (res[4 + d] - vdp) * eh[d];
    }
    return dp;
}

}  // namespace stg
