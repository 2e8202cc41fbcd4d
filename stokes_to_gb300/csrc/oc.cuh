// The optimality-criteria rule of one cell, shared by the update of a handle's design and the
// allocation-free update.
#pragma once
#include "internal.cuh"

namespace stg {

// x_new at the multiplier lam: x sqrt(max(0, -dc) / (lam dv)) within the move and the bounds
__device__ __forceinline__ double oc_new(double x, double dc, double dv, double lam, double move, double lo, double hi) {
    const double B = fmax(0.0, -dc) / (dv * lam);
    return fmin(fmin(hi, x + move), fmax(fmax(lo, x - move), x * sqrt(B)));
}

// The part of it that a bisection on lam keeps: x_new = clamp(oc_scale / sqrt(lam)). Two roots,
// so that max(0, -dc) / dv cannot overflow where max(0, -dc) / (lam dv) does not.
__device__ __forceinline__ double oc_scale(double x, double dc, double dv) { return x * (sqrt(fmax(0.0, -dc)) / sqrt(dv)); }


// What a bisection on lam needs of a cell, formed once; add: acc + vw x_new(lam) at t = 1 / sqrt(lam)
struct OcCell {
    double s, lo, hi, vw;
    __device__ __forceinline__ double at(double t) const { return fmin(hi, fmax(lo, s * t)); }
    __device__ __forceinline__ double add(double t, double acc) const { return fma(vw, at(t), acc); }
};
__device__ __forceinline__ OcCell oc_cell(double x, double dc, double vw, double inv_n, double move, double lo, double hi) {
    return OcCell{oc_scale(x, dc, vw * inv_n), fmax(lo, x - move), fmin(hi, x + move), vw};
}

}  // namespace stg
