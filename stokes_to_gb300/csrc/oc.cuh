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

}  // namespace stg
