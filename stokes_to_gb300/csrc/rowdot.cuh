// Rows of the coarsest inverse times the right-hand side, inside a V-cycle that one cluster runs
// (smallcycle.cu, solver2d.cu): a warp takes R rows, their entries are loaded ahead of the
// barrier that completes the right-hand side, and the rows' FP64 chains run interleaved (one
// row after the other, with its loads behind the barrier, took 15 us of a 37 us cycle at 304
// unknowns; the FP64 pipe alone needs 2.4 us on 16 SMs).
#pragma once
#include "internal.cuh"

namespace stg {

template <int ND, int R>
struct RowDots {
    static constexpr int Q = (ND + 31) / 32;
    double v[R][Q];
    // rows first, first + stride, ... of the row-major inverse
    __device__ __forceinline__ void load(const double* inv, int ld, int first, int stride, int lane) {
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int row = first + k * stride;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int c = lane + 32 * q;
                v[k][q] = row < ND && c < ND ? __ldg(inv + (long long)row * ld + c) : 0.0;
            }
        }
    }
    // out[k] = row k . rd (valid in every lane); rd: ND values in shared memory
    __device__ __forceinline__ void dot(const double* rd, int lane, double (&out)[R]) const {
#pragma unroll
        for (int k = 0; k < R; k++) out[k] = 0.0;
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int c = lane + 32 * q;
            const double b = c < ND ? rd[c] : 0.0;
#pragma unroll
            for (int k = 0; k < R; k++) out[k] += v[k][q] * b;
        }
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < R; k++) out[k] += __shfl_xor_sync(0xffffffffu, out[k], o);
    }
};

}  // namespace stg
