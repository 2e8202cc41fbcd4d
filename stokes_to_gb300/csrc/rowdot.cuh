// Rows of the coarsest inverse times the right-hand side, inside a V-cycle that one cluster runs
// (smallcycle.cu, solver2d.cu). Half a warp takes a row: the FP64 pipe does two lanes per SM and
// clock, so the product's cost is its warp instructions, ND / 16 FMAs and four additions of the
// half-warp sum for two rows (a whole warp a row: ND / 32 and five for one). The entries are
// loaded ahead of the barrier that completes the right-hand side. One row after the other, with
// its loads behind the barrier, took 15 us of a 37 us cycle at 304 unknowns.
#pragma once
#include "internal.cuh"

namespace stg {

template <int ND, int R>
struct RowDots {
    static constexpr int Q = (ND + 15) / 16;
    static constexpr int HALVES = (ND + R - 1) / R;  // half-warps that have rows: h, h + HALVES, ...
    double v[R][Q];
    __device__ __forceinline__ void load(const double* inv, int ld, int h, int lane) {
        if (h >= HALVES) return;
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int row = h + k * HALVES;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int c = (lane & 15) + 16 * q;
                v[k][q] = row < ND && c < ND ? __ldg(inv + (long long)row * ld + c) : 0.0;
            }
        }
    }
    // out[k] = row h + k HALVES times rd (valid in every lane of the half); rd: ND values in
    // shared memory; called by whole warps with h < HALVES in at least one half
    __device__ __forceinline__ void dot(const double* rd, int lane, double (&out)[R]) const {
        double a[R][2];
#pragma unroll
        for (int k = 0; k < R; k++) a[k][0] = a[k][1] = 0.0;
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int c = (lane & 15) + 16 * q;
            const double b = c < ND ? rd[c] : 0.0;
#pragma unroll
            for (int k = 0; k < R; k++) a[k][q & 1] += v[k][q] * b;
        }
#pragma unroll
        for (int k = 0; k < R; k++) out[k] = a[k][0] + a[k][1];
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < R; k++) out[k] += __shfl_xor_sync(0xffffffffu, out[k], o);
    }
};

// Sum of products a b over the lanes of a warp on the FP32 pipe: a = a.x + a.y (split_inverse), the
// products and sums in double-float arithmetic. The FP64 pipe takes 64 clocks of a quarter of an SM
// for an instruction of a warp, these eleven take one each. (Error-free sum after Knuth, product
// after Dekker with an FMA.) Rounded to FP32 the sums are those of an FP64 product, bit for bit, on the
// inverses and V-cycle residuals of 3D grids of 8 to 32 and 2D ones of 16 to 128 cells (error
// against 64 bits 5.9e-8 at most, 2.2e-8 on average, either way).
struct DfSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float v) {  // exact: s + err = s + v
        const float t = s + v, z = t - s;
        c += (s - (t - z)) + (v - z);
        s = t;
    }
    __device__ __forceinline__ void fma(float2 a, float b) {
        const float p = __fmul_rn(a.x, b), e = fmaf(a.x, b, -p);  // a.x b = p + e
        add(p);
        c += fmaf(a.y, b, e);
    }
    __device__ __forceinline__ float warp_total() {
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, s, o), d = __shfl_xor_sync(0xffffffffu, c, o);
            const float t = s + v, z = t - s;
            c = (c + d) + ((s - (t - z)) + (v - z));
            s = t;
        }
        return s + c;
    }
};

// asynchronous copies to shared memory
__device__ __forceinline__ void copy4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

}  // namespace stg
