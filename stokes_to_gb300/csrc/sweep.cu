// Fused smoothing sweep: one colour of the box-Vanka block-Jacobi step on the residual
// equation, x_out = x_in + SHATTER(B^-1 GATHER(r - A x_in)), in a single pass over HBM.
//
// The step is DescentSmoother's P_c applied to the current residual
// (common_cpx/DescentSmoother.cu:31-47, stoke/StokeLike.cu:220-278 and 345-372). The
// residual r - A x_in is never written out: a block owns a 32 (k) x 8 (j) column of slots
// and marches along i through a chunk of planes. Planes of x (tile + two-slot halo in j and k),
// r and P (tile + one-slot halo) are staged in shared-memory rings by asynchronous copies
// (cp.async) issued three planes ahead, the masks by register prefetch; while plane i+3
// streams in, the block forms the residual of plane i+1, the pressure update of every red
// cell of plane i (tile + one-slot low halo) and the new unknowns of plane i. Each sweep
// reads r, x, P and the mask once from HBM and writes x once.
//
// Block algebra. A red cell's block is read by DirectSolveBlockInverse<7> off
// B = M_w A M_w + M_b A M_b (stoke/StokeLike.cu:41-96, 345-372; the masks keep the faces
// of one parity). With one vol value on the free faces and no fixed cell, the face-face
// couplings inside a block cancel (grad-div against curl-curl) and B couples no two red
// blocks, so each block is an arrow matrix solved exactly by its Schur complement:
//   face rows  D_f u_f + c_f p = r_f,  D_f = vol*free_f*(4 + free(left cell) + free(right cell)) + P_f + F_f
//   pressure   sum_f b_f u_f + a p = r_p,  c_f = -vol*free_f (owner's left face) / +vol*free_f (right face),
//              b_f = free_c * c_f,  a = 2 (P_p + F_p) (the pressure diagonal is counted by both masks).
// Every face belongs to exactly one red block (the cell on its low side or on its high
// side, whichever has the colour); faces with neither are left unchanged, as SHATTER
// leaves them. If the Schur complement is 0 (the reference's LU meets a zero pivot) the
// pressure is left unchanged.
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "cell.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace stg {

namespace {

constexpr int SK = 32, SJ = 8;           // output tile (k, j)
constexpr int XK = SK + 4, XJ = SJ + 4;  // x / mask region  [j0-2, j0+SJ+2) x [k0-2, k0+SK+2)
constexpr int RK = SK + 2, RJ = SJ + 2;  // r / rr / P region [j0-1, j0+SJ+1) x [k0-1, k0+SK+1)
constexpr int DK = SK + 1, DJ = SJ + 1;  // dp region        [j0-1, j0+SJ)   x [k0-1, k0+SK)
constexpr int NT = SK * SJ;
constexpr int XN = XJ * XK, RN = RJ * RK;
constexpr int DRED = (DK + 1) / 2;       // red cells per dp row (at most)
static_assert(XN <= 2 * NT && RN <= 2 * NT && DJ * DRED <= NT, "tile regions exceed two elements per thread");

// shared-memory rings: x by plane mod 4, P mod 3, r and rr mod 2, masks mod 5
struct Smem {
    float4 x[4][XN];
    float4 P[3][RN];
    float4 r[2][RN];
    float4 rr[2][RN];
    float dp[DJ * DK];
    float dpp[SJ * SK];
    uint8_t m[5][XN];
};

__device__ __forceinline__ int rx(int p) { return (p + 20) & 3; }
__device__ __forceinline__ int rp(int p) { return (p + 21) % 3; }
__device__ __forceinline__ int r2(int p) { return (p + 20) & 1; }
__device__ __forceinline__ int rm(int p) { return (p + 20) % 5; }

// 16-byte asynchronous global -> shared copy; zero-fills when !ok
__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Per-thread element of a staged region: its shared index, the (j,k) part of its slot
// offset and whether that (j,k) lies inside the allocation.
struct Elem {
    int sidx;   // -1: no element
    int jk;     // (j+1)*sz + (k+1)
    bool ok;    // j, k inside the allocation
    bool box;   // j, k inside [0, n]
};

__device__ __forceinline__ Elem make_elem(const Geom& g, int e, int nelem, int w, int j_org, int k_org) {
    Elem el;
    el.sidx = e < nelem ? e : -1;
    int j = j_org + e / w, k = k_org + e % w;
    el.jk = (j + 1) * g.sz + (k + 1);
    el.ok = e < nelem && j >= -1 && j <= g.n + 1 && k >= -1 && k <= g.n + 2;
    el.box = e < nelem && j >= 0 && j <= g.n && k >= 0 && k <= g.n;
    return el;
}

__device__ __forceinline__ bool plane_ok(int n, int p) { return p >= -1 && p <= n + 1; }

template <bool HAS_X, bool LAP>
__device__ __forceinline__ void residual_plane(Smem& S, const Elem (&R)[2], int n, float vol, int p) {
    const bool pin = p >= 0 && p <= n;
    const int xa = rx(p - 1), xb = rx(p), xc = rx(p + 1);
    const int ma = rm(p - 1), mb = rm(p), mc = rm(p + 1);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int e = R[q].sidx;
        if (e < 0) continue;
        float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
        if (pin && R[q].box) {
            float4 rv = S.r[r2(p)][e];
            if (HAS_X && LAP) {
                // Laplacian form (stencil.cuh): six face neighbours, own row masked
                const int xi = e + (e / RK) * (XK - RK) + XK + 1;
                auto q = [&](int pl, int o) {
                    float4 v = S.x[pl][o];
                    return Q4<float>{v.x, v.y, v.z, v.w};
                };
                const float4 pv = S.P[rp(p)][e];
                float o[4];
                lap_core<float>(q(xb, xi), q(xa, xi), q(xc, xi), q(xb, xi - XK), q(xb, xi + XK), q(xb, xi - 1), q(xb, xi + 1),
                                Q4<float>{pv.x, pv.y, pv.z, pv.w}, vol, o);
                o[0] = rv.x - o[0];
                o[1] = rv.y - o[1];
                o[2] = rv.z - o[2];
                o[3] = rv.w - o[3];
                mask4<float>(S.m[mb][xi], o);
                out = make_float4(o[0], o[1], o[2], o[3]);
            } else if (HAS_X) {
                // rr region index e = rj*RK + rk  ->  x region index (rj+1)*XK + (rk+1)
                const int xi = e + (e / RK) * (XK - RK) + XK + 1;
                auto ld = [&](int a, int b, int c) {
                    const int pl = a < 0 ? xa : (a > 0 ? xc : xb);
                    const int ml = a < 0 ? ma : (a > 0 ? mc : mb);
                    const int o = xi + b * XK + c;
                    float4 v = S.x[pl][o];
                    return nb_make<float>(v.x, v.y, v.z, v.w, S.m[ml][o]);
                };
                uint8_t ms = S.m[mb][xi];
                float o[4];
                stencil_core<float, false>(ld, vol, ms, o);
                float4 xv = S.x[xb][xi];
                float4 pv = S.P[rp(p)][e];
                o[0] += (pv.x + ((ms & MP) ? 1.f : 0.f)) * xv.x;
                o[1] += (pv.y + ((ms & MU) ? 1.f : 0.f)) * xv.y;
                o[2] += (pv.z + ((ms & MV) ? 1.f : 0.f)) * xv.z;
                o[3] += (pv.w + ((ms & MW) ? 1.f : 0.f)) * xv.w;
                out = make_float4(rv.x - o[0], rv.y - o[1], rv.z - o[2], rv.w - o[3]);
            } else {
                out = rv;
            }
        }
        S.rr[r2(p)][e] = out;
    }
}

// pressure update of every red cell of plane p in the dp region, one thread per red cell.
// LAP: every present cell is free and every free face lies between two present cells, so a
// free face's diagonal is 6 vol + P; fixed faces (residual 0) drop out through vL / vR = 0.
template <bool LAP>
__device__ __forceinline__ void pressure_plane(Smem& S, int n, float vol, int p, int j0, int k0, int flag, int tid) {
    if (tid >= DJ * DRED) return;
    const int dj = tid / DRED, q = tid % DRED;
    const int j = j0 - 1 + dj;
    const int dk = ((p + j + flag - (k0 - 1)) & 1) + 2 * q;  // red: (p + j + k + flag) even
    const int k = k0 - 1 + dk;
    if (dk >= DK || p < 0 || j < 0 || k < 0 || !cell_ok(n, p, j, k)) return;
    const int ri = dj * RK + dk;                 // rr / P index of the cell
    const int xi = (dj + 1) * XK + (dk + 1);     // x / mask index of the cell
    float4 rc = S.rr[r2(p)][ri];
    float4 pc = S.P[rp(p)][ri];
    uint8_t m0 = S.m[rm(p)][xi];
    float out;
    if (LAP) {
        const float rL[3] = {rc.y, rc.z, rc.w};
        const float pL[3] = {pc.y, pc.z, pc.w};
        const uint8_t mhi[3] = {S.m[rm(p + 1)][xi], S.m[rm(p)][xi + XK], S.m[rm(p)][xi + 1]};
        const float rh[3] = {S.rr[r2(p + 1)][ri].y, S.rr[r2(p)][ri + RK].z, S.rr[r2(p)][ri + 1].w};
        const float ph[3] = {S.P[rp(p + 1)][ri].y, S.P[rp(p)][ri + RK].z, S.P[rp(p)][ri + 1].w};
        const uint8_t bit[3] = {MU, MV, MW};
        const float v6 = 6.f * vol;
        float num = rc.x, den = 2.f * pc.x;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            float vL = (m0 & bit[d]) ? 0.f : vol, vR = (mhi[d] & bit[d]) ? 0.f : vol;
            float iL = __fdividef(vL, v6 + pL[d]);
            float iR = __fdividef(vR, v6 + ph[d]);
            num += rL[d] * iL - rh[d] * iR;
            den -= vL * iL + vR * iR;
        }
        out = den != 0.f ? __fdividef(num, den) : 0.f;
    } else if (m0 & MP) {
        out = __fdividef(rc.x, 2.f * (pc.x + 1.f));
    } else {
        const float rL[3] = {rc.y, rc.z, rc.w};
        const float pL[3] = {pc.y, pc.z, pc.w};
        const uint8_t mlo[3] = {S.m[rm(p - 1)][xi], S.m[rm(p)][xi - XK], S.m[rm(p)][xi - 1]};
        const uint8_t mhi[3] = {S.m[rm(p + 1)][xi], S.m[rm(p)][xi + XK], S.m[rm(p)][xi + 1]};
        const float rh[3] = {S.rr[r2(p + 1)][ri].y, S.rr[r2(p)][ri + RK].z, S.rr[r2(p)][ri + 1].w};
        const float ph[3] = {S.P[rp(p + 1)][ri].y, S.P[rp(p)][ri + RK].z, S.P[rp(p)][ri + 1].w};
        const uint8_t bit[3] = {MU, MV, MW};
        float num = rc.x, den = 2.f * pc.x;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            bool fixL = m0 & bit[d], fixR = mhi[d] & bit[d];
            float vL = fixL ? 0.f : vol, vR = fixR ? 0.f : vol;
            float iL = __fdividef(1.f, vL * (5.f + ((mlo[d] & MP) ? 0.f : 1.f)) + pL[d] + (fixL ? 1.f : 0.f));
            float iR = __fdividef(1.f, vR * (5.f + ((mhi[d] & MP) ? 0.f : 1.f)) + ph[d] + (fixR ? 1.f : 0.f));
            num += vL * rL[d] * iL - vR * rh[d] * iR;
            den -= vL * vL * iL + vR * vR * iR;
        }
        out = den != 0.f ? __fdividef(num, den) : 0.f;
    }
    S.dp[dj * DK + dk] = out;
}

template <bool HAS_X, bool LAP>
__global__ void __launch_bounds__(NT, 3) k_sweep(Geom g, float vol, const float4* __restrict__ r, const float4* __restrict__ xin,
                                                float4* __restrict__ xout, const uint8_t* __restrict__ m,
                                                const float4* __restrict__ P, int flag, int chunk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    const int n = g.n;
    const int tk = threadIdx.x, tj = threadIdx.y, tid = tj * SK + tk;
    const int k0 = blockIdx.x * SK, j0 = blockIdx.y * SJ, i0 = blockIdx.z * chunk;
    const int i1 = min(i0 + chunk, n + 1);
    const int j = j0 + tj, k = k0 + tk;
    const int plane = g.sy * g.sz;
    const Elem X[2] = {make_elem(g, tid, XN, XK, j0 - 2, k0 - 2), make_elem(g, tid + NT, XN, XK, j0 - 2, k0 - 2)};
    const Elem R[2] = {make_elem(g, tid, RN, RK, j0 - 1, k0 - 1), make_elem(g, tid + NT, RN, RK, j0 - 1, k0 - 1)};
    const bool out_ok = j <= n && k <= n;
    const int out_jk = (j + 1) * g.sz + (k + 1);
    const int oxi = (tj + 2) * XK + (tk + 2), ori = (tj + 1) * RK + (tk + 1), odi = (tj + 1) * DK + (tk + 1);

    auto issue_x = [&](int p) {
        const bool pok = plane_ok(n, p);
        const int base = (p + 1) * plane;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (X[q].sidx >= 0) {
                bool ok = pok && X[q].ok;
                cp16(&S.x[rx(p)][X[q].sidx], ok ? (const void*)(xin + base + X[q].jk) : (const void*)xin, ok);
            }
    };
    auto issue_r = [&](float4* dst, const float4* a, int p) {
        const bool pok = plane_ok(n, p);
        const int base = (p + 1) * plane;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (R[q].sidx >= 0) {
                bool ok = pok && R[q].ok;
                cp16(&dst[R[q].sidx], ok ? (const void*)(a + base + R[q].jk) : (const void*)a, ok);
            }
    };
    uint8_t mreg[2];
    auto fetch_m = [&](int p) {
        const bool pok = plane_ok(n, p);
        const int base = (p + 1) * plane;
#pragma unroll
        for (int q = 0; q < 2; q++) mreg[q] = (pok && X[q].ok) ? __ldg(m + base + X[q].jk) : (uint8_t)MALL;
    };
    auto store_m = [&](int p) {
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (X[q].sidx >= 0) S.m[rm(p)][X[q].sidx] = mreg[q];
    };

    // prologue: planes i0-2 .. i0+2 staged, residual of i0-1 and i0, pressure of i0-1
    if (HAS_X)
        for (int p = i0 - 2; p <= i0 + 1; p++) issue_x(p);
    for (int p = i0 - 1; p <= i0 + 1; p++) issue_r(S.P[rp(p)], P, p);
    issue_r(S.r[r2(i0 - 1)], r, i0 - 1);
    issue_r(S.r[r2(i0)], r, i0);
    cp_commit();
    for (int p = i0 - 2; p <= i0 + 2; p++) {
        fetch_m(p);
        store_m(p);
    }
    cp_wait_all();
    __syncthreads();
    residual_plane<HAS_X, LAP>(S, R, n, vol, i0 - 1);
    __syncthreads();
    if (HAS_X) issue_x(i0 + 2);       // replaces plane i0-2
    issue_r(S.r[r2(i0 + 1)], r, i0 + 1);  // replaces r of i0-1
    cp_commit();
    residual_plane<HAS_X, LAP>(S, R, n, vol, i0);
    __syncthreads();
    pressure_plane<LAP>(S, n, vol, i0 - 1, j0, k0, flag, tid);
    __syncthreads();
    S.dpp[tid] = S.dp[odi];
    cp_wait_all();
    __syncthreads();

    for (int i = i0; i < i1; i++) {
        // stream plane i+3 (x, masks) and i+2 (P, r) while plane i is processed
        if (HAS_X) issue_x(i + 3);
        issue_r(S.P[rp(i + 2)], P, i + 2);
        issue_r(S.r[r2(i + 2)], r, i + 2);
        cp_commit();
        fetch_m(i + 3);
        residual_plane<HAS_X, LAP>(S, R, n, vol, i + 1);
        __syncthreads();
        pressure_plane<LAP>(S, n, vol, i, j0, k0, flag, tid);
        __syncthreads();
        if (out_ok) {
            float4 xo = HAS_X ? S.x[rx(i)][oxi] : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 rv = S.rr[r2(i)][ori];
            float4 pv = S.P[rp(i)][ori];
            uint8_t m0 = S.m[rm(i)][oxi];
            const bool own_red = cell_ok(n, i, j, k) && ((i + j + k + flag) & 1) == 0;
            const float fc = (m0 & MP) ? 0.f : 1.f;
            const float dpown = S.dp[odi];
            if (own_red) xo.x += dpown;
            const float rf[3] = {rv.y, rv.z, rv.w};
            const float pf[3] = {pv.y, pv.z, pv.w};
            const uint8_t bit[3] = {MU, MV, MW};
            uint8_t mlo[3] = {0, 0, 0};
            if (!LAP) {
                mlo[0] = S.m[rm(i - 1)][oxi];
                mlo[1] = S.m[rm(i)][oxi - XK];
                mlo[2] = S.m[rm(i)][oxi - 1];
            }
            const float dplo[3] = {S.dpp[tid], S.dp[odi - DK], S.dp[odi - 1]};
            float upd[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                upd[d] = 0.f;
                int li = i - (d == 0), lj = j - (d == 1), lk = k - (d == 2);
                bool lower_red = !own_red && li >= 0 && lj >= 0 && lk >= 0 && cell_ok(n, li, lj, lk) &&
                                 ((li + lj + lk + flag) & 1) == 0;
                if (!own_red && !lower_red) continue;
                bool fix = m0 & bit[d];
                float v = fix ? 0.f : vol;
                // LAP: a free face has two present cells (fc = 1, lower cell present)
                float D = LAP ? (fix ? 1.f : 6.f * vol + pf[d])
                              : v * (4.f + fc + ((mlo[d] & MP) ? 0.f : 1.f)) + pf[d] + (fix ? 1.f : 0.f);
                float dpo = own_red ? dpown : dplo[d];
                float cf = own_red ? -v : v;
                upd[d] = __fdividef(rf[d] - cf * dpo, D);
            }
            xo.y += upd[0];
            xo.z += upd[1];
            xo.w += upd[2];
            xout[(i + 1) * plane + out_jk] = xo;
        }
        store_m(i + 3);
        cp_wait_all();
        __syncthreads();
        S.dpp[tid] = S.dp[odi];
    }
}

// ---------------------------------------------------------------- Laplacian-form sweep
// The same march and algebra in the Laplacian form (stencil.cuh), written so that the
// plane loop does little besides the arithmetic: ring slots are rotated element offsets
// into flat shared arrays (no modular ring indices), every per-thread index, validity
// flag and global offset is formed once before the march, global plane pointers advance
// by one plane per step, and the mask ring holds 4 planes (the Laplacian form reads no
// mask of the plane below).
struct SmemL {
    float4 x[4 * XN];
    float4 P[3 * RN];
    float4 r[2 * RN];
    float4 rr[2 * RN];
    float dp[DJ * DK];
    float dpp[SJ * SK];
    uint8_t m[4 * XN];
};

struct Stage {
    int s;   // shared index in the plane (-1: none)
    int jk;  // global offset in the plane
};

__device__ __forceinline__ Stage make_stage(const Geom& g, int e, int nelem, int w, int j_org, int k_org) {
    Stage st;
    int j = j_org + e / w, k = k_org + e % w;
    bool ok = e < nelem && j >= -1 && j <= g.n + 1 && k >= -1 && k <= g.n + 2;
    st.s = e < nelem ? e : -1;
    st.jk = ok ? (j + 1) * g.sz + (k + 1) : -1;  // -1: outside the allocation (zero fill)
    return st;
}

__device__ __forceinline__ void cp16s(unsigned dst, const void* src, bool ok) {
    int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

template <bool HAS_X>
__global__ void __launch_bounds__(NT, 3) k_sweep_lap(Geom g, float vol, const float4* __restrict__ r, const float4* __restrict__ xin,
                                                    float4* __restrict__ xout, const uint8_t* __restrict__ m,
                                                    const float4* __restrict__ P, int flag, int chunk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemL& S = *reinterpret_cast<SmemL*>(smem_raw);
    const int n = g.n;
    const int tk = threadIdx.x, tj = threadIdx.y, tid = tj * SK + tk;
    const int k0 = blockIdx.x * SK, j0 = blockIdx.y * SJ, i0 = blockIdx.z * chunk;
    const int i1 = min(i0 + chunk, n + 1);
    const int j = j0 + tj, k = k0 + tk;
    const long long plane = (long long)g.sy * g.sz;
    const float v6 = 6.f * vol;

    // staging elements: x / mask region (X) and P / r region (R), two per thread
    const Stage X0 = make_stage(g, tid, XN, XK, j0 - 2, k0 - 2), X1 = make_stage(g, tid + NT, XN, XK, j0 - 2, k0 - 2);
    const Stage R0 = make_stage(g, tid, RN, RK, j0 - 1, k0 - 1), R1 = make_stage(g, tid + NT, RN, RK, j0 - 1, k0 - 1);
    const unsigned sx = (unsigned)__cvta_generic_to_shared(S.x), sP = (unsigned)__cvta_generic_to_shared(S.P),
                   sr = (unsigned)__cvta_generic_to_shared(S.r);

    // residual elements: rr/P index e and x/mask index xi, and whether (j,k) lies in [0,n]^2
    const int re0 = tid, re1 = tid + NT;
    const int rx0 = re0 + (re0 / RK) * (XK - RK) + XK + 1, rx1 = re1 + (re1 / RK) * (XK - RK) + XK + 1;
    auto in_box = [&](int e) {
        int jj = j0 - 1 + e / RK, kk = k0 - 1 + e % RK;
        return e < RN && jj >= 0 && jj <= n && kk >= 0 && kk <= n;
    };
    const bool rb0 = in_box(re0), rb1 = in_box(re1);

    // pressure-phase cell of this thread for the two plane parities
    const int pdj = tid / DRED, pq = tid % DRED, pj = j0 - 1 + pdj;
    const bool p_thread = tid < DJ * DRED;
    const int ppar0 = (pj + flag - (k0 - 1)) & 1;  // dk = ((p & 1) ^ ppar0) + 2 pq
    // (the two parities as scalars: a runtime-indexed array would live in local memory)
    const int pdk0 = 2 * pq, pdk1 = 2 * pq + 1;
    const bool pok0 = p_thread && pdk0 < DK && pj >= 0 && k0 - 1 + pdk0 >= 0 && pj < n && k0 - 1 + pdk0 < n;
    const bool pok1 = p_thread && pdk1 < DK && pj >= 0 && k0 - 1 + pdk1 >= 0 && pj < n && k0 - 1 + pdk1 < n;

    // update-phase slot
    const bool out_ok = j <= n && k <= n;
    const long long out_jk = (long long)(j + 1) * g.sz + (k + 1);
    const int oxi = (tj + 2) * XK + (tk + 2), ori = (tj + 1) * RK + (tk + 1), odi = (tj + 1) * DK + (tk + 1);
    const bool jk_cell = j < n && k < n;
    const int opar = (j + k + flag) & 1;  // own colour is red when ((i & 1) ^ opar) == 0
    const bool lo_j_ok = j >= 1 && k < n, lo_k_ok = k >= 1 && j < n;

    auto issue_x = [&](int slot, int p, const float4* src) {  // plane p of x into ring slot
        const bool pok = p >= -1 && p <= n + 1;
        if (X0.s >= 0) cp16s(sx + 16u * (slot + X0.s), (pok && X0.jk >= 0) ? (const void*)(src + X0.jk) : (const void*)xin, pok && X0.jk >= 0);
        if (X1.s >= 0) cp16s(sx + 16u * (slot + X1.s), (pok && X1.jk >= 0) ? (const void*)(src + X1.jk) : (const void*)xin, pok && X1.jk >= 0);
    };
    auto issue_r = [&](unsigned base, int slot, int p, const float4* src, const float4* any) {
        const bool pok = p >= -1 && p <= n + 1;
        if (R0.s >= 0) cp16s(base + 16u * (slot + R0.s), (pok && R0.jk >= 0) ? (const void*)(src + R0.jk) : (const void*)any, pok && R0.jk >= 0);
        if (R1.s >= 0) cp16s(base + 16u * (slot + R1.s), (pok && R1.jk >= 0) ? (const void*)(src + R1.jk) : (const void*)any, pok && R1.jk >= 0);
    };
    uint8_t mr0 = MALL, mr1 = MALL;
    auto fetch_m = [&](int p, const uint8_t* src) {
        const bool pok = p >= -1 && p <= n + 1;
        mr0 = (pok && X0.jk >= 0) ? __ldg(src + X0.jk) : (uint8_t)MALL;
        mr1 = (pok && X1.jk >= 0) ? __ldg(src + X1.jk) : (uint8_t)MALL;
    };
    auto store_m = [&](int slot) {
        if (X0.s >= 0) S.m[slot + X0.s] = mr0;
        if (X1.s >= 0) S.m[slot + X1.s] = mr1;
    };

    // residual of plane p: x slots (p-1, p, p+1), r / P / mask slots of p, into rr slot
    auto residual = [&](int p, int xa, int xb, int xc, int rs, int ps, int ms, int rrs) {
        const bool pin = p >= 0 && p <= n;
        auto one = [&](int e, int xi, bool box) {
            float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pin && box) {
                const float4 rv = S.r[rs + e];
                if (HAS_X) {
                    auto q = [&](int idx) {
                        const float4 v = S.x[idx];
                        return Q4<float>{v.x, v.y, v.z, v.w};
                    };
                    const float4 pv = S.P[ps + e];
                    float o[4];
                    lap_core<float>(q(xb + xi), q(xa + xi), q(xc + xi), q(xb + xi - XK), q(xb + xi + XK), q(xb + xi - 1),
                                    q(xb + xi + 1), Q4<float>{pv.x, pv.y, pv.z, pv.w}, vol, o);
                    o[0] = rv.x - o[0];
                    o[1] = rv.y - o[1];
                    o[2] = rv.z - o[2];
                    o[3] = rv.w - o[3];
                    mask4<float>(S.m[ms + xi], o);
                    out = make_float4(o[0], o[1], o[2], o[3]);
                } else {
                    out = rv;  // r is zero on fixed unknowns
                }
            }
            S.rr[rrs + e] = out;
        };
        one(re0, rx0, rb0);
        if (re1 < RN) one(re1, rx1, rb1);
    };

    // pressure update of the red cells of plane p (rr slots p, p+1; P slots p, p+1; mask slots p, p+1)
    auto pressure = [&](int p, int rr0, int rr1, int p0, int p1, int m0s, int m1s) {
        const int b = (p & 1) ^ ppar0;
        if (!(b ? pok1 : pok0) || p < 0 || p >= n) return;
        const int dk = b ? pdk1 : pdk0;
        const int ri = pdj * RK + dk, xi = (pdj + 1) * XK + (dk + 1);
        const float4 rc = S.rr[rr0 + ri], pc = S.P[p0 + ri];
        const uint8_t mo = S.m[m0s + xi];
        const float rL[3] = {rc.y, rc.z, rc.w}, pL[3] = {pc.y, pc.z, pc.w};
        const uint8_t mhi[3] = {S.m[m1s + xi], S.m[m0s + xi + XK], S.m[m0s + xi + 1]};
        const float rh[3] = {S.rr[rr1 + ri].y, S.rr[rr0 + ri + RK].z, S.rr[rr0 + ri + 1].w};
        const float ph[3] = {S.P[p1 + ri].y, S.P[p0 + ri + RK].z, S.P[p0 + ri + 1].w};
        const uint8_t bit[3] = {MU, MV, MW};
        float num = rc.x, den = 2.f * pc.x;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const float vL = (mo & bit[d]) ? 0.f : vol, vR = (mhi[d] & bit[d]) ? 0.f : vol;
            const float iL = __fdividef(vL, v6 + pL[d]), iR = __fdividef(vR, v6 + ph[d]);
            num += rL[d] * iL - rh[d] * iR;
            den -= vL * iL + vR * iR;
        }
        S.dp[pdj * DK + dk] = den != 0.f ? __fdividef(num, den) : 0.f;
    };

    // ring slots as element offsets (rotated each plane)
    int xm1 = 0 * XN, x0 = 1 * XN, x1 = 2 * XN, x2 = 3 * XN;  // x(i-1), x(i), x(i+1), x(i+2)
    int pm1 = 0 * RN, p0 = 1 * RN, p1 = 2 * RN;               // P(i-1), P(i), P(i+1)
    int r0 = 0 * RN, r1 = 1 * RN;                             // r(i), r(i+1)
    int rrm1 = 0 * RN, rr0 = 1 * RN;                          // rr(i-1), rr(i)
    int mm1 = 0 * XN, m0 = 1 * XN, m1 = 2 * XN, m2 = 3 * XN;  // masks of planes i-1 .. i+2

    // prologue: planes i0-2 .. i0+1 of x, i0-1 .. i0+1 of P, i0-1 and i0 of r, masks i0-1 .. i0+2
    const float4* gx = xin + (i0 - 1) * plane;  // plane p lives at (p + 1) * plane: this is plane i0-2
    if (HAS_X) {
        issue_x(xm1, i0 - 2, gx);
        issue_x(x0, i0 - 1, gx + plane);
        issue_x(x1, i0, gx + 2 * plane);
        issue_x(x2, i0 + 1, gx + 3 * plane);
    }
    const float4* gP = P + i0 * plane;
    issue_r(sP, pm1, i0 - 1, gP, P);
    issue_r(sP, p0, i0, gP + plane, P);
    issue_r(sP, p1, i0 + 1, gP + 2 * plane, P);
    const float4* gr = r + i0 * plane;
    issue_r(sr, r0, i0 - 1, gr, r);
    issue_r(sr, r1, i0, gr + plane, r);
    cp_commit();
    const uint8_t* gm = m + i0 * plane;  // plane i0-1
    fetch_m(i0 - 1, gm);
    store_m(mm1);
    fetch_m(i0, gm + plane);
    store_m(m0);
    fetch_m(i0 + 1, gm + 2 * plane);
    store_m(m1);
    fetch_m(i0 + 2, gm + 3 * plane);
    store_m(m2);
    cp_wait_all();
    __syncthreads();
    // residual of i0-1: x(i0-2, i0-1, i0) = slots (xm1, x0, x1), r(i0-1) = r0, P(i0-1) = pm1, mask(i0-1) = mm1
    residual(i0 - 1, xm1, x0, x1, r0, pm1, mm1, rrm1);
    __syncthreads();
    if (HAS_X) issue_x(xm1, i0 + 2, gx + 4 * plane);  // x(i0+2) replaces x(i0-2)
    issue_r(sr, r0, i0 + 1, gr + 2 * plane, r);       // r(i0+1) replaces r(i0-1)
    cp_commit();
    // residual of i0: x(i0-1, i0, i0+1) = (x0, x1, x2), r(i0) = r1, P(i0) = p0, mask(i0) = m0
    residual(i0, x0, x1, x2, r1, p0, m0, rr0);
    __syncthreads();
    pressure(i0 - 1, rrm1, rr0, pm1, p0, mm1, m0);
    __syncthreads();
    S.dpp[tid] = S.dp[odi];
    cp_wait_all();
    __syncthreads();
    // rotate to the loop's view at i = i0: x(i0-1..i0+2) = (x0, x1, x2, xm1), r(i0) = r1,
    // r(i0+1) = r0, rr(i0-1) = rrm1, rr(i0) = rr0, P(i0-1) = pm1, masks i0-1 .. i0+2 unchanged
    {
        int t = xm1;
        xm1 = x0;
        x0 = x1;
        x1 = x2;
        x2 = t;
        t = r0;
        r0 = r1;
        r1 = t;
    }
    gx += 5 * plane;  // plane i0+3
    gP += 3 * plane;  // plane i0+2
    gr += 3 * plane;  // plane i0+2
    gm += 4 * plane;  // plane i0+3
    float4* gout = xout + (i0 + 1) * plane + out_jk;

    for (int i = i0; i < i1; i++) {
        // stream x(i+3) into the slot of x(i-1), P(i+2) into P(i-1), r(i+2) into r(i)
        if (HAS_X) issue_x(xm1, i + 3, gx);
        issue_r(sP, pm1, i + 2, gP, P);
        issue_r(sr, r0, i + 2, gr, r);
        cp_commit();
        fetch_m(i + 3, gm);
        residual(i + 1, x0, x1, x2, r1, p1, m1, rrm1);
        __syncthreads();
        pressure(i, rr0, rrm1, p0, p1, m0, m1);
        __syncthreads();
        if (out_ok) {
            float4 xo = HAS_X ? S.x[x0 + oxi] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 rv = S.rr[rr0 + ori], pv = S.P[p0 + ori];
            const uint8_t mo = S.m[m0 + oxi];
            const bool cell = jk_cell && i < n;
            const bool own_col = ((i & 1) ^ opar) == 0;  // (i + j + k + flag) even
            const bool own_red = cell && own_col;
            const float dpown = S.dp[odi];
            if (own_red) xo.x += dpown;
            // the lower cells have the other colour: red exactly when the own colour is black
            const bool lo_ok[3] = {!own_col && i >= 1 && jk_cell, !own_col && lo_j_ok && i < n, !own_col && lo_k_ok && i < n};
            const float dplo[3] = {S.dpp[tid], S.dp[odi - DK], S.dp[odi - 1]};
            const float rf[3] = {rv.y, rv.z, rv.w}, pf[3] = {pv.y, pv.z, pv.w};
            const uint8_t bit[3] = {MU, MV, MW};
            float upd[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                upd[d] = 0.f;
                if (!own_red && !lo_ok[d]) continue;
                const bool fix = mo & bit[d];
                const float v = fix ? 0.f : vol;
                const float D = fix ? 1.f : v6 + pf[d];
                upd[d] = __fdividef(rf[d] - (own_red ? -v : v) * (own_red ? dpown : dplo[d]), D);
            }
            xo.y += upd[0];
            xo.z += upd[1];
            xo.w += upd[2];
            *gout = xo;
        }
        store_m(mm1);  // mask (i+3) into the slot of mask (i-1)
        cp_wait_all();
        __syncthreads();
        S.dpp[tid] = S.dp[odi];
        // rotate the rings and advance the plane pointers
        {
            int t = xm1;
            xm1 = x0;
            x0 = x1;
            x1 = x2;
            x2 = t;
            t = pm1;
            pm1 = p0;
            p0 = p1;
            p1 = t;
            t = r0;
            r0 = r1;
            r1 = t;
            t = rrm1;
            rrm1 = rr0;
            rr0 = t;
            t = mm1;
            mm1 = m0;
            m0 = m1;
            m1 = m2;
            m2 = t;
        }
        gx += plane;
        gP += plane;
        gr += plane;
        gm += plane;
        gout += plane;
    }
}

// ---------------------------------------------------------------- Laplacian-form sweep, TMA staging
// The Laplacian-form sweep with the planes of x, r and P staged by the tensor-memory
// accelerator: one thread issues one cp.async.bulk.tensor box load per plane and array
// (x: 36 x 12 slots, r and P: 34 x 10 slots, 16 bytes each) into the ring slot, with an
// mbarrier counting the bytes, instead of every thread issuing 16-byte copies. The boxes
// read zero outside the allocation, as the copies did. Everything else is k_sweep_lap.
constexpr int RNP = 344;  // r / P ring slot in float4s: RN padded to 128 bytes (TMA destinations)
constexpr unsigned XBYTES = XN * 16, RBYTES = RN * 16;
static_assert(RNP >= RN && (RNP * 16) % 128 == 0 && (XN * 16) % 128 == 0, "TMA ring slots must be 128-byte aligned");

struct SmemT {
    float4 x[4 * XN];
    float4 P[3 * RNP];
    float4 r[2 * RNP];
    float4 rr[2 * RN];
    float dp[DJ * DK];
    float dpp[SJ * SK];
    uint8_t m[4 * XN];
    unsigned long long bar;
};

// 3D box load of the tensor map at coordinates (c0, c1, c2) into shared memory, counted on bar
__device__ __forceinline__ void tma3(unsigned dst, const CUtensorMap* map, int c0, int c1, int c2, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// arrive on bar expecting `bytes` of transfers in the current phase
__device__ __forceinline__ void arm_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// waits for the phase of the given parity to complete; false after about a second
__device__ __forceinline__ bool wait_phase(unsigned bar, unsigned parity) {
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while (true) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        unsigned long long t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 1000000000ull) return false;
    }
}

__device__ __forceinline__ void fail(int* err) {
    if (threadIdx.x == 0 && threadIdx.y == 0) atomicExch(err, 1);
}

// (the adapters' sweep: the reference smoother to FP32 rounding)
template <bool HAS_X>
__global__ void __launch_bounds__(NT, 3) k_sweep_tma(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmr,
                                                    const __grid_constant__ CUtensorMap tmp, Geom g, float vol,
                                                    float4* __restrict__ xout, const uint8_t* __restrict__ m, int flag, int chunk,
                                                    int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SmemT& S = *reinterpret_cast<SmemT*>(smem_raw);
    float4* RR = S.rr;
    const int n = g.n;
    const int tk = threadIdx.x, tj = threadIdx.y, tid = tj * SK + tk;
    const int k0 = blockIdx.x * SK, j0 = blockIdx.y * SJ, i0 = blockIdx.z * chunk;
    const int i1 = i0 + chunk >= n ? n + 1 : i0 + chunk;  // the last chunk also takes plane n
    const int j = j0 + tj, k = k0 + tk;
    const float v6 = 6.f * vol;

    // staging elements: x / mask region (X) and P / r region (R), two per thread
    const Stage X0 = make_stage(g, tid, XN, XK, j0 - 2, k0 - 2), X1 = make_stage(g, tid + NT, XN, XK, j0 - 2, k0 - 2);
    const unsigned sx = (unsigned)__cvta_generic_to_shared(S.x), sP = (unsigned)__cvta_generic_to_shared(S.P),
                   sr = (unsigned)__cvta_generic_to_shared(S.r);

    // residual elements: rr/P index e and x/mask index xi, and whether (j,k) lies in [0,n]^2
    const int re0 = tid, re1 = tid + NT;
    const int rx0 = re0 + (re0 / RK) * (XK - RK) + XK + 1, rx1 = re1 + (re1 / RK) * (XK - RK) + XK + 1;
    auto in_box = [&](int e) {
        int jj = j0 - 1 + e / RK, kk = k0 - 1 + e % RK;
        return e < RN && jj >= 0 && jj <= n && kk >= 0 && kk <= n;
    };
    const bool rb0 = in_box(re0), rb1 = in_box(re1);

    // pressure-phase cell of this thread for the two plane parities
    const int pdj = tid / DRED, pq = tid % DRED, pj = j0 - 1 + pdj;
    const bool p_thread = tid < DJ * DRED;
    const int ppar0 = (pj + flag - (k0 - 1)) & 1;  // dk = ((p & 1) ^ ppar0) + 2 pq
    // (the two parities as scalars: a runtime-indexed array would live in local memory)
    const int pdk0 = 2 * pq, pdk1 = 2 * pq + 1;
    const bool pok0 = p_thread && pdk0 < DK && pj >= 0 && k0 - 1 + pdk0 >= 0 && pj < n && k0 - 1 + pdk0 < n;
    const bool pok1 = p_thread && pdk1 < DK && pj >= 0 && k0 - 1 + pdk1 >= 0 && pj < n && k0 - 1 + pdk1 < n;

    // update-phase slot
    const bool out_ok = j <= n && k <= n;
    const long long out_jk = (long long)(j + 1) * g.sz + (k + 1);
    const int oxi = (tj + 2) * XK + (tk + 2), ori = (tj + 1) * RK + (tk + 1), odi = (tj + 1) * DK + (tk + 1);
    // the grid's tiles cover [0, n) in j and k: where a tile ends at n, its last lane in k
    // (last row in j) also writes the slot at k = n (j = n)
    const bool ext_k = tk == SK - 1 && k + 1 == n && j <= n, ext_j = tj == SJ - 1 && j + 1 == n && k <= n;

    // plane p of x (region origin j0-2, k0-2) or of r / P (origin j0-1, k0-1) into a ring
    // slot by one TMA box load each; out-of-allocation parts of a box read as zero
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&S.bar);
    auto tma_x = [&](int slot, int p) { tma3(sx + 16u * slot, &tmx, 4 * (k0 - 1), j0 - 1, p + 1, bar); };
    auto tma_r = [&](unsigned base, int slot, int p, const CUtensorMap* tm) { tma3(base + 16u * slot, tm, 4 * k0, j0, p + 1, bar); };
    auto tma_p = [&](int slot, int p) { tma3(sP + 16u * slot, &tmp, 4 * k0, j0, p + 1, bar); };
    uint32_t phase = 0;
    // every thread waits for the current phase; a wait that gives up (about a second) makes
    // the whole block record the error and leave at the next barrier
    auto wait_loads = [&]() {
        const bool ok = wait_phase(bar, phase);
        phase ^= 1u;
        return ok;
    };
    uint8_t mr0 = MALL, mr1 = MALL;
    auto fetch_m = [&](int p, const uint8_t* src) {
        const bool pok = p >= -1 && p <= n + 1;
        mr0 = (pok && X0.jk >= 0) ? __ldg(src + X0.jk) : (uint8_t)MALL;
        mr1 = (pok && X1.jk >= 0) ? __ldg(src + X1.jk) : (uint8_t)MALL;
    };
    auto store_m = [&](int slot) {
        if (X0.s >= 0) S.m[slot + X0.s] = mr0;
        if (X1.s >= 0) S.m[slot + X1.s] = mr1;
    };

    // residual of plane p: x slots (p-1, p, p+1), r / P / mask slots of p, into rr slot
    auto residual = [&](int p, int xa, int xb, int xc, int rs, int ps, int ms, int rrs) {
        const bool pin = p >= 0 && p <= n;
        auto one = [&](int e, int xi, bool box) {
            float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pin && box) {
                const float4 rv = S.r[rs + e];
                if (HAS_X) {
                    auto q = [&](int idx) {
                        const float4 v = S.x[idx];
                        return Q4<float>{v.x, v.y, v.z, v.w};
                    };
                    const float4 pv = S.P[ps + e];
                    float o[4];
                    lap_core<float>(q(xb + xi), q(xa + xi), q(xc + xi), q(xb + xi - XK), q(xb + xi + XK), q(xb + xi - 1),
                                    q(xb + xi + 1), Q4<float>{pv.x, pv.y, pv.z, pv.w}, vol, o);
                    o[0] = rv.x - o[0];
                    o[1] = rv.y - o[1];
                    o[2] = rv.z - o[2];
                    o[3] = rv.w - o[3];
                    mask4<float>(S.m[ms + xi], o);
                    out = make_float4(o[0], o[1], o[2], o[3]);
                } else {
                    out = rv;  // r is zero on fixed unknowns
                }
            }
            RR[rrs + e] = out;
        };
        one(re0, rx0, rb0);
        if (re1 < RN) one(re1, rx1, rb1);
    };

    // pressure update of the red cells of plane p (rr slots p, p+1; P slots p, p+1; mask slots p, p+1)
    auto pressure = [&](int p, int rr0, int rr1, int p0, int p1, int m0s, int m1s) {
        const int b = (p & 1) ^ ppar0;
        if (!(b ? pok1 : pok0) || p < 0 || p >= n) return;
        const int dk = b ? pdk1 : pdk0;
        const int ri = pdj * RK + dk, xi = (pdj + 1) * XK + (dk + 1);
        const float4 rc = RR[rr0 + ri], pc = S.P[p0 + ri];
        const uint8_t mo = S.m[m0s + xi];
        const float rL[3] = {rc.y, rc.z, rc.w}, pL[3] = {pc.y, pc.z, pc.w};
        const uint8_t mhi[3] = {S.m[m1s + xi], S.m[m0s + xi + XK], S.m[m0s + xi + 1]};
        const float rh[3] = {RR[rr1 + ri].y, RR[rr0 + ri + RK].z, RR[rr0 + ri + 1].w};
        const float ph[3] = {S.P[p1 + ri].y, S.P[p0 + ri + RK].z, S.P[p0 + ri + 1].w};
        const uint8_t bit[3] = {MU, MV, MW};
        float num = rc.x, den = 2.f * pc.x;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const float vL = (mo & bit[d]) ? 0.f : vol, vR = (mhi[d] & bit[d]) ? 0.f : vol;
            const float iL = __fdividef(vL, v6 + pL[d]), iR = __fdividef(vR, v6 + ph[d]);
            num += rL[d] * iL - rh[d] * iR;
            den -= vL * iL + vR * iR;
        }
        S.dp[pdj * DK + dk] = den != 0.f ? __fdividef(num, den) : 0.f;
    };

    // ring slots as element offsets (rotated each plane)
    int xm1 = 0 * XN, x0 = 1 * XN, x1 = 2 * XN, x2 = 3 * XN;  // x(i-1), x(i), x(i+1), x(i+2)
    int pm1 = 0 * RNP, p0 = 1 * RNP, p1 = 2 * RNP;         // P(i-1), P(i), P(i+1)
    int r0 = 0 * RNP, r1 = 1 * RNP;                           // r(i), r(i+1)
    int rrm1 = 0 * RN, rr0 = 1 * RN;                          // rr(i-1), rr(i)
    int mm1 = 0 * XN, m0 = 1 * XN, m1 = 2 * XN, m2 = 3 * XN;  // masks of planes i-1 .. i+2

    // new x of slot (i, jj, kk) of the current plane (x / mask index xi, rr / P index ri,
    // dp index di of its own cell), written to dst: the pressure of an own red cell, and
    // each face whose red block is the own cell (red) or the cell below it (the own cell
    // black). dp is read only where that red cell exists, so the high-side slots (jj or
    // kk = n) read nothing outside the dp region; dpp (the cell below in i) only for the
    // thread's own (j, k).
    auto update = [&](int i, int jj, int kk, int xi, int ri, int di, float4* dst) {
        float4 xo = HAS_X ? S.x[x0 + xi] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 rv = RR[rr0 + ri], pv = S.P[p0 + ri];
        const uint8_t mo = S.m[m0 + xi];
        const bool jkc = jj < n && kk < n;
        const bool own_col = ((i + jj + kk + flag) & 1) == 0;
        const bool own_red = jkc && i < n && own_col;
        const float dpown = own_red ? S.dp[di] : 0.f;
        if (own_red) xo.x += dpown;
        // the lower cells have the other colour: red exactly when the own colour is black
        const bool lo_ok[3] = {!own_col && i >= 1 && jkc, !own_col && jj >= 1 && kk < n && i < n,
                               !own_col && kk >= 1 && jj < n && i < n};
        const float dplo[3] = {lo_ok[0] ? S.dpp[tid] : 0.f, lo_ok[1] ? S.dp[di - DK] : 0.f, lo_ok[2] ? S.dp[di - 1] : 0.f};
        const float rf[3] = {rv.y, rv.z, rv.w}, pf[3] = {pv.y, pv.z, pv.w};
        const uint8_t bit[3] = {MU, MV, MW};
        float upd[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            upd[d] = 0.f;
            if (!own_red && !lo_ok[d]) continue;
            const bool fix = mo & bit[d];
            const float v = fix ? 0.f : vol;
            const float D = fix ? 1.f : v6 + pf[d];
            upd[d] = __fdividef(rf[d] - (own_red ? -v : v) * (own_red ? dpown : dplo[d]), D);
        }
        xo.y += upd[0];
        xo.z += upd[1];
        xo.w += upd[2];
        *dst = xo;
    };

    // prologue: planes i0-2 .. i0+1 of x, i0-1 .. i0+1 of P, i0-1 and i0 of r, masks i0-1 .. i0+2
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        arm_tx(bar, (HAS_X ? 4 * XBYTES : 0) + 3 * RBYTES + 2 * RBYTES);
        if (HAS_X) {
            tma_x(xm1, i0 - 2);
            tma_x(x0, i0 - 1);
            tma_x(x1, i0);
            tma_x(x2, i0 + 1);
        }
        tma_p(pm1, i0 - 1);
        tma_p(p0, i0);
        tma_p(p1, i0 + 1);
        tma_r(sr, r0, i0 - 1, &tmr);
        tma_r(sr, r1, i0, &tmr);
    }
    const long long plane = (long long)g.sy * g.sz;
    const uint8_t* gm = m + i0 * plane;  // plane i0-1
    fetch_m(i0 - 1, gm);
    store_m(mm1);
    fetch_m(i0, gm + plane);
    store_m(m0);
    fetch_m(i0 + 1, gm + 2 * plane);
    store_m(m1);
    fetch_m(i0 + 2, gm + 3 * plane);
    store_m(m2);
    if (__syncthreads_or(!wait_loads())) return fail(err);
    // residual of i0-1: x(i0-2, i0-1, i0) = slots (xm1, x0, x1), r(i0-1) = r0, P(i0-1) = pm1, mask(i0-1) = mm1
    residual(i0 - 1, xm1, x0, x1, r0, pm1, mm1, rrm1);
    __syncthreads();
    if (tid == 0) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        arm_tx(bar, (HAS_X ? XBYTES : 0) + RBYTES);
        if (HAS_X) tma_x(xm1, i0 + 2);  // x(i0+2) replaces x(i0-2)
        tma_r(sr, r0, i0 + 1, &tmr);    // r(i0+1) replaces r(i0-1)
    }
    // residual of i0: x(i0-1, i0, i0+1) = (x0, x1, x2), r(i0) = r1, P(i0) = p0, mask(i0) = m0
    residual(i0, x0, x1, x2, r1, p0, m0, rr0);
    __syncthreads();
    pressure(i0 - 1, rrm1, rr0, pm1, p0, mm1, m0);
    __syncthreads();
    S.dpp[tid] = S.dp[odi];
    if (__syncthreads_or(!wait_loads())) return fail(err);
    // rotate to the loop's view at i = i0: x(i0-1..i0+2) = (x0, x1, x2, xm1), r(i0) = r1,
    // r(i0+1) = r0, rr(i0-1) = rrm1, rr(i0) = rr0, P(i0-1) = pm1, masks i0-1 .. i0+2 unchanged
    {
        int t = xm1;
        xm1 = x0;
        x0 = x1;
        x1 = x2;
        x2 = t;
        t = r0;
        r0 = r1;
        r1 = t;
    }
    gm += 4 * plane;  // plane i0+3
    float4* gout = xout + (i0 + 1) * plane + out_jk;

    for (int i = i0; i < i1; i++) {
        // stream x(i+3) into the slot of x(i-1), P(i+2) into P(i-1), r(i+2) into r(i)
        if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            arm_tx(bar, (HAS_X ? XBYTES : 0) + RBYTES + RBYTES);
            if (HAS_X) tma_x(xm1, i + 3);
            tma_p(pm1, i + 2);
            tma_r(sr, r0, i + 2, &tmr);
        }
        fetch_m(i + 3, gm);
        residual(i + 1, x0, x1, x2, r1, p1, m1, rrm1);
        __syncthreads();
        pressure(i, rr0, rrm1, p0, p1, m0, m1);
        __syncthreads();
        if (out_ok) {
            update(i, j, k, oxi, ori, odi, gout);
            // the last tile in k (j) also writes column k = n (row j = n): slots whose only
            // unknowns are the faces on the box's high side, updated by the cells below them
            if (ext_k) update(i, j, k + 1, oxi + 1, ori + 1, odi + 1, gout + 1);
            if (ext_j) update(i, j + 1, k, oxi + XK, ori + RK, odi + DK, gout + g.sz);
            if (ext_j && ext_k) update(i, j + 1, k + 1, oxi + XK + 1, ori + RK + 1, odi + DK + 1, gout + g.sz + 1);
        }
        store_m(mm1);  // mask (i+3) into the slot of mask (i-1)
        if (__syncthreads_or(!wait_loads())) return fail(err);
        S.dpp[tid] = S.dp[odi];
        // rotate the rings and advance the plane pointers
        {
            int t = xm1;
            xm1 = x0;
            x0 = x1;
            x1 = x2;
            x2 = t;
            t = pm1;
            pm1 = p0;
            p0 = p1;
            p1 = t;
            t = r0;
            r0 = r1;
            r1 = t;
            t = rrm1;
            rrm1 = rr0;
            rr0 = t;
            t = mm1;
            mm1 = m0;
            m0 = m1;
            m1 = m2;
            m2 = t;
        }
        gm += plane;
        gout += plane;
    }
}

// ---------------------------------------------------------------- sweep by cells
// The solver's own Laplacian-form sweep (FP16 penalty copy), one thread per red cell: the
// cell's pressure and six faces are exactly the unknowns its block solve changes, and every
// face belongs to one red cell, so a thread forms the seven residuals, solves and updates
// without exchanging residuals or pressure updates with other threads, without a halo of
// redundant residuals, and without the black pressures' rows, which nothing uses.
//
// A block covers TK (k) x TJ (j) slots, TK TJ = 256, and marches along i; a thread owns the
// slot pair (k0 + 2 kk, k0 + 2 kk + 1) of its row, one red and one black slot in every plane.
// Planes of x (one slot more on the low and two on the high side), r and P are staged by one
// TMA box load each, a plane ahead of their use (x ring of five planes, r and P of three).
// Neighbouring lanes work on neighbouring rows, whose red slots have opposite k parity, so a
// warp's 16-byte loads of its red cells (every second slot of two rows) and of any one
// neighbour of theirs fall into distinct banks.
//
// Output: the red slot leaves with its cell. The black slot gets u from the thread's own red
// cell of the plane before, v and w from its neighbours' cells through shared memory, and is
// written a plane later, after the barrier. Faces on the tile's and the chunk's high side
// belong to another block's black slot: they are stored alone, and that block leaves the
// component out. Slots at i, j or k = n hold fixed faces only: 0.
//
// MODE 0: x = 0 (the first sweep: the residual is r); 1: x from memory; 2: x + the parent
// coarse value (the injection: a fine fixed unknown's parent is fixed, so its value is 0),
// added to every plane of x once it has landed; 3 (PAIR): the first two sweeps, colour flag from
// x = 0 and then the other, in one launch. All that a cell of the second colour needs of x are
// its six neighbours, cells of the first. So r and P are staged with one cell more on every
// side, half of the warps form the first colour's cells two planes ahead (p and low faces, high
// faces: sixteen bytes each, twelve loads instead of nineteen for the six neighbours), and the
// others run the second colour from there: r and P are read once, and the first sweep's x is
// neither written nor read; 4: the same from x, with the parents where xc is given (the two sweeps
// after the coarse correction): x lands with two slots more on every side, and the first colour's
// cells hand on the pressure of the pair's other cell too.
//
// Bound: the chain of a plane (land, work, barrier), which four blocks an SM overlap, three of
// PAIR; at 256^3 HBM too (MODE 1 moves 0.98 GB in 180 us, 5.4 TB/s or 0.80 of the measured
// copy; MODE 2 197 us). The form with one thread a slot, residuals exchanged through shared
// memory and 17 instead of 5.7 warp instructions a slot took 290 us; tiles of 512 slots with
// half as many blocks 186 and 204 us. PAIR takes 216 us at 256^3, 33 at 128^3, 9.6 at 64^3 and
// 5.2 at 32^3 against 316, 44, 13.9 and 8.8 of MODE 0 and MODE 1 one after the other; with
// 256-cell tiles in slot order and two blocks an SM it took 250 us, with loads three planes ahead
// 240, with two warps more for the cells around the tile 239.
// MODE 4 holds two blocks an SM: 15.8 us at 64^3 and 8.0 at 32^3 against 17.4 and 9.6 of MODE 2
// and MODE 1, but 420 at 256^3 against 377 (solver.cu fuse_post).
// Staging x by component instead, with 4-byte asynchronous copies (255 us for MODE 1) or through
// registers (270 us), was slower: the transposing stores and the scattered loads of r and P
// then bound it.
template <int TK, bool PAIR = false, bool WIDE = false>
struct CellTile {
    static constexpr int NT = 128;            // threads with a pair of slots
    static constexpr int TJ = 2 * NT / TK, LR = TK / 2;    // rows, pairs of a row
    static constexpr int PW = LR < 16 ? LR : 16;           // pairs of a row in one warp
    // staged x: k0 - 2 .. k0 + TK + 1, j0 - 1 .. j0 + TJ + 1; WIDE (PAIR with x): one cell more on every side
    static constexpr int OX = WIDE ? 1 : 0, XW = TK + 4 + 2 * OX, XR = TJ + 3 + 2 * OX;
    static constexpr int O = PAIR ? 1 : 0;                 // PAIR: r and P of one cell more on every side
    static constexpr int RW = TK + 2 + 2 * O, RR = TJ + 1 + 2 * O;  // staged r and P: k0 - O .. (P: k0 - 1 ..), j0 - O .. j0 + TJ + O
    static constexpr int XPL = (XW * XR + 7) / 8 * 8;      // ring slots, 128-byte multiples (in slots)
    static constexpr int RPL = (RW * RR + 7) / 8 * 8, PPL = (RW * RR + 15) / 16 * 16;
    static constexpr unsigned XB = XW * XR * 16, RB = RW * RR * 16, PB = RW * RR * 8;  // box bytes
    static constexpr int XRING = 5, RRING = PAIR ? 5 : 3;
    // PAIR: first-colour cells by row and pair, low and high halves; a row is four slots off a
    // multiple of 128 bytes, as the two rows of a warp have to be
    static constexpr int FW = LR + 4, FPL = FW * (TJ + 2), FRING = 4;
    static constexpr int VN = 2 * (TJ + 1) * LR, WN = (2 * TJ * (LR + 1) + 1) / 2 * 2;  // sv, sw (floats)
    static constexpr int HALO = 2 * LR + TJ;               // PAIR: first-colour cells around the tile
    static constexpr int THREADS = PAIR ? 2 * NT : NT;
    static constexpr int NX = (XW * XR + THREADS - 1) / THREADS;  // staged x slots of a thread (with parents)
    static constexpr int smem(bool x) { return (PAIR ? FRING * FPL * 32 : 0) + (x ? XRING * XPL * 16 : 0) + RRING * (RPL * 16 + PPL * 8) + 4 * (VN + WN) + 8; }
    static_assert((RRING * PPL * 8 + 4 * VN) % 8 == 0, "the mbarrier lies on an 8-byte boundary");
    static_assert(!PAIR || (FW % 8 == 4 && FPL % 4 == 0), "the staged planes start on 128 bytes");
};

template <int TK, int MODE>
__global__ void __launch_bounds__(CellTile<TK, MODE >= 3>::THREADS, MODE == 3 ? 3 : MODE == 4 ? 2 : 4) k_sweep_cell(
    const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmr,
    const __grid_constant__ CUtensorMap tmp, Geom g, float vol,
    float4* __restrict__ xout, const float* __restrict__ pscale, int flag,
    int chunk, int* __restrict__ err, const float4* __restrict__ xc, int c_plane,
    int c_sz) {
    constexpr bool PAIR = MODE >= 3, STAGE_X = MODE == 1 || MODE == 2 || MODE == 4;
    using C = CellTile<TK, PAIR, MODE == 4>;
    const bool parents = MODE == 2 || (MODE == 4 && xc);
    constexpr int NT = C::NT, TJ = C::TJ, XW = C::XW, RW = C::RW, FW = C::FW;
    // (no static shared memory: the TMA destinations start at the window's aligned origin)
    extern __shared__ __align__(1024) unsigned char cell_smem[];
    float4* sf = reinterpret_cast<float4*>(cell_smem);
    float4* sx = sf + (PAIR ? 2 * C::FRING * C::FPL : 0);
    float4* sr = sx + (STAGE_X ? C::XRING * C::XPL : 0);
    uint2* sp = reinterpret_cast<uint2*>(sr + C::RRING * C::RPL);
    float (*sv)[TJ + 1][C::LR] = reinterpret_cast<float (*)[TJ + 1][C::LR]>(sp + C::RRING * C::PPL);  // [2]
    float (*sw)[TJ][C::LR + 1] = reinterpret_cast<float (*)[TJ][C::LR + 1]>(reinterpret_cast<float*>(sv) + C::VN);  // [2]
    unsigned long long* s_bar = reinterpret_cast<unsigned long long*>(reinterpret_cast<float*>(sw) + C::WN);
    const int n = g.n, tid = threadIdx.x, ct = tid & (NT - 1), lane = tid & 31, pr = lane >> 1;
    constexpr int WR = 32 / C::PW, WK = C::LR / C::PW;  // rows of a warp, warps side by side in k
    const int wid = ct >> 5;
    const int tj = (wid / WK) * WR + 2 * (pr / C::PW) + (lane & 1), kk = (wid % WK) * C::PW + pr % C::PW;
    const int k0 = blockIdx.x * TK, j0 = blockIdx.y * TJ, i0 = blockIdx.z * chunk;
    const int i1 = min(i0 + chunk, n);
    const int j = j0 + tj, kp0 = k0 + 2 * kk;
    const bool first = PAIR && tid >= NT;  // forms the first colour's cells
    const bool live = j < n && kp0 < n && !first;
    const int colour = PAIR ? flag ^ 1 : flag;  // written by the others
    const int plane = g.sy * g.sz;
    const float psc = __ldg(pscale), v6 = 6.f * vol;

    // box loads counted on one mbarrier; plane p of the box sits at p + 1 in the arrays, row j
    // at j + 1, slot k at k + 1 (coordinates in 8-byte units along k)
    const unsigned bar = (unsigned)__cvta_generic_to_shared(s_bar);
    const unsigned bx = (unsigned)__cvta_generic_to_shared(sx), br = (unsigned)__cvta_generic_to_shared(sr),
                   bp_ = (unsigned)__cvta_generic_to_shared(sp);
    auto xslot = [&](int p) { return ((p + C::XRING) % C::XRING) * C::XPL; };
    auto load_x = [&](int p) { tma3(bx + 16u * xslot(p), &tmx, 2 * (k0 - 1), j0 - C::OX, p + 1, bar); };
    auto load_rp = [&](int p) {
        const int s = (p + C::RRING) % C::RRING;
        tma3(br + 16u * (s * C::RPL), &tmr, 2 * (k0 + 1 - C::O), j0 + 1 - C::O, p + 1, bar);
        tma3(bp_ + 8u * (s * C::PPL), &tmp, k0, j0 + 1 - C::O, p + 1, bar);
    };
    unsigned phase = 0;
    auto wait_loads = [&]() {
        const bool ok = wait_phase(bar, phase);
        phase ^= 1u;
        return ok;
    };

    // MODE 2: the parent values of the thread's share of a staged plane, and adding them
    float4 cv[C::NX];
    int co[C::NX];  // offset in a coarse plane, -1: none
    if (parents) {
#pragma unroll
        for (int q = 0; q < C::NX; q++) {
            const int e = tid + q * C::THREADS, jj = j0 - 1 - C::OX + e / XW, k = k0 - 2 + e % XW;
            co[q] = e < XW * C::XR && k >= -1 && jj >= -1 && jj <= n + 1 && k <= n + 1 ? ((jj >> 1) + 1) * c_sz + ((k >> 1) + 1) : -1;
        }
    }
    auto fetch_coarse = [&](int p) {
        const float4* src = xc + (long long)((p >> 1) + 1) * c_plane;
#pragma unroll
        for (int q = 0; q < C::NX; q++)
            if (co[q] >= 0)  // (volatile: issued here, not where the values are used)
                asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                             : "=f"(cv[q].x), "=f"(cv[q].y), "=f"(cv[q].z), "=f"(cv[q].w)
                             : "l"(src + co[q]));
    };
    auto add_coarse = [&](int p) {
        float4* dst = sx + xslot(p) + tid;
#pragma unroll
        for (int q = 0; q < C::NX; q++) {
            if (co[q] < 0) continue;
            float4 v = dst[q * C::THREADS];
            v.x += cv[q].x;
            v.y += cv[q].y;
            v.z += cv[q].z;
            v.w += cv[q].w;
            dst[q * C::THREADS] = v;
        }
    };

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        arm_tx(bar, (STAGE_X ? (4 + C::OX) * C::XB : 0) + (PAIR ? 5 : 2) * (C::RB + C::PB));
        if (STAGE_X)
            for (int p = i0 - 1 - C::OX; p <= i0 + 2; p++) load_x(p);
        for (int p = PAIR ? i0 - 1 : i0; p <= (PAIR ? i0 + 3 : i0 + 1); p++) load_rp(p);
    }
    auto add_parents = [&](int first_plane, int last_plane) {  // planes 2 P and 2 P + 1 share their parents
        for (int p = first_plane; p <= last_plane; p++) {
            if (p > first_plane && ((p & 1) == 0)) fetch_coarse(p);
            add_coarse(p);
        }
    };
    if (parents) fetch_coarse(i0 - 1 - C::OX);
    if (__syncthreads_or(!wait_loads())) return fail(err);
    if (parents) {
        add_parents(i0 - 1 - C::OX, i0 + 2);
        __syncthreads();
    }

    // PAIR: the first colour's cells of plane p in the tile and around it (0 outside the domain):
    // pressure and low faces, high faces and the pressure of the pair's other cell; pair -1 and
    // LR are the cells beside a row
    auto fcell = [&](int p) { return sf + 2 * (p & (C::FRING - 1)) * C::FPL; };
    auto first_cell = [&](int p, int row, int c) {
        const int jj = j0 + row, k = k0 + c;
        float p0 = 0.f, po = 0.f, lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
        if (p >= 0 && p < n && jj >= 0 && jj < n && k >= 0 && k < n) {
            const int sl = (p + C::RRING) % C::RRING, sn = sl + 1 < C::RRING ? sl + 1 : 0, ro = (row + 1) * RW + c + 1;
            const float4* R = sr + sl * C::RPL + ro;
            float raw[7];
            cell_penalty<RW>(sp + sl * C::PPL + ro, sp + sn * C::PPL + ro, psc, raw);
            const float4 r0 = *R;
            float res[7] = {r0.x, r0.y, r0.z, r0.w, sr[sn * C::RPL + ro].y, R[RW].z, R[1].w};
            if (MODE == 4) {
                const float4* B = sx + (row + 2) * XW + c + 2;
                slot_residual<XW>(B + xslot(p - 1), B + xslot(p), B + xslot(p + 1), B + xslot(p + 2), vol, raw, p0, lo, hi, res);
                po = B[xslot(p) + (c & 1 ? -1 : 1)].x;
            }
            p0 += cell_solve(vol, v6, raw, res, lo, hi);
        }
        float4* F = fcell(p) + (row + 1) * FW + ((c + 2) >> 1);
        F[0] = make_float4(p0, lo[0], lo[1], lo[2]);
        F[C::FPL] = make_float4(hi[0], hi[1], hi[2], po);
    };
    auto first_tile = [&](int p) { first_cell(p, tj, 2 * kk + ((p + j + flag) & 1)); };
    auto first_halo = [&](int p) {
        if (ct < 2 * C::LR) {  // the rows below and above
            const int row = ct < C::LR ? -1 : TJ;
            first_cell(p, row, 2 * (ct % C::LR) + ((p + j0 + row + flag) & 1));
        } else if (ct < C::HALO) {  // one cell of each row, left or right of it
            const int row = ct - 2 * C::LR;
            first_cell(p, row, (p + j0 + row + flag) & 1 ? -1 : TK);
        }
    };
    auto first_plane = [&](int p) {
        first_tile(p);
        first_halo(p);
    };
    if (PAIR) {
        if (first)
            first_plane(i0);
        else
            first_tile(i0 - 1);  // (nothing needs the cells around it)
        if (MODE == 4) {  // x of two planes more, in place of the first two
            __syncthreads();
            if (tid == 0) {
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                arm_tx(bar, 2 * C::XB);
                load_x(i0 + 3);
                load_x(i0 + 4);
            }
            if (parents && ((i0 + 3) & 1) == 0) fetch_coarse(i0 + 3);
            const bool ok = wait_loads();
            if (parents) add_parents(i0 + 3, i0 + 4);
            if (__syncthreads_or(!ok)) return fail(err);
        }
        if (first) first_plane(i0 + 1);
        __syncthreads();
    }

    float ukeep = 0.f;               // u of this plane's black slot: the last plane's cell's high face
    float bp = 0.f, bu = 0.f;        // p and u of the last plane's black slot
    const bool own_v = tj > 0 || j0 == 0;  // the black slots' v is this block's
    auto write_black = [&](int i) {  // black slot of plane i
        const int q = (i + j + colour) & 1;
        const int s = g.slot(i, j, kp0 + 1 - q);
        const bool own_u = i > i0 || i0 == 0, own_w = q == 0 || kk > 0 || k0 == 0;
        const float bv = tj > 0 ? sv[i & 1][tj][kk] : 0.f;
        const float bw = sw[i & 1][tj][q == 0 ? kk + 1 : kk];
        if (own_u && own_v && own_w) {
            xout[s] = make_float4(bp, bu, bv, q == 0 || kk > 0 ? bw : 0.f);
        } else {
            float* o = reinterpret_cast<float*>(xout + s);
            o[0] = bp;
            if (own_u) o[1] = bu;
            if (own_v) o[2] = bv;
            if (own_w) o[3] = q == 0 || kk > 0 ? bw : 0.f;
        }
    };

    int base = xslot(i0), rs = i0 % C::RRING;  // ring slots of plane i
    for (int i = i0; i < i1; i++) {
        const bool more = i + 1 < i1;
        // x(i + 3) into the slot of x(i - 2) (PAIR: i + 5, i), r and P of i + 2 (i + 4) into those of i - 1
        if (more && tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            arm_tx(bar, (STAGE_X ? C::XB : 0) + C::RB + C::PB);
            if (STAGE_X) load_x(PAIR ? i + 5 : i + 3);
            load_rp(PAIR ? i + 4 : i + 2);
        }
        if (parents && more && ((i + 3) & 1) == 0) fetch_coarse(PAIR ? i + 5 : i + 3);  // an odd plane's parents are the last plane's
        if (i > i0 && live) write_black(i - 1);
        const int rn = rs + 1 < C::RRING ? rs + 1 : 0;  // ring slot of r and P of plane i + 1
        if (PAIR && first && more) first_plane(i + 2);
        if (live) {
            const int q = (i + j + colour) & 1;  // red: (i + j + k + colour) even, k0 even
            const int ro = (tj + C::O) * RW + 2 * kk + q + C::O;
            const float4* R = sr + rs * C::RPL + ro;
            float raw[7];
            cell_penalty<RW>(sp + rs * C::PPL + ro + 1 - C::O, sp + rn * C::PPL + ro + 1 - C::O, psc, raw);
            const float4 r0 = *R;
            float res[7] = {r0.x, r0.y, r0.z, r0.w, sr[rn * C::RPL + ro].y, R[RW].z, R[1].w};
            float p0 = 0.f, pb = 0.f, lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
            if (PAIR) {
                const int o = (tj + 1) * FW + kk + 1;
                if (MODE == 4) p0 = fcell(i)[C::FPL + o].w;
                neighbour_residual<FW, C::FPL>(fcell(i - 1) + o, fcell(i) + o, fcell(i + 1) + o, q, vol, raw, p0, lo, hi, res, pb);
            } else if (MODE) {
                constexpr int XP = C::XPL, XL = (C::XRING - 1) * XP;
                const float4* B = sx + base + (tj + 1) * XW + 2 * kk + q + 2;
                const float4* A = B + (base >= XP ? -XP : XL);                             // plane i - 1
                const float4* D = B + (base < XL ? XP : -XL);                              // plane i + 1
                const float4* E = B + (base < XL - XP ? 2 * XP : -(C::XRING - 2) * XP);    // plane i + 2
                slot_residual<XW>(A, B, D, E, vol, raw, p0, lo, hi, res);
                pb = q ? B[-1].x : B[1].x;
            }
            const float dp = cell_solve(vol, v6, raw, res, lo, hi);
            const int k = kp0 + q;
            const int s = g.slot(i, j, k);
            xout[s] = make_float4(p0 + dp, lo[0], lo[1], lo[2]);
            // high faces that lie in another block's slots
            if (!more && i1 < n) reinterpret_cast<float*>(xout + s + plane)[1] = hi[0];
            if (tj == TJ - 1 && j + 1 < n) reinterpret_cast<float*>(xout + s + g.sz)[2] = hi[1];
            if (q && kk == C::LR - 1 && k + 1 < n) reinterpret_cast<float*>(xout + s + 1)[3] = hi[2];
            sv[i & 1][tj + 1][kk] = hi[1];
            sw[i & 1][tj][kk + 1] = hi[2];
            bp = pb;
            bu = ukeep;
            ukeep = hi[0];
        }
        base = base < (C::XRING - 1) * C::XPL ? base + C::XPL : 0;
        rs = rn;
        if (!more) break;
        const bool ok = wait_loads();
        if (parents) add_coarse(PAIR ? i + 5 : i + 3);
        if (__syncthreads_or(!ok)) return fail(err);
    }
    __syncthreads();
    if (live) write_black(i1 - 1);
    // the slots at k, j and i = n
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool end_k = k0 + TK >= n, end_j = j0 + TJ >= n;
    const int ie = i1 == n ? n : i1 - 1;  // the last chunk also takes plane n
    for (int i = i0; i <= ie; i++) {
        if (i == n && live) xout[g.slot(n, j, kp0)] = xout[g.slot(n, j, kp0 + 1)] = z;
        if (end_k && kk == 0 && j < n) xout[g.slot(i, j, n)] = z;
        if (end_j && tj == 0 && kp0 < n) xout[g.slot(i, n, kp0)] = xout[g.slot(i, n, kp0 + 1)] = z;
        if (end_k && end_j && tid == 0) xout[g.slot(i, n, n)] = z;
    }
}

}  // namespace

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's tensor-map encoder, fetched through the runtime (no link against the driver
// library); null when unavailable, in which case the sweep stages with cp.async
EncodeTiled encoder() {
    static EncodeTiled fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
        cudaGetLastError();
    }
    return fn;
}

// tensor map of a slot array of g as FP32 [planes][rows][4 (n+4)], box (4 bk) x bj x 1
bool slot_map(EncodeTiled enc, CUtensorMap* map, const void* base, const Geom& g, int bk, int bj) {
    const cuuint64_t dims[3] = {(cuuint64_t)g.sz * 4, (cuuint64_t)g.sy, (cuuint64_t)g.sx};
    const cuuint64_t strides[2] = {(cuuint64_t)g.sz * 16, (cuuint64_t)g.sy * g.sz * 16};
    const cuuint32_t box[3] = {(cuuint32_t)(4 * bk), (cuuint32_t)bj, 1}, es[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// per device: kernel attributes set, and the flag a TMA sweep sets when its wait gave up
bool g_attr_set[MAX_DEVICES] = {}, g_tattr_set[MAX_DEVICES] = {};
int* g_sweep_err[MAX_DEVICES] = {};
int g_sms[MAX_DEVICES] = {};

// Planes per block of the sweep by cells on an n^3 box: a block marches through its chunk
// plane after plane (its prologue costs about four), and the blocks run in waves of SMs x
// resident blocks, so the chunk minimises waves x (chunk + 4), the longest chain of planes an
// SM works through (n = 256: 37 planes in three waves, n = 128: 15 in one, n = 64: 2 in one).
int cell_chunk(int dev, int n, int tk, int tj, int resident) {
    if (!g_sms[dev] && cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) g_sms[dev] = 0;
    const long long slots = (long long)resident * (g_sms[dev] > 0 ? g_sms[dev] : 152);
    const long long plane_blocks = (long long)((n + tk - 1) / tk) * ((n + tj - 1) / tj);
    int best = 1;
    long long best_cost = -1;
    for (int c = 1; c <= n; c++) {
        const long long blocks = plane_blocks * ((n + c - 1) / c);
        const long long cost = ((blocks + slots - 1) / slots) * (c + 4);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = c;
        }
    }
    return best;
}

// tensor map of an array of `per`-word slots (8-byte words: 2 for FP32 slots, 1 for FP16
// ones), box bk slots x bj rows x 1 plane; parts of a box outside the array read as zero
bool cell_map(EncodeTiled enc, CUtensorMap* map, const void* base, const Geom& g, int per, int bk, int bj) {
    const cuuint64_t dims[3] = {(cuuint64_t)g.sz * per, (cuuint64_t)g.sy, (cuuint64_t)g.sx};
    const cuuint64_t strides[2] = {(cuuint64_t)g.sz * per * 8, (cuuint64_t)g.sy * g.sz * per * 8};
    const cuuint32_t box[3] = {(cuuint32_t)(per * bk), (cuuint32_t)bj, 1}, es[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TK>
int launch_cell(cudaStream_t st, int dev, EncodeTiled enc, const Geom& g, float vol, const float4* r, const float4* xin, float4* xout,
                const __half* P16, const float* psc, int flag, const float4* xc, const Geom* gc, bool pair, bool* done) {
    using C = CellTile<TK>;
    using CP = CellTile<TK, true>;
    using CX = CellTile<TK, true, true>;
    static bool set[MAX_DEVICES] = {};
    if (!set[dev]) {
        STG_CK(cudaFuncSetAttribute(k_sweep_cell<TK, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(false)));
        STG_CK(cudaFuncSetAttribute(k_sweep_cell<TK, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(true)));
        STG_CK(cudaFuncSetAttribute(k_sweep_cell<TK, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(true)));
        STG_CK(cudaFuncSetAttribute(k_sweep_cell<TK, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, CP::smem(false)));
        STG_CK(cudaFuncSetAttribute(k_sweep_cell<TK, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, CX::smem(true)));
        set[dev] = true;
    }
    CUtensorMap mx{}, mr{}, mp{};
    const int rw = pair ? CP::RW : C::RW, rr = pair ? CP::RR : C::RR;
    *done = cell_map(enc, &mr, r, g, 2, rw, rr) && cell_map(enc, &mp, P16, g, 1, rw, rr) &&
            (!xin || cell_map(enc, &mx, xin, g, 2, pair ? CX::XW : C::XW, pair ? CX::XR : C::XR));
    if (!*done) return STG_OK;
    const int tj = pair ? CP::TJ : C::TJ, chunk = cell_chunk(dev, g.n, TK, tj, pair ? (xin ? 2 : 3) : xin ? 4 : 8);
    const dim3 grid((g.n + TK - 1) / TK, (g.n + tj - 1) / tj, (g.n + chunk - 1) / chunk);
    int* err = g_sweep_err[dev];
    if (pair && !xin)
        k_sweep_cell<TK, 3><<<grid, CP::THREADS, CP::smem(false), st>>>(mr, mr, mp, g, vol, xout, psc, flag, chunk, err, nullptr, 0, 0);
    else if (pair)
        k_sweep_cell<TK, 4><<<grid, CX::THREADS, CX::smem(true), st>>>(mx, mr, mp, g, vol, xout, psc, flag, chunk, err, xc,
                                                                        xc ? gc->sy * gc->sz : 0, xc ? gc->sz : 0);
    else if (!xin)
        k_sweep_cell<TK, 0><<<grid, C::NT, C::smem(false), st>>>(mr, mr, mp, g, vol, xout, psc, flag, chunk, err, nullptr, 0, 0);
    else if (!xc)
        k_sweep_cell<TK, 1><<<grid, C::NT, C::smem(true), st>>>(mx, mr, mp, g, vol, xout, psc, flag, chunk, err, nullptr, 0, 0);
    else
        k_sweep_cell<TK, 2><<<grid, C::NT, C::smem(true), st>>>(mx, mr, mp, g, vol, xout, psc, flag, chunk, err, xc, gc->sy * gc->sz, gc->sz);
    STG_LAUNCH_CK();
    return STG_OK;
}

// the flag a TMA sweep sets when its wait gave up, per device
int sweep_err_init(cudaStream_t st, int dev) {
    if (g_sweep_err[dev]) return STG_OK;
    STG_CK(cudaMalloc((void**)&g_sweep_err[dev], sizeof(int)));
    STG_CK(cudaMemsetAsync(g_sweep_err[dev], 0, sizeof(int), st));
    return STG_OK;
}

}  // namespace

bool sweep_tma_available() { return encoder() != nullptr; }

int sweep_status(cudaStream_t st, int* timed_out) {
    *timed_out = 0;
    const int dev = device_slot();
    if (dev < 0 || !g_sweep_err[dev]) return STG_OK;
    STG_CK(cudaMemcpyAsync(timed_out, g_sweep_err[dev], sizeof(int), cudaMemcpyDeviceToHost, st));
    STG_CK(cudaStreamSynchronize(st));
    return STG_OK;
}

int sweep32(cudaStream_t st, const Geom& g, float vol, const float4* r, const float4* xin, float4* xout, const uint8_t* m,
            const float4* P, int flag, bool lap, const __half* P16, const float* p16_scale, const float4* xc, const Geom* gc, bool pair) {
    const int dev = device_slot();
    if (dev < 0) {
        set_error("sweep32: device ordinal beyond %d", MAX_DEVICES - 1);
        return STG_E_UNSUPPORTED;
    }
    const int smem = (int)sizeof(Smem), smem_l = (int)sizeof(SmemL);
    if (!g_attr_set[dev]) {
        STG_CK(cudaFuncSetAttribute(k_sweep<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        STG_CK(cudaFuncSetAttribute(k_sweep<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        STG_CK(cudaFuncSetAttribute(k_sweep_lap<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_l));
        STG_CK(cudaFuncSetAttribute(k_sweep_lap<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_l));
        g_attr_set[dev] = true;
    }
    if (lap && P16 && p16_scale && encoder()) {
        // the solver's own sweeps; a narrower tile (with more rows) where a row has fewer slots: levels
        // of 8 and 16 cells that no cluster launch takes (linear prolongation, smallcycle.cu small_cycle_ok)
        STG_TRY(sweep_err_init(st, dev));
        bool done = false;
        const auto go = g.n > 16 ? launch_cell<32> : launch_cell<16>;
        STG_TRY(go(st, dev, encoder(), g, vol, r, xin, xout, P16, p16_scale, flag, xc, gc, pair, &done));
        if (done) return STG_OK;
    }
    if (xc || pair) {
        set_error("sweep32: the fused prolongation and the pair of sweeps need the TMA sweep by cells");
        return STG_E_UNSUPPORTED;
    }
    // planes per block: long marches on big grids (prologue amortised), short ones on the
    // coarse levels, where the sequential march, not bandwidth, sets the time
    const int chunk = g.n >= 192 ? 32 : g.n >= 96 ? 8 : g.n >= 48 ? 4 : g.n >= 24 ? 2 : 1;
    dim3 grid((g.n + SK) / SK, (g.n + SJ) / SJ, (g.n + chunk) / chunk), block(SK, SJ);
    // the TMA sweep's tiles and chunks cover [0, n) and take the high-side slots (k, j or
    // i = n) with the last ones
    const dim3 grid_t((g.n + SK - 1) / SK, (g.n + SJ - 1) / SJ, (g.n + chunk - 1) / chunk);
    if (lap && encoder()) {
        const int smem_t = (int)sizeof(SmemT);
        if (!g_tattr_set[dev]) {
            STG_CK(cudaFuncSetAttribute(k_sweep_tma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_t));
            STG_CK(cudaFuncSetAttribute(k_sweep_tma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_t));
            STG_TRY(sweep_err_init(st, dev));
            g_tattr_set[dev] = true;
        }
        CUtensorMap mx{}, mr{}, mp{};
        const EncodeTiled enc = encoder();
        const bool ok = (!xin || slot_map(enc, &mx, xin, g, XK, XJ)) && slot_map(enc, &mr, r, g, RK, RJ) && slot_map(enc, &mp, P, g, RK, RJ);
        if (ok) {
            int* err = g_sweep_err[dev];
            if (xin)
                k_sweep_tma<true><<<grid_t, block, smem_t, st>>>(mx, mr, mp, g, vol, xout, m, flag, chunk, err);
            else
                k_sweep_tma<false><<<grid_t, block, smem_t, st>>>(mr, mr, mp, g, vol, xout, m, flag, chunk, err);
            STG_LAUNCH_CK();
            return STG_OK;
        }
    }
    if (xin && lap)
        k_sweep_lap<true><<<grid, block, smem_l, st>>>(g, vol, r, xin, xout, m, P, flag, chunk);
    else if (xin)
        k_sweep<true, false><<<grid, block, smem, st>>>(g, vol, r, xin, xout, m, P, flag, chunk);
    else if (lap)
        k_sweep_lap<false><<<grid, block, smem_l, st>>>(g, vol, r, xin, xout, m, P, flag, chunk);
    else
        k_sweep<false, false><<<grid, block, smem, st>>>(g, vol, r, xin, xout, m, P, flag, chunk);
    STG_LAUNCH_CK();
    return STG_OK;
}

}  // namespace stg
