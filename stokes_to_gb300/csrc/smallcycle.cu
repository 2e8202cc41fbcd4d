// The V-cycle of the smallest levels (at most 16 cells an axis, down to the 4^3 coarsest solve)
// in one launch of one thread-block cluster, for the solver's own Laplacian form.
//
// These levels have at most 4913 slots: as kernels of their own, the ten sweeps and transfers
// and the coarsest solve cost 2 to 5 us each, nearly all of it launch and drain. Here barriers
// separate the passes. Same arithmetic as the kernels it stands for: sweep.cu k_sweep_cell,
// kernels.cu k_restrict_fine32 and k_prolong_add32, dense.cu k_gemv.
//
// Two kernels: k_cycle16 for one sweep a colour from 16^3 down, in shared memory; k_small_cycle for
// the other sweep counts and for 8^3 grids, through L2, bound by latency: 25.1 us for the eleven
// passes from 16^3, 2.3 us each (a round of L2 loads, the stores' way back and the barrier).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstddef>
#include <utility>

#include "cell.cuh"
#include "ctx.h"
#include "rowdot.cuh"
#include "stencil.cuh"

namespace stg {

namespace {

constexpr int CT = 256;   // threads of a block: 16 blocks hold the 4096 slots of a 16^3 level
constexpr int ND = 304;     // unknowns of the 4^3 coarsest level
constexpr int MAXS = 4;   // levels in the cluster part

struct SLevel {
    int n, ln, di, dj;  // cells per axis (4 2^l) and their log2, slot strides along i and j (k: 1)
    float vol;
    const float4* r;
    float4 *rw, *xa, *xb;  // rw: r as the restriction writes it
    const uint2* P16;
    const float* psc;
    const float4* P32;
    const uint8_t* m;
    __device__ int slot(int i, int j, int k) const { return (i + 1) * di + (j + 1) * dj + k + 1; }
};
struct SCycle {
    SLevel lv[MAXS];
    int top, per;  // per: sweeps a colour
    int mixed;     // coarse corrections rounded to BF16
    int ld;
    const double* inv;
    const float2* inv2;  // the same as sums of two floats, row-major ND x ND
    const int *slot_of, *comp_of;
};

// vectors that change during the launch are read through L2
__device__ __forceinline__ float4 ld4(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ float ld1(const float4* p, int c) { return __ldcg(reinterpret_cast<const float*>(p) + c); }

// A solved cell (i, j, k) into the slots of xo, and what no red cell owns: the black pressure pb of
// its pair, and the black cell's faces on the domain boundary (fixed: 0).
__device__ __forceinline__ void store_cell(const SLevel& L, float4* xo, int n, int i, int j, int k, int q, int s, float p,
                                           const float lo[3], const float hi[3], float pb) {
    float* o = reinterpret_cast<float*>(xo);
    const int sb = q ? s - 1 : s + 1, kb = q ? k - 1 : k + 1;
    xo[s] = make_float4(p, lo[0], lo[1], lo[2]);
    o[4ll * (s + L.di) + 1] = hi[0];
    o[4ll * (s + L.dj) + 2] = hi[1];
    o[4ll * (s + 1) + 3] = hi[2];
    o[4ll * sb] = pb;
    if (i == 0) o[4ll * sb + 1] = 0.f;
    if (j == 0) o[4ll * sb + 2] = 0.f;
    if (kb == 0) o[4ll * sb + 3] = 0.f;
    if (i == n - 1) o[4ll * (sb + L.di) + 1] = 0.f;
    if (j == n - 1) o[4ll * (sb + L.dj) + 2] = 0.f;
    if (kb == n - 1) o[4ll * (sb + 1) + 3] = 0.f;
}

// One colour of the smoother, a thread per pair of slots along k (one red, one black cell):
// the red cell's seven unknowns are solved, the black pressure copied. HX false: x = 0. PRO: x
// is first corrected by the parents' values of xc on C.
template <bool HX, bool PRO>
__device__ __forceinline__ void small_sweep(const SLevel& L, int flag, const float4* x, const SLevel& C, const float4* xc, bool mixed,
                                            float4* xo, int t0, int step) {
    const int n = L.n, ln = L.ln;
    const float vol = L.vol, v6 = 6.f * vol, psc = __ldg(L.psc);
    for (int t = t0; t < 1 << (3 * ln - 1); t += step) {
        const int kk = t & ((n >> 1) - 1), j = (t >> (ln - 1)) & (n - 1), i = t >> (2 * ln - 1);
        const int q = (i + j + flag) & 1, k = 2 * kk + q;
        const int s = L.slot(i, j, k);
        auto coarse = [&](int a, int b, int c) {
            float4 v = ld4(xc + C.slot((i + a) >> 1, (j + b) >> 1, (k + c) >> 1));
            if (mixed) {
                v.x = __bfloat162float(__float2bfloat16_rn(v.x));
                v.y = __bfloat162float(__float2bfloat16_rn(v.y));
                v.z = __bfloat162float(__float2bfloat16_rn(v.z));
                v.w = __bfloat162float(__float2bfloat16_rn(v.w));
            }
            return v;
        };
        auto X = [&](int a, int b, int c) {
            float4 v = ld4(x + s + a * L.di + b * L.dj + c);
            if (PRO) {
                const float4 e = coarse(a, b, c);
                v.x += e.x;
                v.y += e.y;
                v.z += e.z;
                v.w += e.w;
            }
            return v;
        };
        const __half* ph = reinterpret_cast<const __half*>(L.P16);
        const uint2 po = __ldg(L.P16 + s);
        const float2 pa = __half22float2(*reinterpret_cast<const __half2*>(&po.x)),
                     pz = __half22float2(*reinterpret_cast<const __half2*>(&po.y));
        const float raw[7] = {pa.x * psc, pa.y * psc, pz.x * psc, pz.y * psc, __half2float(__ldg(ph + 4ll * (s + L.di) + 1)) * psc,
                              __half2float(__ldg(ph + 4ll * (s + L.dj) + 2)) * psc, __half2float(__ldg(ph + 4ll * (s + 1) + 3)) * psc};
        const float4 r0 = ld4(L.r + s);
        float res[7] = {r0.x, r0.y, r0.z, r0.w, ld1(L.r + s + L.di, 1), ld1(L.r + s + L.dj, 2), ld1(L.r + s + 1, 3)};
        float p0 = 0.f, pb = 0.f, lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
        if (HX) {
            const float4 c = X(0, 0, 0), xm = X(-1, 0, 0), xp = X(1, 0, 0), ym = X(0, -1, 0), yp = X(0, 1, 0), zm = X(0, 0, -1),
                         zp = X(0, 0, 1), xy = X(1, 1, 0), xz = X(1, 0, 1), yz = X(0, 1, 1);
            p0 = c.x;
            pb = q ? zm.x : zp.x;
            lo[0] = c.y;
            lo[1] = c.z;
            lo[2] = c.w;
            hi[0] = xp.y;
            hi[1] = yp.z;
            hi[2] = zp.w;
            const float lap_lo[3] = {6.f * c.y - (xm.y + xp.y) - (ym.y + yp.y) - (zm.y + zp.y),
                                     6.f * c.z - (xm.z + xp.z) - (ym.z + yp.z) - (zm.z + zp.z),
                                     6.f * c.w - (xm.w + xp.w) - (ym.w + yp.w) - (zm.w + zp.w)};
            const float lap_hi[3] = {6.f * xp.y - (c.y + X(2, 0, 0).y) - (X(1, -1, 0).y + xy.y) - (X(1, 0, -1).y + xz.y),
                                     6.f * yp.z - (X(-1, 1, 0).z + xy.z) - (c.z + X(0, 2, 0).z) - (X(0, 1, -1).z + yz.z),
                                     6.f * zp.w - (X(-1, 0, 1).w + xz.w) - (X(0, -1, 1).w + yz.w) - (c.w + X(0, 0, 2).w)};
            const float p_lo[3] = {xm.x, ym.x, zm.x}, p_hi[3] = {xp.x, yp.x, zp.x};
            cell_residual(vol, raw, p0, lap_lo, lap_hi, p_lo, p_hi, lo, hi, res);
        }
        const float dp = cell_solve(vol, v6, raw, res, lo, hi);
        store_cell(L, xo, n, i, j, k, q, s, p0 + dp, lo, hi, pb);
    }
}

// C.rw = the 8-child sums of r - A x, masked: a lane per fine slot, the children of a coarse
// slot in eight neighbouring lanes
__device__ __forceinline__ void small_restrict(const SLevel& L, const float4* x, const SLevel& C, int t0, int step) {
    const int n = L.n, nc = C.n, lc = C.ln;
    for (int t = t0; t < n * n * n; t += step) {  // n^3 and the step are multiples of 32
        const int ch = t & 7, c = t >> 3;
        const int K = c & (nc - 1), J = (c >> lc) & (nc - 1), I = c >> (2 * lc);
        const int s = L.slot(2 * I + (ch >> 2), 2 * J + ((ch >> 1) & 1), 2 * K + (ch & 1));
        auto q4 = [&](int o) {
            const float4 v = ld4(x + s + o);
            return Q4<float>{v.x, v.y, v.z, v.w};
        };
        const float4 r = ld4(L.r + s), pv = __ldg(L.P32 + s);
        float o[4];
        lap_core<float>(q4(0), q4(-L.di), q4(L.di), q4(-L.dj), q4(L.dj), q4(-1), q4(1), Q4<float>{pv.x, pv.y, pv.z, pv.w}, L.vol, o);
        o[0] = r.x - o[0];
        o[1] = r.y - o[1];
        o[2] = r.z - o[2];
        o[3] = r.w - o[3];
        mask4<float>(__ldg(L.m + s), o);
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int d = 4; d >= 1; d >>= 1) o[q] += __shfl_xor_sync(0xffffffffu, o[q], d);
        if (ch == 0) {
            const int sc = C.slot(I, J, K);
            mask4<float>(__ldg(C.m + sc), o);
            C.rw[sc] = make_float4(o[0], o[1], o[2], o[3]);
        }
    }
}

__global__ void __launch_bounds__(CT) k_small_cycle(const __grid_constant__ SCycle S) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int t0 = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31), step = gridDim.x * CT;
    // this warp's rows of the coarsest inverse and this thread's entries of its right-hand side
    using Rows = RowDots<ND, 2>;
    const int lane = threadIdx.x & 31, half = t0 >> 4;
    Rows rows;
    int at[(ND + CT - 1) / CT];  // offset of entry threadIdx.x + q CT in the coarsest vector
    for (int i = S.top; i >= 1; i--) {
        const SLevel &L = S.lv[i], &C = S.lv[i - 1];
        float4 *x = L.xa, *y = L.xb;
        small_sweep<false, false>(L, 0, nullptr, C, nullptr, false, x, t0, step);
        cl.sync();
        for (int q = 1; q < 2 * S.per; q++) {
            small_sweep<true, false>(L, q / S.per, x, C, nullptr, false, y, t0, step);
            cl.sync();
            float4* z = x;
            x = y;
            y = z;
        }
        small_restrict(L, x, C, t0, step);
        if (i == 1) {
            rows.load(S.inv, S.ld, half, lane);
#pragma unroll
            for (int q = 0; q < (ND + CT - 1) / CT; q++) {
                const int c = threadIdx.x + q * CT;
                at[q] = c < ND ? 4 * __ldg(S.slot_of + c) + __ldg(S.comp_of + c) : 0;
            }
        }
        cl.sync();
    }
    {  // coarsest solve (dense.cu k_gemv)
        __shared__ double rd[ND];
        const SLevel& L = S.lv[0];
#pragma unroll
        for (int q = 0; q < (ND + CT - 1) / CT; q++)
            if (threadIdx.x + q * CT < ND) rd[threadIdx.x + q * CT] = (double)__ldcg(reinterpret_cast<const float*>(L.r) + at[q]);
        __syncthreads();
        if (t0 >> 5 < (Rows::HALVES + 1) / 2) {
            double s[2];
            rows.dot(rd, lane, s);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int row = half + k * Rows::HALVES;
                if ((lane & 15) == k && half < Rows::HALVES && row < ND)
                    reinterpret_cast<float*>(L.xa)[4ll * __ldg(S.slot_of + row) + __ldg(S.comp_of + row)] = (float)s[k];
            }
        }
        cl.sync();
    }
    for (int i = 1; i <= S.top; i++) {
        const SLevel &L = S.lv[i], &C = S.lv[i - 1];
        const float4* xc = i == 1 ? C.xa : C.xb;
        // the pre-smoother's 2 per sweeps (an even number) ended in xb
        float4 *x = L.xb, *y = L.xa;
        for (int q = 0; q < 2 * S.per; q++) {
            const int flag = 1 - q / S.per;
            if (q == 0)
                small_sweep<true, true>(L, flag, x, C, xc, S.mixed != 0, y, t0, step);
            else
                small_sweep<true, false>(L, flag, x, C, nullptr, false, y, t0, step);
            if (q + 1 < 2 * S.per || i < S.top) cl.sync();
            float4* z = x;
            x = y;
            y = z;
        }
    }
}


// ---------------------------------------------------------------- 16^3, 8^3 and 4^3 in shared memory
// The same cycle with one sweep a colour from 16^3 down, without a trip through L2 between its
// passes: block b has plane b of the 16^3 level, with the red cells of the planes beside it, which
// it forms itself, and every block has all of the 8^3 level and a sixteenth of the coarsest
// inverse's rows. So the two sweeps before and after the coarse correction meet at block barriers,
// and three exchanges cross the cluster: the pre-smoothed planes, each to the seven blocks that
// read it, the planes' shares of the restricted residual and the coarsest solution, to all.
//
// x lies in slot order where its next reader has the same colour, else as cells (cell.cuh
// neighbour_residual). The coarsest product runs on the FP32 pipe, the inverse's entries as
// sums of two floats (set-up, split_inverse), products and sums in double-float arithmetic: the
// FP64 pipe, two lanes a clock and SM, would take 2 us more.
// (Rounded to FP32 the rows' products have the error of FP64 ones, 5.7e-8 at most and 2.1e-8 on
// average, on matrices of entries over nine decades too: the rounding to FP32 is all of it.)
//
// Bound: latency, a chain of fifteen block-wide passes of 0.3 to 0.7 us and the exchanges, 1 to
// 1.5 us each. 16.0 us a cycle; k_small_cycle takes 25.1. With the planes that post-sweeps read
// formed by every block itself instead of sent (nine red and seven black planes): 18.5 us, bound by
// the uncoalesced loads; with the 8^3 level in one block that sends its results: 21.9 us.
constexpr int PT = 1024;                        // threads of a block
constexpr int XW16 = 20, XP16 = 19 * XW16;      // x of a 16^3 plane: slots -1 .. 17
constexpr int FW16 = 12, FH16 = 18 * FW16;      // its cells of a colour: rows and pairs -1 .. 16 and 8
constexpr int XW8 = 12, XP8 = 11 * XW8;         // the 8^3 level likewise
constexpr int FW8 = 12, FH8 = 10 * FW8;
constexpr int RW8 = 9, RP8 = 9 * RW8;           // its right-hand side and penalties: slots 0 .. 8
constexpr int PW8 = 10, PP8 = 9 * PW8;
constexpr int SLOTS4 = 7 * 56;                  // slots of the 4^3 level as in memory
constexpr int DOT_ROWS = ND / 16;               // rows of the coarsest inverse of a block
struct CycleShared {
    float4 x[6 * XP16];        // planes b - 2 .. b + 3
    float4 f[3 * 2 * FH16];    // planes b - 1 .. b + 1
    float4 x8[11 * XP8];
    float4 r8[9 * RP8];
    float4 z8[512];            // the 8^3 correction
    float4 s4[SLOTS4];         // the 4^3 right-hand side (x .. s4 start as 0)
    union {
        float4 f8[10 * 2 * FH8];  // (cleared once c is read)
        struct {               // the pre-smoothed planes b - 3 .. b + 3: black cells, their pairs' red pressures
            float4 lo[7][128], hi[7][128];
            float p[7][128];
        } c;
    };
    float4 e4[SLOTS4];         // and solution
    float4 part[16][64];       // each plane's share of the restricted residual
    float4 r[4 * XP16];        // r and FP16 penalties, planes b - 1 .. b + 2
    uint2 p[4 * XP16];
    float4 pen[XP16];          // FP32 penalties of plane b
    float4 pen8[512];          // and of the 8^3 slots
    uint2 p8[9 * PP8];         // their FP16 copy
    float rd[ND];
    int at[ND];                // entry of the coarsest vector in s4 and e4
    uint8_t m8[512], m4[64], m[XP16];
};
static_assert(ND % 16 == 0 && DOT_ROWS <= 2 * 16 && ND <= 512, "two rows a warp of half a block");
static_assert(sizeof(CycleShared) <= 227 * 1024, "the shared memory of an SM");

// a cell's right-hand side from slots in shared memory (pitches RW, RP)
template <int RW, int RP>
__device__ __forceinline__ void cell_rhs(const float4* R, float res[7]) {
    const float4 r0 = R[0];
    res[0] = r0.x;
    res[1] = r0.y;
    res[2] = r0.z;
    res[3] = r0.w;
    res[4] = R[RP].y;
    res[5] = R[RW].z;
    res[6] = R[1].w;
}
// a solved cell into the slots of x (pitches XW, XP; up: the next plane is there)
template <int XW, int XP>
__device__ __forceinline__ void store_slots(float4* X, float p, const float lo[3], const float hi[3], int q, float pb, bool up) {
    X[0] = make_float4(p, lo[0], lo[1], lo[2]);
    if (up) X[XP].y = hi[0];
    X[XW].z = hi[1];
    X[1].w = hi[2];
    X[q ? -1 : 1].x = pb;
}

__global__ void __launch_bounds__(PT, 1) k_cycle16(const __grid_constant__ SCycle S) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char cycle_smem[];
    CycleShared& M = *reinterpret_cast<CycleShared*>(cycle_smem);
    const SLevel &L = S.lv[2], &L8 = S.lv[1], &L4 = S.lv[0];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float vol = L.vol, v6 = 6.f * vol, vol8 = L8.vol, v68 = 6.f * vol8;
    auto started = cl.barrier_arrive();
    auto zero = [&](void* from, const void* to, int first) {  // by the threads from `first` on
        const float4* e = static_cast<const float4*>(to);
        if (tid >= first)
            for (float4* z = static_cast<float4*>(from) + tid - first; z < e; z += PT - first) *z = make_float4(0.f, 0.f, 0.f, 0.f);
    };

    {  // what the passes read of memory
        const int s0 = L.slot(b - 1, -1, -1);
        for (int t = tid; t < 4 * XP16; t += PT) copy16(&M.r[t], L.r + s0 + t);
        for (int t = tid; t < 2 * XP16; t += PT) copy16(&M.p[2 * t], L.P16 + s0 + 2 * t);
    }
    if (tid >= PT - XP16) copy16(&M.pen[tid - (PT - XP16)], L.P32 + L.slot(b, -1, -1) + tid - (PT - XP16));
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (tid < 512) copy16(&M.pen8[tid], L8.P32 + L8.slot(tid >> 6, (tid >> 3) & 7, tid & 7));
    if (tid < 729) copy8(&M.p8[(tid / 81) * PP8 + (tid / 9 % 9) * PW8 + tid % 9], L8.P16 + L8.slot(tid / 81, tid / 9 % 9, tid % 9));
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const uint8_t m = tid < XP16 ? __ldg(L.m + L.slot(b, -1, -1) + tid) : 0;
    const uint8_t m8 = tid < 512 ? __ldg(L8.m + L8.slot(tid >> 6, (tid >> 3) & 7, tid & 7)) : 0;
    const uint8_t m4 = tid < 64 ? __ldg(L4.m + L4.slot(tid >> 4, (tid >> 2) & 3, tid & 3)) : 0;
    const int at = tid < ND ? 4 * __ldg(S.slot_of + tid) + __ldg(S.comp_of + tid) : 0;
    const float psc = __ldg(L.psc), psc8 = __ldg(L8.psc);
    zero(M.x, M.x8, 0);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();

    // a thread's cell of the 16^3 level: row j, pair kk of plane b - 1 + d
    const int d = tid >> 7, i = b - 1 + d, j = (tid >> 3) & 15, kk = tid & 7, q0 = (i + j) & 1;
    const bool near = d < 3 && i >= 0 && i < 16;
    const float4* R = M.r + d * XP16 + (j + 1) * XW16 + 2 * kk + 1;
    const uint2* Q = M.p + d * XP16 + (j + 1) * XW16 + 2 * kk + 1;
    float4* F = M.f + d * 2 * FH16 + (j + 1) * FW16 + kk + 1;
    if (near) {  // red, from x = 0
        float raw[7], res[7], lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
        cell_penalty<XW16>(Q + q0, Q + q0 + XP16, psc, raw);
        cell_rhs<XW16, XP16>(R + q0, res);
        const float dp = cell_solve(vol, v6, raw, res, lo, hi);
        F[0] = make_float4(dp, lo[0], lo[1], lo[2]);
        F[FH16] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
    zero(M.x8, M.f8, 3 * 128);
    if (tid < 512) M.m8[tid] = m8;
    if (tid < 64) M.m4[tid] = m4;
    if (tid < ND) M.at[tid] = at;
    if (tid < XP16) M.m[tid] = m;
    __syncthreads();
    if (d == 1) {  // black
        const int q = 1 - q0;
        float raw[7], res[7], lo[3], hi[3], pb;
        cell_penalty<XW16>(Q + q, Q + q + XP16, psc, raw);
        cell_rhs<XW16, XP16>(R + q, res);
        neighbour_residual<FW16, FH16>(F - 2 * FH16, F, F + 2 * FH16, q, vol, raw, 0.f, lo, hi, res, pb);
        const float dp = cell_solve(vol, v6, raw, res, lo, hi);
        M.c.lo[3][tid & 127] = make_float4(dp, lo[0], lo[1], lo[2]);
        M.c.hi[3][tid & 127] = make_float4(hi[0], hi[1], hi[2], 0.f);
        M.c.p[3][tid & 127] = pb;
    }
    __syncthreads();
    cl.barrier_wait(std::move(started));  // every block runs before its shared memory is written
    {
        const int to = b - 3 + d, c = tid & 127;
        if (d < 7 && to >= 0 && to < 16 && to != b) {
            auto& C = cl.map_shared_rank(&M, to)->c;
            C.lo[6 - d][c] = M.c.lo[3][c];
            C.hi[6 - d][c] = M.c.hi[3][c];
            C.p[6 - d][c] = M.c.p[3][c];
        }
    }
    cl.sync();
    if (d < 7) {  // into the slots of x; of plane b - 3 only u on the next plane
        const int p = b - 3 + d, q = (p + j + 1) & 1, c = tid & 127;
        if (p >= 0 && p < 16) {
            const float4 l = M.c.lo[d][c], h = M.c.hi[d][c];
            const float lo[3] = {l.y, l.z, l.w}, hi[3] = {h.x, h.y, h.z};
            float4* X = M.x + (d - 1) * XP16 + (j + 1) * XW16 + 2 * kk + q + 1;
            if (d == 0)
                X[XP16].y = hi[0];
            else
                store_slots<XW16, XP16>(X, l.x, lo, hi, q, M.c.p[d][c], d < 6);
        }
    }
    __syncthreads();
    // this plane's share of the restricted residual: a lane per slot, the four children of a
    // coarse slot in neighbouring lanes, each of which sends the sum to four blocks
    if (tid < 256) {
        const int c = tid >> 2, s = (2 * (c >> 3) + ((tid >> 1) & 1) + 1) * XW16 + 2 * (c & 7) + (tid & 1) + 1;
        const float4* X = M.x + 2 * XP16 + s;
        const float4 r = M.r[XP16 + s], pv = M.pen[s];
        auto q4 = [&](int o) { return Q4<float>{X[o].x, X[o].y, X[o].z, X[o].w}; };
        float o[4];
        lap_core<float>(q4(0), q4(-XP16), q4(XP16), q4(-XW16), q4(XW16), q4(-1), q4(1), Q4<float>{pv.x, pv.y, pv.z, pv.w}, vol, o);
        o[0] = r.x - o[0];
        o[1] = r.y - o[1];
        o[2] = r.z - o[2];
        o[3] = r.w - o[3];
        mask4<float>(M.m[s], o);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            o[q] += __shfl_xor_sync(0xffffffffu, o[q], 2);
            o[q] += __shfl_xor_sync(0xffffffffu, o[q], 1);
        }
#pragma unroll
        for (int to = 0; to < 16; to += 4) cl.map_shared_rank(&M.part[0][0], to + (tid & 3))[b * 64 + c] = make_float4(o[0], o[1], o[2], o[3]);
    }
    zero(M.f8, M.e4, 256);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    cl.sync();
    // a thread's cell of the 8^3 level: a red one for the first 256, a black one for the next
    const int kk8 = tid & 3, j8 = (tid >> 2) & 7, i8 = (tid >> 5) & 7, q8 = (i8 + j8 + (tid >> 8)) & 1;
    const bool red8 = tid < 256, black8 = tid >= 256 && tid < 512;
    const float4* R8 = M.r8 + i8 * RP8 + j8 * RW8 + 2 * kk8 + q8;
    const uint2* Q8 = M.p8 + i8 * PP8 + j8 * PW8 + 2 * kk8 + q8;
    float4* F8 = M.f8 + (i8 + 1) * 2 * FH8 + (j8 + 1) * FW8 + kk8 + 1;
    float4* X8 = M.x8 + (i8 + 1) * XP8 + (j8 + 1) * XW8 + 2 * kk8 + q8 + 1;
    // the first half of the warps works on the 8^3 level, the other has the block's rows of the
    // coarsest inverse on their way meanwhile
    float2 a[2][(ND + 31) / 32];
    const int dot = warp - 16;  // rows b + 16 dot and, of the first three, b + 16 (dot + 16)
    if (dot >= 0) {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int q = 0; q < (ND + 31) / 32; q++) {
                const int c = lane + 32 * q, r = dot + 16 * h;
                a[h][q] = r < DOT_ROWS && c < ND ? __ldg(S.inv2 + (long long)(b + 16 * r) * ND + c) : make_float2(0.f, 0.f);
            }
    } else {
        auto half_sync = [] { asm volatile("bar.sync 1, 512;\n" ::: "memory"); };
        {
            const int k8 = tid & 7, j8 = (tid >> 3) & 7, i8 = tid >> 6;
            const float4 u = M.part[2 * i8][j8 * 8 + k8], w = M.part[2 * i8 + 1][j8 * 8 + k8];
            float o[4] = {u.x + w.x, u.y + w.y, u.z + w.z, u.w + w.w};
            mask4<float>(M.m8[tid], o);
            M.r8[i8 * RP8 + j8 * RW8 + k8] = make_float4(o[0], o[1], o[2], o[3]);
        }
        half_sync();
        if (red8) {
            float raw[7], res[7], lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
            cell_penalty<PW8>(Q8, Q8 + PP8, psc8, raw);
            cell_rhs<RW8, RP8>(R8, res);
            const float dp = cell_solve(vol8, v68, raw, res, lo, hi);
            F8[0] = make_float4(dp, lo[0], lo[1], lo[2]);
            F8[FH8] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
        half_sync();
        if (black8) {
            float raw[7], res[7], lo[3], hi[3], pb;
            cell_penalty<PW8>(Q8, Q8 + PP8, psc8, raw);
            cell_rhs<RW8, RP8>(R8, res);
            neighbour_residual<FW8, FH8>(F8 - 2 * FH8, F8, F8 + 2 * FH8, q8, vol8, raw, 0.f, lo, hi, res, pb);
            const float dp = cell_solve(vol8, v68, raw, res, lo, hi);
            store_slots<XW8, XP8>(X8, dp, lo, hi, q8, pb, true);
        }
        half_sync();
        {  // restriction: the eight children of a coarse slot in neighbouring lanes
            const int c = tid >> 3, K = c & 3, J = (c >> 2) & 3, I = c >> 4;
            const int fi = 2 * I + ((tid >> 2) & 1), fj = 2 * J + ((tid >> 1) & 1), fk = 2 * K + (tid & 1), e = (fi * 8 + fj) * 8 + fk;
            const float4* X = M.x8 + (fi + 1) * XP8 + (fj + 1) * XW8 + fk + 1;
            const float4 r = M.r8[fi * RP8 + fj * RW8 + fk], pv = M.pen8[e];
            auto q4 = [&](int o) { return Q4<float>{X[o].x, X[o].y, X[o].z, X[o].w}; };
            float o[4];
            lap_core<float>(q4(0), q4(-XP8), q4(XP8), q4(-XW8), q4(XW8), q4(-1), q4(1), Q4<float>{pv.x, pv.y, pv.z, pv.w}, vol8, o);
            o[0] = r.x - o[0];
            o[1] = r.y - o[1];
            o[2] = r.z - o[2];
            o[3] = r.w - o[3];
            mask4<float>(M.m8[e], o);
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int d = 4; d >= 1; d >>= 1) o[q] += __shfl_xor_sync(0xffffffffu, o[q], d);
            if ((tid & 7) == 0) {
                mask4<float>(M.m4[c], o);
                M.s4[L4.slot(I, J, K)] = make_float4(o[0], o[1], o[2], o[3]);
            }
        }
        half_sync();
        if (tid < ND) M.rd[tid] = reinterpret_cast<const float*>(M.s4)[M.at[tid]];
    }
    __syncthreads();
    if (dot >= 0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = dot + 16 * h;
            if (r >= DOT_ROWS) break;
            DfSum sum;
#pragma unroll
            for (int q = 0; q < (ND + 31) / 32; q++) {
                const int c = lane + 32 * q;
                if (c < ND) sum.fma(a[h][q], M.rd[c]);
            }
            const float v = sum.warp_total();
            if (lane < 16) reinterpret_cast<float*>(cl.map_shared_rank(&M.e4[0], lane))[M.at[b + 16 * r]] = v;
        }
    }
    cl.sync();
    auto add = [&](float4& x, float4 e) {  // a coarse correction, as the prolongation reads it
        if (S.mixed) {
            e.x = __bfloat162float(__float2bfloat16_rn(e.x));
            e.y = __bfloat162float(__float2bfloat16_rn(e.y));
            e.z = __bfloat162float(__float2bfloat16_rn(e.z));
            e.w = __bfloat162float(__float2bfloat16_rn(e.w));
        }
        x = make_float4(x.x + e.x, x.y + e.y, x.z + e.z, x.w + e.w);
    };
    if (tid < 512) {
        const int k = tid & 7, jj = (tid >> 3) & 7, i = tid >> 6;
        add(M.x8[(i + 1) * XP8 + (jj + 1) * XW8 + k + 1], M.e4[L4.slot(i >> 1, jj >> 1, k >> 1)]);
    }
    __syncthreads();
    if (black8) {
        float raw[7], res[7], lo[3], hi[3], p0;
        cell_penalty<PW8>(Q8, Q8 + PP8, psc8, raw);
        cell_rhs<RW8, RP8>(R8, res);
        slot_residual<XW8>(X8 - XP8, X8, X8 + XP8, X8 + 2 * XP8, vol8, raw, p0, lo, hi, res);
        const float dp = cell_solve(vol8, v68, raw, res, lo, hi);
        F8[0] = make_float4(p0 + dp, lo[0], lo[1], lo[2]);
        F8[FH8] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
    __syncthreads();
    if (red8) {
        float raw[7], res[7], lo[3], hi[3], pb;
        cell_penalty<PW8>(Q8, Q8 + PP8, psc8, raw);
        cell_rhs<RW8, RP8>(R8, res);
        const float p0 = X8[0].x;
        neighbour_residual<FW8, FH8>(F8 - 2 * FH8, F8, F8 + 2 * FH8, q8, vol8, raw, p0, lo, hi, res, pb);
        const float dp = cell_solve(vol8, v68, raw, res, lo, hi);
        float4* Z = M.z8 + (i8 * 8 + j8) * 8 + 2 * kk8 + q8;
        Z[0] = make_float4(p0 + dp, lo[0], lo[1], lo[2]);
        if (i8 < 7) Z[64].y = hi[0];
        if (j8 < 7) Z[8].z = hi[1];
        if (2 * kk8 + q8 < 7) Z[1].w = hi[2];
        Z[q8 ? -1 : 1].x = pb;
    }
    __syncthreads();
    for (int t = tid; t < 6 * 256; t += PT) {
        const int p = b - 2 + (t >> 8), jj = (t >> 4) & 15, k = t & 15;
        if (p >= 0 && p < 16) add(M.x[(t >> 8) * XP16 + (jj + 1) * XW16 + k + 1], M.z8[((p >> 1) * 8 + (jj >> 1)) * 8 + (k >> 1)]);
    }
    __syncthreads();
    if (near) {  // black
        const int q = 1 - q0;
        float raw[7], res[7], lo[3], hi[3], p0;
        cell_penalty<XW16>(Q + q, Q + q + XP16, psc, raw);
        cell_rhs<XW16, XP16>(R + q, res);
        const float4* X = M.x + (d + 1) * XP16 + (j + 1) * XW16 + 2 * kk + q + 1;
        slot_residual<XW16>(X - XP16, X, X + XP16, X + 2 * XP16, vol, raw, p0, lo, hi, res);
        const float dp = cell_solve(vol, v6, raw, res, lo, hi);
        F[0] = make_float4(p0 + dp, lo[0], lo[1], lo[2]);
        F[FH16] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
    __syncthreads();
    if (d == 1) {  // red
        float raw[7], res[7], lo[3], hi[3], pb;
        cell_penalty<XW16>(Q + q0, Q + q0 + XP16, psc, raw);
        cell_rhs<XW16, XP16>(R + q0, res);
        const int k = 2 * kk + q0;
        const float p0 = M.x[2 * XP16 + (j + 1) * XW16 + k + 1].x;
        neighbour_residual<FW16, FH16>(F - 2 * FH16, F, F + 2 * FH16, q0, vol, raw, p0, lo, hi, res, pb);
        const float dp = cell_solve(vol, v6, raw, res, lo, hi);
        store_cell(L, L.xb, 16, b, j, k, q0, L.slot(b, j, k), p0 + dp, lo, hi, pb);
    }
}

}  // namespace

// Blocks of the cluster (more than the portable eight: the coarsest solve's rows need the warps of
// all of them)
constexpr int BLOCKS = 16;
static_assert(RowDots<ND, 2>::HALVES <= BLOCKS * CT / 16, "a half-warp for every pair of rows");

static cudaLaunchConfig_t config(cudaStream_t st, bool in_smem, cudaLaunchAttribute (&at)[1]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(BLOCKS);
    cfg.blockDim = dim3(in_smem ? PT : CT);
    cfg.dynamicSmemBytes = in_smem ? sizeof(CycleShared) : 0;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = BLOCKS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// whether the device runs such a cluster
static bool cluster_ok(int dev, bool in_smem) {
    static int state[2][MAX_DEVICES] = {};  // 0 unknown, 1 no, 2 yes
    int& st = state[in_smem][dev];
    if (!st) {
        int can = 0;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = config(nullptr, in_smem, at);
        const auto kernel = in_smem ? k_cycle16 : k_small_cycle;
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&can, kernel, &cfg) == cudaSuccess && can > 0;
        cudaGetLastError();
        st = ok ? 2 : 1;
    }
    return st == 2;
}

// Levels of 8 and 16 cells an axis over the 4^3 coarsest one: at 32^3 a cluster's pass takes as
// long as a launch of the whole GPU, and larger coarsest inverses (12^3: 7344 unknowns) need the
// grid-wide product.
bool small_cycle_ok(const stg_t* h, int top) {
    const Level& L = h->lv[top];
    if (top < 1 || top >= MAXS || L.g.n > 16 || (L.g.n & (L.g.n - 1)) || h->dense.nd != ND || h->reference_cycle || !fast(h, L) || !L.P16 || h->opts.prolong == 1)
        return false;
    const int dev = device_slot();
    return dev >= 0 && cluster_ok(dev, false);
}

int small_cycle(stg_t* h, int top, const float4* rhs) {
    SCycle S{};
    S.top = top;
    S.per = sweeps_per_colour(h);
    S.mixed = h->opts.method == STG_METHOD_MIXED;
    S.ld = 2 * h->dense.nd;
    S.inv = h->dense.inv;
    S.slot_of = h->dense.slot_of;
    S.comp_of = h->dense.comp_of;
    for (int i = 0; i <= top; i++) {
        Level& L = h->lv[i];
        int ln = 0;
        while (1 << ln < L.g.n) ln++;
        S.lv[i] = SLevel{L.g.n, ln, L.g.di(), L.g.dj(), (float)L.vol, i == top && rhs ? rhs : L.r, L.r, L.xa, L.xb,
                         reinterpret_cast<const uint2*>(L.P16), h->d_pscale + i, L.P32, L.m};
        L.cur = i == 0 ? 0 : 1;
    }
    S.inv2 = h->dense.inv2;
    // k_cycle16 is for one sweep a colour from 16^3; the other sweep counts and tops pass through L2
    const bool in_smem = top == 2 && S.per == 1 && S.inv2 && cluster_ok(device_slot(), true);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(h->st, in_smem, at);
    STG_CK(cudaLaunchKernelEx(&cfg, in_smem ? k_cycle16 : k_small_cycle, S));
    count_launch();
    return STG_OK;
}

}  // namespace stg
