// The V-cycle of the smallest levels (at most 16 cells an axis, down to the 4^3 coarsest solve)
// in one launch of one thread-block cluster, for the solver's own Laplacian form.
//
// These levels have at most 4913 slots: as kernels of their own, the ten sweeps and transfers
// and the coarsest solve cost 2 to 5 us each, nearly all of it launch and drain. Here a pass is
// separated from the next by a cluster barrier, and every thread reads its neighbourhood
// straight from L2. Same arithmetic as the kernels it stands for: sweep.cu k_sweep_cell,
// kernels.cu k_restrict_fine32 and k_prolong_add32, dense.cu k_gemv.
//
// Bound: latency, about 1.5 us a pass (one round of L2 loads and the barrier).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

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
    const int *slot_of, *comp_of;
};

// vectors that change during the launch are read through L2
__device__ __forceinline__ float4 ld4(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ float ld1(const float4* p, int c) { return __ldcg(reinterpret_cast<const float*>(p) + c); }

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
        const int s = L.slot(i, j, k), sb = q ? s - 1 : s + 1;
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
            const float lu = 6.f * c.y - (xm.y + xp.y) - (ym.y + yp.y) - (zm.y + zp.y);
            const float hu = 6.f * xp.y - (c.y + X(2, 0, 0).y) - (X(1, -1, 0).y + xy.y) - (X(1, 0, -1).y + xz.y);
            const float lv = 6.f * c.z - (xm.z + xp.z) - (ym.z + yp.z) - (zm.z + zp.z);
            const float hv = 6.f * yp.z - (X(-1, 1, 0).z + xy.z) - (c.z + X(0, 2, 0).z) - (X(0, 1, -1).z + yz.z);
            const float lw = 6.f * c.w - (xm.w + xp.w) - (ym.w + yp.w) - (zm.w + zp.w);
            const float hw = 6.f * zp.w - (X(-1, 0, 1).w + xz.w) - (X(0, -1, 1).w + yz.w) - (c.w + X(0, 0, 2).w);
            float pen[7];
#pragma unroll
            for (int d = 0; d < 7; d++) pen[d] = fminf(raw[d], 1e38f);
            res[0] -= vol * ((hi[0] - lo[0]) + (hi[1] - lo[1]) + (hi[2] - lo[2])) + pen[0] * p0;
            res[1] -= vol * (lu - (p0 - xm.x)) + pen[1] * lo[0];
            res[2] -= vol * (lv - (p0 - ym.x)) + pen[2] * lo[1];
            res[3] -= vol * (lw - (p0 - zm.x)) + pen[3] * lo[2];
            res[4] -= vol * (hu - (xp.x - p0)) + pen[4] * hi[0];
            res[5] -= vol * (hv - (yp.x - p0)) + pen[5] * hi[1];
            res[6] -= vol * (hw - (zp.x - p0)) + pen[6] * hi[2];
        }
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
        // the cell's unknowns, and what no red cell owns: the black pressure, and the black
        // cell's faces on the domain boundary (fixed: 0)
        float* o = reinterpret_cast<float*>(xo);
        xo[s] = make_float4(p0 + dp, lo[0], lo[1], lo[2]);
        o[4ll * (s + L.di) + 1] = hi[0];
        o[4ll * (s + L.dj) + 2] = hi[1];
        o[4ll * (s + 1) + 3] = hi[2];
        o[4ll * sb] = pb;
        const int kb = q ? k - 1 : k + 1;
        if (i == 0) o[4ll * sb + 1] = 0.f;
        if (j == 0) o[4ll * sb + 2] = 0.f;
        if (kb == 0) o[4ll * sb + 3] = 0.f;
        if (i == n - 1) o[4ll * (sb + L.di) + 1] = 0.f;
        if (j == n - 1) o[4ll * (sb + L.dj) + 2] = 0.f;
        if (kb == n - 1) o[4ll * (sb + 1) + 3] = 0.f;
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

}  // namespace

// Blocks of the cluster (more than the portable eight: the coarsest solve's rows need the warps of
// all of them)
constexpr int BLOCKS = 16;
static_assert(RowDots<ND, 2>::HALVES <= BLOCKS * CT / 16, "a half-warp for every pair of rows");

static cudaLaunchConfig_t config(cudaStream_t st, cudaLaunchAttribute (&at)[1]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(BLOCKS);
    cfg.blockDim = dim3(CT);
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = BLOCKS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// whether the device runs such a cluster
static bool cluster_ok(int dev) {
    static int state[MAX_DEVICES] = {};  // 0 unknown, 1 no, 2 yes
    if (!state[dev]) {
        int can = 0;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = config(nullptr, at);
        const bool ok = cudaFuncSetAttribute(k_small_cycle, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&can, k_small_cycle, &cfg) == cudaSuccess && can > 0;
        cudaGetLastError();
        state[dev] = ok ? 2 : 1;
    }
    return state[dev] == 2;
}

// Levels of 8 and 16 cells an axis over the 4^3 coarsest one: at 32^3 a cluster's pass takes as
// long as a launch of the whole GPU, and larger coarsest inverses (12^3: 7344 unknowns) need the
// grid-wide product.
bool small_cycle_ok(const stg_t* h, int top) {
    const Level& L = h->lv[top];
    if (top < 1 || top >= MAXS || L.g.n > 16 || (L.g.n & (L.g.n - 1)) || h->dense.nd != ND || h->reference_cycle || !fast(h, L) || !L.P16 || h->opts.prolong == 1)
        return false;
    const int dev = device_slot();
    return dev >= 0 && cluster_ok(dev);
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
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(h->st, at);
    STG_CK(cudaLaunchKernelEx(&cfg, k_small_cycle, S));
    count_launch();
    return STG_OK;
}

}  // namespace stg
