// Design-loop kernels: Brinkman penalty from the density (FluidTopoOpt3D::Update_Fluid),
// the adjoint chain rule (FluidTopoOpt3D::Update_Grad), the density filter, the
// optimality-criteria volume pass and the seeded density generator.
//
// Cell arrays are in the simplex Field order: (i*N + j)*N + k in 3D, i*N + j in 2D.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <utility>

#include "alpha.cuh"
#include "kernels.h"
#include "oc.cuh"
#include "oc_form.h"
#include "stencil.cuh"

namespace stg {

namespace {

constexpr int TPB = 256;

__device__ __forceinline__ long long cidx(int n, int i, int j, int k) { return ((long long)i * n + j) * n + k; }

// face penalty = 1/2 alpha(left cell) + 1/2 alpha(right cell), zero on fixed / absent faces
__global__ void k_face_penalty(Geom g, const double* __restrict__ rho, stg_alpha L, const uint8_t* __restrict__ m,
                               d4* __restrict__ P64, float4* __restrict__ P32) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= g.box()) return;
    int i, j, k;
    g.box_ijk(t, i, j, k);
    const int n = g.n;
    int s = g.slot(i, j, k);
    uint8_t mm = m[s];
    double own = cell_ok(n, i, j, k) ? 0.5 * alpha_of(rho[cidx(n, i, j, k)], L) : 0.0;
    double f[3];
    for (int d = 0; d < 3; d++) {
        int li = i - (d == 0), lj = j - (d == 1), lk = k - (d == 2);
        double lo = (li >= 0 && lj >= 0 && lk >= 0 && cell_ok(n, li, lj, lk)) ? 0.5 * alpha_of(rho[cidx(n, li, lj, lk)], L) : 0.0;
        f[d] = lo + own;
    }
    double u = (mm & MU) ? 0.0 : f[0], v = (mm & MV) ? 0.0 : f[1], w = (mm & MW) ? 0.0 : f[2];
    store4(P64, s, 0.0, u, v, w);
    P32[s] = make_float4(0.f, (float)u, (float)v, (float)w);
}

// dJ/drho_c = 1/2 alpha'(rho_c) sum_{6 faces} (-u lambda + 1/2 u^2)   (FluidTopoOpt3D.cpp:264-281)
__global__ void k_sensitivity(Geom g, const double* __restrict__ rho, stg_alpha L, const d4* __restrict__ x,
                              const d4* __restrict__ lam, double* __restrict__ grad) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    const int n = g.n;
    if (t >= (long long)n * n * n) return;
    int k = (int)(t % n), j = (int)((t / n) % n), i = (int)(t / ((long long)n * n));
    const double* xs = reinterpret_cast<const double*>(x);
    const double* ls = reinterpret_cast<const double*>(lam);
    double sum = 0.0;
    for (int d = 0; d < 3; d++) {
        int s0 = g.slot(i, j, k), s1 = g.slot(i + (d == 0), j + (d == 1), k + (d == 2));
        double u0 = xs[4ll * s0 + 1 + d], l0 = ls[4ll * s0 + 1 + d];
        double u1 = xs[4ll * s1 + 1 + d], l1 = ls[4ll * s1 + 1 + d];
        sum += -(u0 * l0) + (0.5 * u0) * u0;
        sum += -(u1 * l1) + (0.5 * u1) * u1;
    }
    double r = rho[t];
    grad[t] = sum * (0.5 * dalpha_of(r, L));
}

// Linear hat filter: out_i = sum_j w_ij in_j / W_i (forward) or sum_j w_ji in_j / W_j
// (transpose), w_ij = max(0, rmin - |c_i - c_j|) over cells inside the domain, W_i =
// sum_j w_ij. W (for the transpose in_j / W_j) is computed once per call by k_filter_wsum, so
// the transpose reads it instead of re-summing every neighbour's weights. dim 2 runs the same
// loops with a single k plane (nz = 1, no k offsets). Loop order and arithmetic are the same in
// both kernels, so W_i and the sums are identical wherever they are formed.
__device__ __forceinline__ double hat_w(double rmin, int a, int b, int c) { return rmin - sqrt((double)(a * a + b * b + c * c)); }

// the weights rmin - |o| of every offset o, computed once on the host (IEEE sqrt, so the
// same values as hat_w); used when the stencil fits (radius R <= 3)
constexpr int WTAB_MAX = 343;
struct WTab {
    double w[WTAB_MAX];
};
template <bool TAB>
__device__ __forceinline__ double weight(const WTab& T, double rmin, int R, int Rz, int a, int b, int c) {
    if (TAB) return T.w[((a + R) * (2 * R + 1) + (b + R)) * (2 * Rz + 1) + (c + Rz)];
    return hat_w(rmin, a, b, c);
}

// in (the transpose): in_t / W_t instead of W_t, the value every neighbour's sum takes, so one
// FP64 division a cell rather than one a neighbour (64^3, radius 1.5: the transpose was 71 us,
// now 31)
template <bool TAB>
__global__ void k_filter_wsum(int n, int nz, double rmin, int R, int Rz, WTab T, const double* __restrict__ in, double* __restrict__ W) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= (long long)n * n * nz) return;
    int k = (int)(t % nz), j = (int)((t / nz) % n), i = (int)(t / ((long long)n * nz));
    double s = 0;
    for (int a = -R; a <= R; a++)
        for (int b = -R; b <= R; b++)
            for (int c = -Rz; c <= Rz; c++) {
                int ii = i + a, jj = j + b, kk = k + c;
                if (ii < 0 || jj < 0 || kk < 0 || ii >= n || jj >= n || kk >= nz) continue;
                double w = weight<TAB>(T, rmin, R, Rz, a, b, c);
                if (w > 0) s += w;
            }
    W[t] = in ? in[t] / s : s;
}

template <bool TAB>
__global__ void k_filter(int n, int nz, double rmin, int R, int Rz, WTab T, const double* __restrict__ in,
                         const double* __restrict__ W, double* __restrict__ out, int transpose) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= (long long)n * n * nz) return;
    int k = (int)(t % nz), j = (int)((t / nz) % n), i = (int)(t / ((long long)n * nz));
    double s = 0;
    for (int a = -R; a <= R; a++)
        for (int b = -R; b <= R; b++)
            for (int c = -Rz; c <= Rz; c++) {
                int ii = i + a, jj = j + b, kk = k + c;
                if (ii < 0 || jj < 0 || kk < 0 || ii >= n || jj >= n || kk >= nz) continue;
                double w = weight<TAB>(T, rmin, R, Rz, a, b, c);
                if (w <= 0) continue;
                const long long q = ((long long)ii * n + jj) * nz + kk;
                s += w * (transpose ? W[q] : in[q]);
            }
    out[t] = transpose ? s : s / W[t];
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// seeded density: U[0,1) from a SplitMix64 hash of (seed, Field index)
__global__ void k_uniform(long long nc, uint64_t seed, double* __restrict__ out) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= nc) return;
    uint64_t z = seed * 0x9E3779B97F4A7C15ull + (uint64_t)t + 0x632BE59BD9B4E019ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    out[t] = (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// 1D Gaussian along one axis (stride), clamp-to-edge; clip after the last axis
__global__ void k_blur(int n, long long nc, long long stride, const double* __restrict__ w, int R, const double* __restrict__ in,
                       double* __restrict__ out, int clip) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= nc) return;
    int c = (int)((t / stride) % n);
    double acc = 0;
    for (int q = -R; q <= R; q++) {
        int cc = min(n - 1, max(0, c + q));
        acc += w[q + R] * in[t + (long long)(cc - c) * stride];
    }
    out[t] = clip ? fmin(1.0, fmax(0.0, acc)) : acc;
}

// The OC update searches the multiplier l at which the filtered volume sum vw x_new(l) meets the
// target: the bracket [0, 1e9] widened by decades while its upper end still overshoots, then
// bisected to relative width 1e-9 (at most 200 steps), all in one launch. What bounds it is the
// FP64 unit, which each quarter of an SM has half a lane of: 64 clocks for any FP64 instruction
// of a warp, more than ninety until its result is there. Therefore
// - x_new = clamp(s / sqrt(l)) with s formed once (oc_scale), four instructions a cell and probe
//   where the root and the division of oc_new take fifty;
// - a block has one warp for each quarter where registers can hold the cells (OC_T): the
//   sums over warps and blocks, the bracket and 1 / sqrt(l), which every warp forms alike, then
//   cost no quarter more than once;
// - 1 / sqrt(l) of both possible next probes is formed while the blocks' sums travel.
// Before and after, an update: 64^2 cells 271 us, now 112; 64^3 1010 us, now 299 (cells in
// registers); 128^3 4.41 ms, now 1.71 (cells read for each probe).

// The bracket; every warp has the same sums and takes the same steps.
struct OcBracket {
    double l1 = 0.0, l2 = 1e9, lam = 1e9;
    int widened = 0, steps = 0;
    bool widen = true;

    // the next probe after an overshooting volume, or after another (the bracket's end permitting)
    __device__ __forceinline__ double candidate(bool over) const {
        const double up = widen ? 10.0 * l2 : l2;
        if (widen && over && widened + 1 < 60) return up;
        return 0.5 * ((over ? lam : l1) + (over ? up : lam));
    }
    // takes the volume's answer; false once the bracket is narrow enough
    __device__ __forceinline__ bool step(bool over) {
        const double next = candidate(over);
        if (widen) {
            if (over) {
                l1 = l2;
                l2 *= 10.0;
                widen = ++widened < 60;
            } else {
                widen = false;
            }
        } else {
            (over ? l1 : l2) = lam;
            steps++;
        }
        lam = next;
        return widen || ((l2 - l1) > 1e-9 * (l1 + l2) && steps < 200);
    }
};

// The update by the blocks of one cluster (CLUSTER: at most OC_CLUSTER_MAX cells; each warp's
// sum goes straight into every block's shared memory) or of a cooperative launch (through part).
// Both have two buffers of sums, so that a probe never overwrites those that the previous one's
// reduction still reads. A thread holds its cells in R registers each, at most, or, R = 0, reads
// them for each probe with s in xnew (it reads and writes its own cells only).
template <bool CLUSTER, int R>
__global__ void __launch_bounds__(OC_T<R>) k_oc_bisect(int ncell, const double* __restrict__ x, const double* __restrict__ dc,
                                                             const double* __restrict__ vw, double target, double move,
                                                             double lo, double hi, double* xnew, double* __restrict__ part,
                                                             double* __restrict__ lambda_out) {
    namespace cg = cooperative_groups;
    constexpr int T = OC_T<R>, W = T / 32;
    __shared__ double sum[2][CLUSTER ? OC_CB * W : W];
    const cg::cluster_group cluster = cg::this_cluster();
    cg::grid_group grid = cg::this_grid();
    const int nblk = gridDim.x, rank = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double inv_n = 1.0 / ncell;
    const long long q0 = (long long)rank * T + threadIdx.x, dq = (long long)nblk * T;
    OcCell c[R ? R : 1];
    // the rounds that have cells: the same for the block, so that a probe branches past the others
    const int held = (int)min((long long)R, (ncell - (long long)rank * T + dq - 1) / dq);
    if (R) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const long long q = q0 + r * dq;
            c[r] = OcCell{0.0, 0.0, 0.0, 0.0};
            if (q < ncell) c[r] = oc_cell(x[q], dc[q], vw[q], inv_n, move, lo, hi);
        }
    } else {
        for (long long q = q0; q < ncell; q += dq) xnew[q] = oc_scale(x[q], dc[q], vw[q] * inv_n);
    }
    if (CLUSTER) cluster.sync();  // every block runs before its shared memory is written
    OcBracket br;
    double t = rsqrt(br.lam);
    bool more = true;
    for (int buf = 0; more; buf ^= 1) {
        double acc = 0.0, tc, v = 0.0;
        if (R) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (r == held) break;
                acc = c[r].add(t, acc);
            }
        } else {
            for (long long q = q0; q < ncell; q += dq) {
                const double xi = x[q];
                acc = OcCell{xnew[q], fmax(lo, xi - move), fmin(hi, xi + move), vw[q]}.add(t, acc);
            }
        }
        acc = warp_sum(acc);
        if (CLUSTER) {
            if (lane < OC_CB) cluster.map_shared_rank(&sum[buf][0], lane)[rank * W + warp] = acc;
            auto token = cluster.barrier_arrive();
            tc = rsqrt(br.candidate(lane == 1));
            cluster.barrier_wait(std::move(token));
#pragma unroll
            for (int p = 0; p < OC_CB * W; p += 32) v += sum[buf][p + lane];
        } else {
            if (lane == 0) sum[buf][warp] = acc;
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int w = 0; w < W; w++) v += sum[buf][w];
                part[buf * nblk + rank] = v;
                v = 0.0;
            }
            auto token = grid.barrier_arrive();
            tc = rsqrt(br.candidate(lane == 1));
            grid.barrier_wait(std::move(token));
            for (int p = lane; p < nblk; p += 32) v += part[buf * nblk + p];
        }
        v = warp_sum(v);
        const bool over = br.widen ? !(v <= target) : v > target;  // (a NaN target: the least design)
        t = __shfl_sync(0xffffffffu, tc, over ? 1 : 0);
        more = br.step(over);
    }
    for (long long q = q0; q < ncell; q += dq) xnew[q] = oc_new(x[q], dc[q], vw[q] * inv_n, br.lam, move, lo, hi);
    if (rank == 0 && threadIdx.x == 0) *lambda_out = br.lam;
}

}  // namespace

int face_penalty_from_density(cudaStream_t st, const Geom& g, const double* rho, const stg_alpha& law, const uint8_t* m,
                              d4* P64, float4* P32) {
    k_face_penalty<<<grid_for(g.box(), TPB), TPB, 0, st>>>(g, rho, law, m, P64, P32);
    STG_LAUNCH_CK();
    return STG_OK;
}

int sensitivity(cudaStream_t st, const Geom& g, const double* rho, const stg_alpha& law, const d4* x, const d4* lam,
                double* grad) {
    long long nc = (long long)g.n * g.n * g.n;
    k_sensitivity<<<grid_for(nc, TPB), TPB, 0, st>>>(g, rho, law, x, lam, grad);
    STG_LAUNCH_CK();
    return STG_OK;
}

int density_filter(cudaStream_t st, int dim, int n, double rmin, const double* in, double* out, int transpose, double* W) {
    int R = (int)ceil(rmin) - 1;
    if (R < 0) R = 0;
    const int nz = dim == 3 ? n : 1, Rz = dim == 3 ? R : 0;
    long long nc = (long long)n * n * nz;
    WTab T{};
    const int nt = (2 * R + 1) * (2 * R + 1) * (2 * Rz + 1);
    const bool tab = nt <= WTAB_MAX;
    if (tab)
        for (int a = -R; a <= R; a++)
            for (int b = -R; b <= R; b++)
                for (int c = -Rz; c <= Rz; c++)
                    T.w[((a + R) * (2 * R + 1) + (b + R)) * (2 * Rz + 1) + (c + Rz)] = rmin - sqrt((double)(a * a + b * b + c * c));
    if (tab)
        k_filter_wsum<true><<<grid_for(nc, TPB), TPB, 0, st>>>(n, nz, rmin, R, Rz, T, transpose ? in : nullptr, W);
    else
        k_filter_wsum<false><<<grid_for(nc, TPB), TPB, 0, st>>>(n, nz, rmin, R, Rz, T, transpose ? in : nullptr, W);
    STG_LAUNCH_CK();
    if (tab)
        k_filter<true><<<grid_for(nc, TPB), TPB, 0, st>>>(n, nz, rmin, R, Rz, T, in, W, out, transpose);
    else
        k_filter<false><<<grid_for(nc, TPB), TPB, 0, st>>>(n, nz, rmin, R, Rz, T, in, W, out, transpose);
    STG_LAUNCH_CK();
    return STG_OK;
}

static cudaLaunchConfig_t oc_cluster(cudaStream_t st, cudaLaunchAttribute (&at)[1]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(OC_CB);
    cfg.blockDim = dim3(OC_T<OC_CR>);
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = OC_CB;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

int oc_form_here(long long ncell, OcForm* f) {
    int dev = 0, sms = 0, clusters = 0;
    STG_CK(cudaGetDevice(&dev));
    STG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (ncell <= OC_CLUSTER_MAX) {
        const void* kernel = (const void*)k_oc_bisect<true, OC_CR>;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = oc_cluster(nullptr, at);
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
            clusters = 0;
            cudaGetLastError();
        }
    }
    *f = oc_form(ncell, sms, clusters > 0);
    return STG_OK;
}

int oc_update_device(cudaStream_t st, int ncell, const double* x, const double* dc, const double* vw, double frac,
                     double move, double lo, double hi, double* xnew, double* parts, size_t nparts, double* lambda_out) {
    double target = frac * ncell;
    void* args[] = {&ncell, &x, &dc, &vw, &target, &move, &lo, &hi, &xnew, &parts, &lambda_out};
    OcForm f;
    STG_TRY(oc_form_here(ncell, &f));
    if ((size_t)f.parts() > nparts) {
        set_error("oc_update_device: %d block sums in an array of %zu", f.parts(), nparts);
        return STG_E_INVALID;
    }
    if (f.cluster) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = oc_cluster(st, at);
        STG_CK(cudaLaunchKernelExC(&cfg, (const void*)k_oc_bisect<true, OC_CR>, args));
        return STG_OK;
    }
    int per_sm = 0;
    const void* kernel = f.held ? (const void*)k_oc_bisect<false, OC_GR> : (const void*)k_oc_bisect<false, 0>;
    STG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, f.threads, 0));
    if (per_sm < 1) {
        set_error("the OC bisection kernel cannot be made resident");
        return STG_E_CUDA;
    }
    STG_CK(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)f.blocks), dim3((unsigned)f.threads), args, 0, st));
    return STG_OK;
}

int density_noise(cudaStream_t st, int dim, int n, uint64_t seed, const double* w, int R, double* out, double* tmp) {
    long long nc = dim == 3 ? (long long)n * n * n : (long long)n * n;
    unsigned gb = grid_for(nc, TPB);
    k_uniform<<<gb, TPB, 0, st>>>(nc, seed, out);
    STG_LAUNCH_CK();
    if (R >= 0 && w) {
        const long long strides3[3] = {(long long)n * n, n, 1}, strides2[2] = {n, 1};
        double* a = out;
        double* b = tmp;
        for (int ax = 0; ax < dim; ax++) {
            k_blur<<<gb, TPB, 0, st>>>(n, nc, dim == 3 ? strides3[ax] : strides2[ax], w, R, a, b, ax == dim - 1);
            STG_LAUNCH_CK();
            double* c = a;
            a = b;
            b = c;
        }
        // an odd number of passes leaves the result in tmp
        if (a != out) STG_CK(cudaMemcpyAsync(out, a, sizeof(double) * nc, cudaMemcpyDeviceToDevice, st));
    }
    return STG_OK;
}

}  // namespace stg
