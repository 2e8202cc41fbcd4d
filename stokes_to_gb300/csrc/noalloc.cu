// Allocation-free optimality-criteria update (stg_oc_update_noalloc).
//
// Who needs it: callers that cannot call cudaMalloc - host applications that reserve
// the whole GPU for their own memory pool up front, plugins running under another
// framework's allocator budget, and latency-sensitive design loops that cannot afford
// the device-wide synchronisation that cudaMalloc/cudaFree imply. They pass their own
// device arrays for the design, the sensitivity and the result; the only scratch this
// entry point needs (the per-block partial sums of the volume reduction and a small
// table of filter weight sums) lives in the fixed array below, which every GPU that
// loads this library holds until the process exits.
//
// The bisection, each cell's arithmetic and the order of the volume's sums (topo.cu k_oc_bisect,
// in whichever form a handle of this size would take) are the ones of stg_oc_update, with the
// filter volume weights vw_j = sum_i w_ij / W_i formed on the fly instead of being read from a
// buffer, so both entry points return the same design and multiplier, bit for bit. 1 / W_i depends only on how far
// cell i lies from each pair of domain faces (clamped at the filter radius R), so it is read
// from a table of (R+1)^6 classes built once per call, in the summation order of the
// handle's filter; a probe then costs (2R+1)^3 table reads and multiply-adds per cell, and
// no division among them. Bound: the FP64 unit with large filters (64^3, radius 4: 15.3 ms an
// update of some sixty probes), the host's round trip per probe with small ones (32^3, radius 1.5:
// 1.35 ms; 64^3: 2.9 ms, 3.3 with sums in an order of their own, 256 cells a block).
#include <climits>
#include <cmath>
#include <mutex>

#include "kernels.h"
#include "oc.cuh"
#include "oc_form.h"

namespace stg {

namespace {

constexpr int TPB = 256;
constexpr int NOALLOC_PARTS = 1216;           // partial sums: one a warp of the register forms
constexpr int NOALLOC_MAX_N = 1024;           // largest design: 1024^3 cells
constexpr int NOALLOC_MAX_R = 3;              // largest filter radius index: rmin <= 4
constexpr int NOALLOC_CLASSES = 4096;         // (R+1)^6 weight-sum classes at R = 3
constexpr int NOALLOC_TAB = 343;              // (2R+1)^3 filter weights at R = 3
constexpr int SCR_SUM = NOALLOC_PARTS;        // reduced volume
constexpr int SCR_WCLASS = 1280;              // start of the class table (256-byte aligned)
constexpr int NOALLOC_SCRATCH = SCR_WCLASS + NOALLOC_CLASSES;  // 5376 doubles = 42 KB

static_assert(OC_MAX_BLOCKS * (OC_T<OC_GR> / 32) <= NOALLOC_PARTS, "a partial sum for every warp");

// Scratch shared by every call on a device. Calls that overlap on the GPU race on it.
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_SCRATCH];

std::mutex g_mu;
double* g_scratch_ptr[256] = {};

// Device address of the scratch on the current device, resolved once per device.
int scratch_on_current_device(double** out) {
    int dev = 0;
    STG_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) {
        set_error("device ordinal %d out of range", dev);
        return STG_E_INVALID;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress", __FILE__, __LINE__);
        g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_ptr[dev];
    return STG_OK;
}

// filter weights rmin - |o| for every offset o in [-R, R]^3, formed on the host with
// IEEE sqrt exactly as the handle's filter table
struct WTabNA {
    double w[NOALLOC_TAB];
};

// one axis's class: (how far the cell may reach down, how far up), each clamped at R
__device__ __forceinline__ int axis_class(int i, int n, int R) {
    const int lo = min(i, R), hi = min(n - 1 - i, R);
    return lo * (R + 1) + hi;
}

// 1 / W for every class, W the sum of the positive weights over the offsets the class allows,
// in the loop order of the handle's weight-sum kernel (a, then b, then c), so the values are
// bit-identical to the ones behind the weights that stg_oc_update reads
__global__ void k_wsum_classes(int R, WTabNA T, double* __restrict__ wc) {
    const int per = (R + 1) * (R + 1);
    const int ncls = per * per * per;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ncls) return;
    const int cz = t % per, cy = (t / per) % per, cx = t / (per * per);
    const int xlo = cx / (R + 1), xhi = cx % (R + 1), ylo = cy / (R + 1), yhi = cy % (R + 1), zlo = cz / (R + 1),
              zhi = cz % (R + 1);
    const int D = 2 * R + 1;
    double s = 0;
    for (int a = -R; a <= R; a++)
        for (int b = -R; b <= R; b++)
            for (int c = -R; c <= R; c++) {
                if (a < -xlo || a > xhi || b < -ylo || b > yhi || c < -zlo || c > zhi) continue;
                const double w = T.w[((a + R) * D + (b + R)) * D + (c + R)];
                if (w > 0) s += w;
            }
    wc[t] = 1.0 / s;
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// vw_j = sum_i w_ij / W_i of cell t, summed in the handle filter's transpose order
__device__ __forceinline__ double cell_weight(int n, int R, const WTabNA& T, const double* wcls, long long t) {
    const int per = (R + 1) * (R + 1), D = 2 * R + 1;
    const int k = (int)(t % n), j = (int)((t / n) % n), i = (int)(t / ((long long)n * n));
    double vw = 0;
    for (int a = -R; a <= R; a++) {
        const int ii = i + a;
        if (ii < 0 || ii >= n) continue;
        const int ca = axis_class(ii, n, R) * per * per;
        for (int b = -R; b <= R; b++) {
            const int jj = j + b;
            if (jj < 0 || jj >= n) continue;
            const int cb = ca + axis_class(jj, n, R) * per;
            for (int c = -R; c <= R; c++) {
                const int kk = k + c;
                if (kk < 0 || kk >= n) continue;
                const double w = T.w[((a + R) * D + (b + R)) * D + (c + R)];
                if (w <= 0) continue;
                vw += w * wcls[cb + axis_class(kk, n, R)];
            }
        }
    }
    return vw;
}

// What the kernels share: the problem, and its class table into shared memory
struct NaIn {
    int n, R;
    WTabNA T;
    const double *wclass, *x, *dc;
    double move, lo, hi;
    __device__ __forceinline__ long long cells() const { return (long long)n * n * n; }
    __device__ __forceinline__ void table(double* wcls) const {
        const int ncls = (R + 1) * (R + 1) * (R + 1) * (R + 1) * (R + 1) * (R + 1);
        for (int c = threadIdx.x; c < ncls; c += blockDim.x) wcls[c] = wclass[c];
        __syncthreads();
    }
    __device__ __forceinline__ OcCell cell(const double* wcls, long long t, double inv_n) const {
        return oc_cell(x[t], dc[t], cell_weight(n, R, T, wcls, t), inv_n, move, lo, hi);
    }
};

// One bisection probe where the handle's update holds a thread's cells, dq apart, in registers:
// block b forms the sum of its warp b. The block's eight warps take the cells' rounds in turn
// (the weights are the work: one warp would be a chain of up to sixteen cells), beginning with
// another warp in each block, since two rounds keep two quarters of an SM busy only; the first
// adds them up in the thread's order.
__global__ void __launch_bounds__(TPB) k_noalloc_held(const __grid_constant__ NaIn in, int dq, int rounds, double lam,
                                                      double* __restrict__ part) {
    __shared__ double wcls[NOALLOC_CLASSES], sv[OC_GR][32], sx[OC_GR][32];
    in.table(wcls);
    const long long nc = in.cells();
    const double inv_n = 1.0 / (double)nc, t = rsqrt(lam);
    const int lane = threadIdx.x & 31;
    for (int r = ((threadIdx.x >> 5) + blockIdx.x + (blockIdx.x >> 6)) % (TPB / 32); r < rounds; r += TPB / 32) {
        const long long q = blockIdx.x * 32ll + lane + (long long)r * dq;
        double v = 0.0, x = 0.0;
        if (q < nc) {
            const OcCell c = in.cell(wcls, q, inv_n);
            v = c.vw;
            x = c.at(t);
        }
        sv[r][lane] = v;
        sx[r][lane] = x;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    double acc = 0.0;
    for (int r = 0; r < rounds; r++) acc = fma(sv[r][lane], sx[r][lane], acc);
    acc = warp_sum(acc);
    if (lane == 0) part[blockIdx.x] = acc;
}

// and where it reads them for each probe: the same blocks and threads
__global__ void __launch_bounds__(OC_T<0>) k_noalloc_read(const __grid_constant__ NaIn in, double lam, double* __restrict__ part) {
    __shared__ double wcls[NOALLOC_CLASSES], sh[OC_T<0> / 32];
    in.table(wcls);
    const long long nc = in.cells();
    const double inv_n = 1.0 / (double)nc, t = rsqrt(lam);
    double acc = 0.0;
    for (long long q = (long long)blockIdx.x * OC_T<0> + threadIdx.x; q < nc; q += (long long)gridDim.x * OC_T<0>)
        acc = in.cell(wcls, q, inv_n).add(t, acc);
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < OC_T<0> / 32; w++) v += sh[w];
        part[blockIdx.x] = v;
    }
}

// The sum of `ranks` blocks' sums of PER warps each, in the order of k_oc_bisect's warps; all
// loads of a lane are in flight together
template <int PER>
__global__ void k_noalloc_sum(const double* __restrict__ part, int ranks, double* __restrict__ out) {
    constexpr int Q = (OC_MAX_BLOCKS + 31) / 32;
    double s[Q][PER], v = 0.0;
#pragma unroll
    for (int q = 0; q < Q; q++)
#pragma unroll
        for (int w = 0; w < PER; w++) {
            const int p = threadIdx.x + 32 * q;
            s[q][w] = p < ranks ? part[p * PER + w] : 0.0;
        }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        if (32 * q >= ranks) break;
        double t = s[q][0];
#pragma unroll
        for (int w = 1; w < PER; w++) t += s[q][w];
        v += t;
    }
    v = warp_sum(v);
    if (threadIdx.x == 0) *out = v;
}

// x_new at the multiplier. x and xnew may be the same array (each element is read before it is
// written by one thread).
__global__ void __launch_bounds__(TPB) k_noalloc_new(const __grid_constant__ NaIn in, double lam, double* xnew) {
    __shared__ double wcls[NOALLOC_CLASSES];
    in.table(wcls);
    const long long nc = in.cells();
    const double inv_n = 1.0 / (double)nc;
    for (long long q = (long long)blockIdx.x * TPB + threadIdx.x; q < nc; q += (long long)gridDim.x * TPB)
        xnew[q] = oc_new(in.x[q], in.dc[q], cell_weight(in.n, in.R, in.T, wcls, q) * inv_n, lam, in.move, in.lo, in.hi);
}

}  // namespace

}  // namespace stg

using namespace stg;

extern "C" int stg_oc_update_noalloc(int n, double rmin, const double* d_x, const double* d_dc, double frac, double move,
                                     double lo, double hi, double* d_xnew, double* lambda_out, void* cuda_stream) {
    if (n < 1 || n > NOALLOC_MAX_N) {
        set_error("stg_oc_update_noalloc: N = %d outside 1..%d (designs of at most 1024^3 cells)", n, NOALLOC_MAX_N);
        return STG_E_INVALID;
    }
    if (!d_x || !d_dc || !d_xnew) {
        set_error("stg_oc_update_noalloc: null device array");
        return STG_E_INVALID;
    }
    if (!(rmin > 0) || !(rmin <= NOALLOC_MAX_R + 1)) {
        set_error("stg_oc_update_noalloc: filter radius rmin = %g outside (0, %d]", rmin, NOALLOC_MAX_R + 1);
        return STG_E_INVALID;
    }
    double* scratch = nullptr;
    STG_TRY(scratch_on_current_device(&scratch));
    cudaStream_t st = (cudaStream_t)cuda_stream;
    int R = (int)ceil(rmin) - 1;
    if (R < 0) R = 0;
    const int D = 2 * R + 1;
    WTabNA T{};
    for (int a = -R; a <= R; a++)
        for (int b = -R; b <= R; b++)
            for (int c = -R; c <= R; c++) T.w[((a + R) * D + (b + R)) * D + (c + R)] = rmin - sqrt((double)(a * a + b * b + c * c));
    const long long nc = (long long)n * n * n;
    OcForm f;
    STG_TRY(oc_form_here(nc, &f));
    double* part = scratch;
    double* sum = scratch + SCR_SUM;        // reduced volume
    double* wclass = scratch + SCR_WCLASS;  // 1 / W per class
    const NaIn in{n, R, T, wclass, d_x, d_dc, move, lo, hi};
    const int ncls = (R + 1) * (R + 1) * (R + 1) * (R + 1) * (R + 1) * (R + 1);
    k_wsum_classes<<<(ncls + 127) / 128, 128, 0, st>>>(R, T, wclass);
    STG_LAUNCH_CK();
    double l1 = 0.0, l2 = 1e9, lmid = 0.0, target = frac * (double)nc;
    int steps = 0;
    const double tol = 1e-9;
    auto volume = [&](double lam, double* vol) -> int {
        if (f.held) {
            const int warps = f.blocks * (f.threads / 32), dq = f.blocks * f.threads;
            k_noalloc_held<<<warps, TPB, 0, st>>>(in, dq, (int)((nc + dq - 1) / dq), lam, part);
            STG_LAUNCH_CK();
            if (f.cluster)  // its blocks add every warp's sum themselves
                k_noalloc_sum<1><<<1, 32, 0, st>>>(part, warps, sum);
            else
                k_noalloc_sum<OC_T<OC_GR> / 32><<<1, 32, 0, st>>>(part, f.blocks, sum);
        } else {
            k_noalloc_read<<<f.blocks, OC_T<0>, 0, st>>>(in, lam, part);
            STG_LAUNCH_CK();
            k_noalloc_sum<1><<<1, 32, 0, st>>>(part, f.blocks, sum);
        }
        STG_LAUNCH_CK();
        STG_CK(cudaMemcpyAsync(vol, sum, sizeof(double), cudaMemcpyDeviceToHost, st));
        STG_CK(cudaStreamSynchronize(st));
        return STG_OK;
    };
    // bracket widened by decades while its upper end overshoots the volume (stg_oc_update)
    for (int k = 0; k < 60; k++) {
        double vol = 0;
        STG_TRY(volume(l2, &vol));
        if (vol <= target) break;
        l1 = l2;
        l2 *= 10.0;
    }
    while ((l2 - l1) > tol * (l1 + l2) && steps < 200) {
        lmid = 0.5 * (l1 + l2);
        double vol = 0;
        STG_TRY(volume(lmid, &vol));
        if (vol > target)
            l1 = lmid;
        else
            l2 = lmid;
        steps++;
    }
    lmid = 0.5 * (l1 + l2);
    const long long g = (nc + TPB - 1) / TPB;
    k_noalloc_new<<<(unsigned)(g < 1216 ? g : 1216), TPB, 0, st>>>(in, lmid, d_xnew);
    STG_LAUNCH_CK();
    STG_CK(cudaStreamSynchronize(st));
    if (lambda_out) *lambda_out = lmid;
    return STG_OK;
}
