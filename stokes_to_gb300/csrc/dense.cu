// Coarsest-level direct solve (DirectSolve3D, stoke/StokeLike.cu:374-648) on the GPU.
//
// The dense matrix is read off the same nine probes as the reference: two cell probes
// coloured by (x+y+z+flag) mod 2 and seven face probes coloured by
// (x + 2y + 3z + magic[d] + flag) mod 7, magic = {2,4,5}; each probe image entry is
// stored at the column the colouring rule assigns to its row (:431-603). Cell-cell
// entries are never recorded (as in the reference); with `closed` the pressure block
// gets +1 everywhere (:605-608). Unknowns that exist only as padding in the reference
// layout are identity rows decoupled from the rest, so the dense system here keeps the
// unknowns that exist. It is inverted once per set-up by block elimination
// (k_inv_blocks), or, where that does not apply, by Gauss-Jordan elimination with partial
// pivoting on [A | I] (double-buffered in L2); either is one cooperative launch with a
// grid-wide barrier between its steps. The inverse is applied as a GEMV inside each V-cycle.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "fp64bits.cuh"
#include "kernels.h"
#include "stencil.cuh"

namespace stg {

namespace {

constexpr int TPB = 256;

__device__ __forceinline__ void probe_of(int q, int& kind, int& flag) {
    kind = q < 2 ? 0 : 1;
    flag = q < 2 ? q : q - 2;
}
__global__ void k_probe(Geom g, int first, d4* __restrict__ probe) {
    int kind, flag;
    probe_of(first + blockIdx.y, kind, flag);
    probe += (long long)blockIdx.y * g.nslot;
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= g.box()) return;
    int i, j, k;
    g.box_ijk(t, i, j, k);
    const int n = g.n;
    const int magic[3] = {2, 4, 5};
    double v[4] = {0, 0, 0, 0};
    if (kind == 0) {
        if (cell_ok(n, i, j, k)) v[0] = ((i + j + k + flag) % 2 == 0) ? 1.0 : 0.0;
    } else {
        for (int d = 0; d < 3; d++)
            if (face_ok(n, d, i, j, k)) v[d + 1] = ((i + 2 * j + 3 * k + magic[d] + flag) % 7 == 0) ? 1.0 : 0.0;
    }
    store4(probe, g.slot(i, j, k), v[0], v[1], v[2], v[3]);
}

// Scatter one probe image into the dense matrix (column-major, nd x nd).
__global__ void k_scatter(Geom g, int first, int nd, const int* __restrict__ slot_of, const int* __restrict__ comp_of,
                          const int* __restrict__ dense_of, const d4* __restrict__ image, double* __restrict__ A) {
    int row = blockIdx.x * TPB + threadIdx.x;
    if (row >= nd) return;
    int kind, flag;
    probe_of(first + blockIdx.y, kind, flag);
    image += (long long)blockIdx.y * g.nslot;
    const int n = g.n;
    int s = slot_of[row], c = comp_of[row];
    // logical coordinates of the slot
    int k = s % g.sz - 1, r = s / g.sz;
    int j = r % g.sy - 1, i = r / g.sy - 1;
    double val = reinterpret_cast<const double*>(image)[4ll * s + c];
    int ci = -1, cj = 0, ck = 0, cc = 0;
    if (kind == 0) {
        if (c == 0) return;  // cell rows are not read from the cell probes
        int d = c - 1;
        ci = i;
        cj = j;
        ck = k;
        if ((i + j + k + flag) % 2 == 1) {
            if (d == 0) ci--;
            if (d == 1) cj--;
            if (d == 2) ck--;
        }
        if (!(ci >= 0 && cj >= 0 && ck >= 0 && cell_ok(n, ci, cj, ck))) return;
        cc = 0;
    } else {
        const int magic[3] = {2, 4, 5};
        ci = i;
        cj = j;
        ck = k;
        if (c == 0) {
            switch ((i + 2 * j + 3 * k + flag) % 7) {
                case 1: cc = 2; cj++; break;
                case 2: cc = 3; break;
                case 3: cc = 2; break;
                case 4: cc = 1; ci++; break;
                case 5: cc = 1; break;
                case 6: cc = 3; ck++; break;
                default: return;
            }
        } else {
            int d = c - 1;
            cc = c;
            switch ((i + 2 * j + 3 * k + magic[d] + flag) % 7) {
                case 1: ci--; break;
                case 2: cj--; break;
                case 3: ck--; break;
                case 4: ck++; break;
                case 5: cj++; break;
                case 6: ci++; break;
                default: break;
            }
        }
        // a column outside the existing unknowns is a padding column of the reference layout
        if (ci < 0 || cj < 0 || ck < 0 || !face_ok(n, cc - 1, ci, cj, ck)) return;
    }
    int col = dense_of[4 * g.slot(ci, cj, ck) + cc];
    if (col < 0) return;
    A[(long long)row * 2 * nd + col] = val;
}

__global__ void k_closed(int nd, const int* __restrict__ comp_of, double* __restrict__ A) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= (long long)nd * nd) return;
    int row = (int)(t / nd), col = (int)(t % nd);
    if (comp_of[row] == 0 && comp_of[col] == 0) A[(long long)row * 2 * nd + col] += 1.0;
}

// [A | I]: zero the left half (filled by the probes), identity on the right half
__global__ void k_aug_init(int nd, double* __restrict__ A) {
    long long t = (long long)blockIdx.x * TPB + threadIdx.x;
    if (t >= 2ll * nd * nd) return;
    int row = (int)(t / (2 * nd)), col = (int)(t % (2 * nd));
    A[t] = (col >= nd && col - nd == row) ? 1.0 : 0.0;
}

// Pivot of column k among rows k..nd-1 of the row-major nd x 2nd matrix (largest |a|, the
// first on ties, as LAPACK), found by every block; loads through L2 (the cooperative
// kernel rewrites the buffers during its launch).
__device__ __forceinline__ int gj_pivot(int nd, int k, const double* in) {
    __shared__ double sv[TPB / 32];
    __shared__ int si[TPB / 32];
    __shared__ int sp;
    const int W = 2 * nd;
    double best = -1.0;
    int bi = nd;
    for (int r = k + threadIdx.x; r < nd; r += TPB) {
        const double a = fabs(__ldcg(in + (long long)r * W + k));
        if (a > best || (a == best && r < bi)) {
            best = a;
            bi = r;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    if ((threadIdx.x & 31) == 0) {
        sv[threadIdx.x >> 5] = best;
        si[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = -1.0;
        int ii = nd;
        for (int w = 0; w < TPB / 32; w++)
            if (sv[w] > b || (sv[w] == b && si[w] < ii)) {
                b = sv[w];
                ii = si[w];
            }
        sp = ii < nd ? ii : k;  // a column of NaN has no largest entry: stay in the matrix
    }
    __syncthreads();
    return sp;
}

// One Gauss-Jordan pivot step, rows row0, row0 + rstep, ... of the output: row k <- row
// p / a_pk, row p <- row k - a_kk row k', other rows i <- row i - a_ik row k'. The
// reciprocal of the pivot is formed once per block (an FP64 division per thread costs
// more than the row on GB300's FP64 pipe).
__device__ __forceinline__ void gj_rows(int nd, int k, int p, const double* in, double* out, int* info, int row0, int rstep) {
    __shared__ double s_inv;
    const int W = 2 * nd;
    const double piv = __ldcg(in + (long long)p * W + k);
    if (threadIdx.x == 0) s_inv = piv != 0.0 ? 1.0 / piv : 0.0;
    __syncthreads();
    const double inv = s_inv;
    for (int row = row0; row < nd; row += rstep) {
        if (piv == 0.0) {
            if (row == 0 && threadIdx.x == 0 && *info == 0) *info = k + 1;
            for (int c = threadIdx.x; c < W; c += TPB) out[(long long)row * W + c] = __ldcg(in + (long long)row * W + c);
            continue;
        }
        const int src = row == k ? p : (row == p ? k : row);
        const double f = row == k ? 0.0 : __ldcg(in + (long long)src * W + k);
        for (int c = threadIdx.x; c < W; c += TPB) {
            const double pr = __ldcg(in + (long long)p * W + c) * inv;
            out[(long long)row * W + c] = row == k ? pr : __ldcg(in + (long long)src * W + c) - f * pr;
        }
    }
    __syncthreads();  // s_inv and the pivot's shared words are rewritten by the next step
}

// One pivot step per launch (block b handles row b); the fallback where a cooperative
// launch is unavailable.
__global__ void __launch_bounds__(TPB) k_gj_step(int nd, int k, const double* in, double* out, int* info) {
    const int p = gj_pivot(nd, k, in);
    gj_rows(nd, k, p, in, out, info, blockIdx.x, nd);
}

// All nd pivot steps in one cooperative launch, a grid-wide barrier between them (the
// launch gaps of nd dependent kernels were most of the set-up time): the operations of
// k_gj_step in the same order, so the same inverse bit for bit. Step k reads buffer k mod
// 2 and writes the other.
__device__ __forceinline__ void gj_all(int nd, double* a, double* b, int* info) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    for (int k = 0; k < nd; k++) {
        const double* in = (k & 1) ? b : a;
        double* out = (k & 1) ? a : b;
        const int p = gj_pivot(nd, k, in);
        gj_rows(nd, k, p, in, out, info, blockIdx.x, gridDim.x);
        grid.sync();
    }
}
__global__ void __launch_bounds__(TPB) k_gj_all(int nd, double* a, double* b, int* info) { gj_all(nd, a, b, info); }

// ---------------------------------------------------------------- block inversion
// The coarsest matrix is a symmetric saddle point [K B^T; B C]: K (faces) positive definite, C
// (cells) the cell penalties plus, on a closed domain, ones everywhere. With the ones moved to
// one bordering unknown l,
//   M = [K B^T 0; B C0 e; 0 e^T -1],   C0 = C - e e^T  (its Schur complement over l is A),
// elimination in the order faces, cells, l meets positive pivots on the faces and negative
// ones on the cells, which is stable without a pivot search; only the last block, which
// holds l and the last cells, pivots inside itself. So the inverse is formed block by block, in
// place: for a diagonal block p of B unknowns and D = M_pp^-1,
//   M_ij -= M_ip D M_pj,  M_pj = D M_pj,  M_ip = -M_ip D,  M_pp = D.
// The faces of different axes are uncoupled until cells are eliminated, so one step takes a block
// of every axis (S pivots). M stays symmetric up to signs (M_ji = M_ij^T, negated where just
// one of i and j has been eliminated), so only the tiles i <= j are kept and updated, and the
// column panel M_ip is the row panel's transpose: N^3 FP64 operations, less the tiles that are
// zero, instead of the pivoted elimination's 4 nd^3.
// A step: every block of the grid inverts the S pivot tiles for itself; the products E = D M_pj
// are shared out; grid barrier; the tiles are shared out; grid barrier.
// A pivot of the wrong sign (a negative penalty), faces that are coupled across axes (open
// boundaries) or a matrix that is not symmetric end the attempt, in every block alike, and the
// pivoted elimination above runs on the untouched [A | I] instead.
//
// Bound: the FP64 pipe, two FMAs per SM and clock, at nd = 2112 (set-up of a 96^2 handle: 276 ms
// pivoted, 14.6 with full square updates and FP64 tile inverses, 8.2 now); at nd = 304 the chain
// of 10 steps of about 25 us (whole set-up of a 16^3 handle 2.2 ms pivoted, 0.36 now); at
// nd = 7344 (12^3: grids of 24, 48, 96) the set-up takes 0.173 s, 10.95 pivoted. Tile
// width: 16 keeps the chain of small inversions short, 32 halves the panel traffic where the
// products dominate.

// Inverse of an FP64 tile to about 2^-44 in double-float arithmetic (error-free sums after Knuth,
// products after Dekker, with an FMA) by one warp: the FP64 pipe's
// latency makes a pivot of the same elimination cost 1900 clocks, the FP32 pipe's 300. Lane: row
// lane / LPR, columns CE (lane % LPR) .. in registers. s becomes the inverse, hi its FP32 values.
struct D2 {
    float h, l;
};
__device__ __forceinline__ D2 d2_norm(float h, float l) {
    const float t = h + l;
    return D2{t, l - (t - h)};
}
__device__ __forceinline__ D2 d2_mul(D2 a, D2 b) {
    const float p = a.h * b.h;
    return d2_norm(p, fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p))));
}
__device__ __forceinline__ D2 d2_sub(D2 a, D2 b) {  // a - b
    const float t = a.h - b.h, bb = t - a.h;
    return d2_norm(t, ((a.h - (t - bb)) - (b.h + bb)) + (a.l - b.l));
}
__device__ __forceinline__ D2 d2_inv(D2 a) {
    const float r = __fdividef(1.f, a.h);  // a few 2^-24 off; the residual below is exact to second order
    const float e = fmaf(-a.l, r, fmaf(-a.h, r, 1.f));  // 1 - a r
    return d2_norm(r, r * fmaf(e, e, e));
}
__device__ __forceinline__ D2 d2_shfl(D2 a, int src) {
    return D2{__shfl_sync(0xffffffffu, a.h, src), __shfl_sync(0xffffffffu, a.l, src)};
}

template <int B>
__device__ __forceinline__ bool tile_inverse(double (&s)[B][B + 1], float (&hi)[B][B + 1], bool local_pivot, bool positive) {
    constexpr int LPR = 32 / B, CE = B / LPR;
    const int lane = threadIdx.x & 31, r = lane / LPR, h = lane % LPR;
    D2 a[CE];
#pragma unroll
    for (int c = 0; c < CE; c++) split_bits(s[r][h * CE + c], a[c].h, a[c].l);
    int col = 0;  // lane q: the pivot row of step q
    // the columns rotate by one a step, so that the pivot column is always the first and the loop
    // stays small (unrolled over the pivots it ran from instruction-cache misses: 186 thousand
    // clocks a 32 x 32 tile); B steps bring them back in order
#pragma unroll 1
    for (int q = 0; q < B; q++) {
        D2 f = d2_shfl(a[0], r * LPR);  // the pivot column's entry of the own row
        if (local_pivot) {
            // (a NaN counts as infinity: every lane has to come to the same row, since the lanes
            // exchange rows together)
            const float v = fabsf(f.h);
            float best = r < q ? -1.f : v <= 3e38f ? v : INFINITY;
            int bi = r;
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            const int p = bi;
            if (p != q) {  // exchange rows p and q
                const int src = (r == q ? p : r == p ? q : r) * LPR + h;
#pragma unroll
                for (int c = 0; c < CE; c++) a[c] = d2_shfl(a[c], src);
                f = d2_shfl(f, src);
            }
            if (lane == q) col = p;
        }
        const D2 piv = d2_shfl(f, q * LPR);
        // NaN and infinity fail as well. The pivot is the same in all lanes, so all leave: going on after
        // a pivot of 0 (the last cell of a closed domain without its ones) would fill the tile with NaN.
        const float want = local_pivot ? fabsf(piv.h) : (positive ? piv.h : -piv.h);
        if (!(want > 0.f && want < 1e37f)) return false;
        const D2 inv = d2_inv(piv);
        const D2 g = r == q ? D2{-inv.h, -inv.l} : d2_mul(f, inv);
        const D2 own{-g.h, -g.l};  // the pivot column's new entry
        D2 first = own;            // the first column's, which moves to the end
#pragma unroll
        for (int c = 0; c < CE; c++) {
            const D2 row = d2_shfl(a[c], q * LPR + h);
            const D2 v = d2_sub(r == q ? D2{0.f, 0.f} : a[c], d2_mul(g, row));
            if (c > 0)
                a[c - 1] = v;
            else if (h > 0)
                first = v;  // (on the row's first lane it is the pivot column)
        }
        // the row's lanes hand their first column on: lane h takes lane h + 1's, the last the pivot's
        a[CE - 1] = LPR > 1 ? d2_shfl(first, r * LPR + (h + 1) % LPR) : first;
    }
#pragma unroll
    for (int c = 0; c < CE; c++) {
        s[r][h * CE + c] = f2d_bits(a[c].h) + f2d_bits(a[c].l);
        hi[r][h * CE + c] = a[c].h;
    }
    __syncwarp();
    if (local_pivot) {  // undo the row exchanges on the columns, last first
        for (int q = B - 1; q >= 0; q--) {
            const int p = __shfl_sync(0xffffffffu, col, q);
            if (p != q && h == 0) {
                const double t = s[r][q];
                s[r][q] = s[r][p];
                s[r][p] = t;
                const float u = hi[r][q];
                hi[r][q] = hi[r][p];
                hi[r][p] = u;
            }
            __syncwarp();
        }
    }
    return true;
}

// Shared memory of a block: 59 KB for 32-wide tiles of three axes, which makes it dynamic (a kernel's
// own declarations end at 48 KB); the others declare their arrays one by one (as members of one
// struct 6 registers more, and a set-up of 192^2 takes 7.77 instead of 7.73 ms)
template <int B, int S>
struct InvShared {
    double D[S][B][B + 1], E[B][B + 1], A[B][B + 1];
    float H[S][B][B + 1], F[B][B + 1];
    int bad;
    static constexpr size_t dynamic() { return sizeof(InvShared) > 48 * 1024 ? sizeof(InvShared) : 0; }
};
template <class W, class T, int ID>  // member `in` of the window W, or array ID of type T of its own
__device__ __forceinline__ T& inv_array(T W::*in) {
    extern __shared__ __align__(16) unsigned char inv_window[];
    if constexpr (W::dynamic() > 0) {
        return reinterpret_cast<W*>(inv_window)->*in;
    } else {
        __shared__ T own;
        return own;
    }
}

// perm[q], q < N: the unknown at position q, -1 for a decoupled filler, -2 for l. The
// positions hold S face sections of TF tiles each (one axis a section), then the cells' tiles.
// ws: N^2 + 3 S B N doubles (the pivoted elimination's second buffer).
template <int B, int S>
__global__ void __launch_bounds__(TPB) k_inv_blocks(int nd, int N, int TF, const int* __restrict__ perm, int closed, double* a,
                                                    double* ws, int* info) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    using W = InvShared<B, S>;
    auto& sD = inv_array<W, double[S][B][B + 1], 0>(&W::D);
    auto& sE = inv_array<W, double[B][B + 1], 1>(&W::E);
    auto& sA = inv_array<W, double[B][B + 1], 2>(&W::A);
    auto& sH = inv_array<W, float[S][B][B + 1], 3>(&W::H);
    auto& sF = inv_array<W, float[B][B + 1], 4>(&W::F);
    int& s_bad = inv_array<W, int, 5>(&W::bad);
    const int T = N / B, tid = threadIdx.x, TC = S * TF, cell0 = TC * B;
    constexpr int EPT = B * B / TPB;  // tile elements of a thread: rows r0 + e (TPB / B), column c0
    const int c0 = tid % B, r0 = tid / B;
    constexpr int RS = TPB / B;
    double* M = ws;
    // pivot tiles of step k: s TF + k for the sections s < S while k < TF, then TC + (k - TF)
    const int steps = TF + (T - TC);
    auto pivots = [&](int k) { return k < TF ? S : 1; };
    auto pivot = [&](int k, int q) { return k < TF ? q * TF + k : TC + (k - TF); };
    auto pivot_of = [&](int k, int i) {  // i is pivot .. of step k, or -1
        for (int q = 0; q < pivots(k); q++)
            if (i == pivot(k, q)) return q;
        return -1;
    };
    // M_ip = sign(i) M_pi^T for a pivot p of step k: -1 where i is already eliminated
    auto sign = [&](int k, int i) { return (i < TC ? (k >= TF || i % TF < k) : i - TC < k - TF) ? -1.0 : 1.0; };
    // while faces are eliminated, pivot q of section q is coupled to its own section and the cells only
    auto apart = [&](int k, int q, int i) { return k < TF && i < TC && i / TF != q; };
    // panels: row tiles M_pj of pivot q of step k (two parities), and E = D M_pj
    auto panel = [&](int k, int q, int j) { return ws + (long long)N * N + ((long long)((k & 1) * S + q) * N + (long long)j * B) * B; };
    auto epanel = [&](int q, int j) { return ws + (long long)N * N + ((long long)(2 * S + q) * N + (long long)j * B) * B; };
    auto put = [&](int i, int j, int r, int k, double v) {  // element (r, c0) of tile i <= j, and the panels of step k
        M[(long long)(i * B + r) * N + j * B + c0] = v;
        const int pi = pivot_of(k, i), pj = pivot_of(k, j);
        if (pi >= 0) panel(k, pi, j)[r * B + c0] = v;
        if (pj >= 0 && i != j) panel(k, pj, i)[c0 * B + r] = sign(k, i) * v;
    };
    auto tile_of = [&](int t, int& i, int& j) {  // t-th of the tiles i <= j
        j = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
        while (j * (j + 1) / 2 > t) j--;
        while ((j + 1) * (j + 2) / 2 <= t) j++;
        i = t - j * (j + 1) / 2;
    };
    const int tiles = T * (T + 1) / 2;
    // the bordered matrix in the elimination order; *info = -1: not of the form
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        int i, j;
        tile_of(t, i, j);
        const bool ap = i < TC && j < TC && i / TF != j / TF;
#pragma unroll
        for (int e = 0; e < EPT; e++) {
            const int r = r0 + e * RS, x = i * B + r, y = j * B + c0;
            const int px = __ldg(perm + x), py = __ldg(perm + y);
            double v;
            if (px >= 0 && py >= 0) {
                v = a[(long long)px * 2 * nd + py];
                if (fabs(v - a[(long long)py * 2 * nd + px]) > 1e-12 * fabs(v)) atomicExch(info, -1);
                if (closed && x >= cell0 && y >= cell0) v -= 1.0;
            } else if (x == y)
                v = x >= cell0 ? -1.0 : 1.0;  // l, or a filler with its section's sign
            else
                v = (closed && ((px == -2 && py >= 0 && y >= cell0) || (py == -2 && px >= 0 && x >= cell0))) ? 1.0 : 0.0;
            if (ap && v != 0.0) atomicExch(info, -1);
            put(i, j, r, 0, v);
        }
    }
    grid.sync();
    bool good = __ldcg(info) == 0;
    auto load = [&](double (&s)[B][B + 1], const double* tile) {  // false: all zero
        bool nz = false;
#pragma unroll
        for (int e = 0; e < EPT; e++) {
            const int r = r0 + e * RS;
            const double v = __ldcg(tile + r * B + c0);
            nz = nz || v != 0.0;
            s[r][c0] = v;
        }
        return __syncthreads_or(nz) != 0;
    };
    auto product = [&](const double (&x)[B][B + 1], const double (&y)[B][B + 1], int r) {  // row r of x y
        double acc = 0.0;
#pragma unroll
        for (int q = 0; q < B; q++) acc += x[r][q] * y[q][c0];
        return acc;
    };
    auto product_t = [&](const double (&x)[B][B + 1], const double (&y)[B][B + 1], int r) {  // row r of x^T y
        double acc = 0.0;
#pragma unroll
        for (int q = 0; q < B; q++) acc += x[q][r] * y[q][c0];
        return acc;
    };
    for (int k = 0; k < steps && good; k++) {
        const int np = pivots(k);
        const bool last = k == steps - 1;
        if (tid == 0) s_bad = 0;
        for (int q = 0; q < np; q++) load(sD[q], panel(k, q, pivot(k, q)));
        if (tid < 32 * np) {
            const bool ok = tile_inverse<B>(sD[tid / 32], sH[tid / 32], last, k < TF);
            if (!__all_sync(0xffffffffu, ok) && (tid & 31) == 0) atomicExch(&s_bad, 1);
        }
        __syncthreads();
        good = s_bad == 0;
        if (!good) break;
        // Newton steps X += X (I - M_pp X) bring it to FP64 (one, unless the tile is ill-conditioned):
        // the residual in FP64, the correction, at most 2^-20 of X, in FP32
        for (int q = 0; q < np && good; q++) {
            load(sA, panel(k, q, pivot(k, q)));
            bool rough = true;
            for (int it = 0; it < 3 && rough; it++) {
                bool big = false;
#pragma unroll
                for (int e = 0; e < EPT; e++) {
                    const int r = r0 + e * RS;
                    const float f = (float)((r == c0 ? 1.0 : 0.0) - product(sA, sD[q], r));
                    big = big || !(fabsf(f) < 1e-8f);
                    sF[r][c0] = f;
                }
                rough = __syncthreads_or(big) != 0;  // this step leaves the square of the residual
#pragma unroll
                for (int e = 0; e < EPT; e++) {
                    const int r = r0 + e * RS;
                    float f = 0.f;
#pragma unroll
                    for (int u = 0; u < B; u++) f = fmaf(sH[q][r][u], sF[u][c0], f);
                    sD[q][r][c0] += (double)f;
                }
                __syncthreads();
            }
            good = !rough;
        }
        if (!good) break;
        for (int item = blockIdx.x; item < T * np; item += gridDim.x) {
            const int j = item / np, q = item - j * np;
            if (pivot_of(k, j) >= 0 || apart(k, q, j)) continue;
            const bool nz = load(sA, panel(k, q, j));
#pragma unroll
            for (int e = 0; e < EPT; e++) {
                const int r = r0 + e * RS;
                epanel(q, j)[r * B + c0] = nz ? product(sD[q], sA, r) : 0.0;
            }
            __syncthreads();
        }
        grid.sync();
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            int i, j;
            tile_of(t, i, j);
            const int ip = pivot_of(k, i), jp = pivot_of(k, j);
            const bool keep = last || pivot_of(k + 1, i) >= 0 || pivot_of(k + 1, j) >= 0;  // written even when unchanged
            double v[EPT];
            bool changed = true;
            if (ip >= 0 && jp >= 0) {
#pragma unroll
                for (int e = 0; e < EPT; e++) v[e] = ip == jp ? sD[ip][r0 + e * RS][c0] : 0.0;
            } else if (ip >= 0) {
#pragma unroll
                for (int e = 0; e < EPT; e++) v[e] = apart(k, ip, j) ? 0.0 : __ldcg(epanel(ip, j) + (r0 + e * RS) * B + c0);
            } else if (jp >= 0) {
                const double sg = -sign(k, i);
                const bool nz = !apart(k, jp, i) && load(sA, panel(k, jp, i));
#pragma unroll
                for (int e = 0; e < EPT; e++) v[e] = nz ? sg * product_t(sA, sD[jp], r0 + e * RS) : 0.0;
            } else {
                changed = keep;
#pragma unroll
                for (int e = 0; e < EPT; e++) v[e] = __ldcg(M + (long long)(i * B + r0 + e * RS) * N + j * B + c0);
                const double sg = sign(k, i);
                for (int q = 0; q < np; q++) {
                    if (apart(k, q, i) || apart(k, q, j)) continue;
                    if (load(sA, panel(k, q, i)) && load(sE, epanel(q, j))) {
                        changed = true;
#pragma unroll
                        for (int e = 0; e < EPT; e++) v[e] -= sg * product_t(sA, sE, r0 + e * RS);
                    }
                    __syncthreads();
                }
            }
            if (changed) {
#pragma unroll
                for (int e = 0; e < EPT; e++) {
                    const int r = r0 + e * RS;
                    if (!last) {
                        put(i, j, r, k + 1, v[e]);
                        continue;
                    }
                    const int px = __ldg(perm + i * B + r), py = __ldg(perm + j * B + c0);
                    if (px >= 0 && py >= 0) {
                        a[(long long)px * 2 * nd + nd + py] = v[e];
                        if (i != j) a[(long long)py * 2 * nd + nd + px] = v[e];
                    }
                }
            }
            __syncthreads();
        }
        if (!last) grid.sync();
    }
    if (good) return;
    grid.sync();  // every block has left the workspace
    if (blockIdx.x == 0 && tid == 0) *info = 0;
    grid.sync();
    gj_all(nd, a, ws, info);
}

template <class V>
__device__ __forceinline__ double comp_value(const V* r, int s, int c);
template <>
__device__ __forceinline__ double comp_value<float4>(const float4* r, int s, int c) {
    return (double)reinterpret_cast<const float*>(r)[4ll * s + c];
}
template <>
__device__ __forceinline__ double comp_value<d4>(const d4* r, int s, int c) {
    return reinterpret_cast<const double*>(r)[4ll * s + c];
}

template <class V>
__global__ void k_gather(int nd, const int* __restrict__ slot_of, const int* __restrict__ comp_of, const V* __restrict__ r,
                         double* __restrict__ rd) {
    int q = blockIdx.x * TPB + threadIdx.x;
    if (q < nd) rd[q] = comp_value<V>(r, slot_of[q], comp_of[q]);
}

// one warp per row: x[row] = sum_c Ainv[row, c] rd[c], scattered into the slot vector
template <class T>
__global__ void k_gemv(int nd, const double* __restrict__ Ainv, int ld, const double* __restrict__ rd,
                       const int* __restrict__ slot_of, const int* __restrict__ comp_of, T* __restrict__ x) {
    int row = (blockIdx.x * TPB + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (row >= nd) return;
    double s = 0;
    for (int c = lane; c < nd; c += 32) s += Ainv[(long long)row * ld + c] * rd[c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[4ll * slot_of[row] + comp_of[row]] = (T)s;
}

}  // namespace

namespace {
__global__ void k_split_inverse(int nd, const double* __restrict__ inv, int ld, float2* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nd * nd) return;
    const double a = inv[(long long)(t / nd) * ld + t % nd];
    const float hi = (float)a;
    out[t] = make_float2(hi, (float)(a - (double)hi));
}
}  // namespace

int split_inverse(cudaStream_t st, int nd, const double* inv, int ld, float2* out) {
    k_split_inverse<<<(nd * nd + 255) / 256, 256, 0, st>>>(nd, inv, ld, out);
    STG_LAUNCH_CK();
    return STG_OK;
}

int dense_init(cudaStream_t st, DenseCoarse& D, const Geom& g) {
    std::vector<int> slot_of, comp_of, dense_of((size_t)g.nslot * 4, -1);
    const int n = g.n;
    for (int i = 0; i <= n; i++)
        for (int j = 0; j <= n; j++)
            for (int k = 0; k <= n; k++) {
                int s = g.slot(i, j, k);
                for (int c = 0; c < 4; c++) {
                    bool ok = c == 0 ? cell_ok(n, i, j, k) : face_ok(n, c - 1, i, j, k);
                    if (!ok) continue;
                    dense_of[4 * (size_t)s + c] = (int)slot_of.size();
                    slot_of.push_back(s);
                    comp_of.push_back(c);
                }
            }
    D.nd = (int)slot_of.size();
    size_t nd = D.nd;
    STG_CK(cudaMalloc(&D.slot_of, sizeof(int) * nd));
    STG_CK(cudaMalloc(&D.comp_of, sizeof(int) * nd));
    STG_CK(cudaMalloc(&D.dense_of, sizeof(int) * dense_of.size()));
    STG_CK(cudaMalloc(&D.A, sizeof(double) * 2 * nd * nd));
    STG_CK(cudaMalloc(&D.Ainv, sizeof(double) * 2 * nd * nd));
    if (n == 4) STG_CK(cudaMalloc(&D.inv2, sizeof(float2) * nd * nd));
    STG_CK(cudaMalloc(&D.piv, sizeof(int) * nd));
    STG_CK(cudaMalloc(&D.info, sizeof(int)));
    STG_CK(cudaMalloc(&D.probe, sizeof(d4) * g.nslot * PROBES));
    STG_CK(cudaMalloc(&D.image, sizeof(d4) * g.nslot * PROBES));
    STG_CK(cudaMalloc(&D.rd, sizeof(double) * nd));
    std::vector<std::vector<int>> faces(3);
    std::vector<int> cells;
    for (int q = 0; q < D.nd; q++) (comp_of[q] ? faces[comp_of[q] - 1] : cells).push_back(q);
    STG_TRY(inv_order(D.order, faces, cells));
    STG_CK(cudaMemcpy(D.slot_of, slot_of.data(), sizeof(int) * nd, cudaMemcpyHostToDevice));
    STG_CK(cudaMemcpy(D.comp_of, comp_of.data(), sizeof(int) * nd, cudaMemcpyHostToDevice));
    STG_CK(cudaMemcpy(D.dense_of, dense_of.data(), sizeof(int) * dense_of.size(), cudaMemcpyHostToDevice));
    STG_CK(cudaMemsetAsync(D.probe, 0, sizeof(d4) * g.nslot * PROBES, st));
    STG_CK(cudaMemsetAsync(D.image, 0, sizeof(d4) * g.nslot * PROBES, st));
    return STG_OK;
}

void dense_free(DenseCoarse& D) {
    cudaFree(D.slot_of);
    cudaFree(D.comp_of);
    cudaFree(D.dense_of);
    cudaFree(D.A);
    cudaFree(D.Ainv);
    cudaFree(D.inv2);
    cudaFree(D.piv);
    cudaFree(D.info);
    cudaFree(D.probe);
    cudaFree(D.image);
    cudaFree(D.rd);
    inv_order_free(D.order);
    D = DenseCoarse();
}

int op64v(cudaStream_t st, const Geom& g, const d4* x, const uint8_t* m, const d4* P, const d4* V, const d4* b, d4* out,
          int mode, double* part, int* nb_out);

int dense_setup_v(cudaStream_t st, DenseCoarse& D, const Geom& g, const d4* V, const uint8_t* m, const d4* P64, int closed,
                  const std::function<int(double*, int)>& extra) {
    const int nd = D.nd;
    k_aug_init<<<grid_for(2ll * nd * nd, TPB), TPB, 0, st>>>(nd, D.A);
    STG_LAUNCH_CK();
    for (int q = 0; q < PROBES; q++) {
        k_probe<<<grid_for(g.box(), TPB), TPB, 0, st>>>(g, q, D.probe);
        STG_LAUNCH_CK();
        STG_TRY(op64v(st, g, D.probe, m, P64, V, nullptr, D.image, 0, nullptr, nullptr));
        k_scatter<<<grid_for(nd, TPB), TPB, 0, st>>>(g, q, nd, D.slot_of, D.comp_of, D.dense_of, D.image, D.A);
        STG_LAUNCH_CK();
    }
    if (closed) {
        k_closed<<<grid_for((long long)nd * nd, TPB), TPB, 0, st>>>(nd, D.comp_of, D.A);
        STG_LAUNCH_CK();
    }
    if (extra) STG_TRY(extra(D.A, nd));
    return gj_invert(st, nd, D.A, D.Ainv, D.info, &D.inv, true);
}

int dense_setup(cudaStream_t st, DenseCoarse& D, const Geom& g, double vol, const uint8_t* m, const d4* P64, int closed,
                bool invert) {
    const int nd = D.nd;
    k_aug_init<<<grid_for(2ll * nd * nd, TPB), TPB, 0, st>>>(nd, D.A);
    STG_LAUNCH_CK();
    // all probes at once: three launches of a few us each, nine times three took 95 us of a set-up
    k_probe<<<dim3(grid_for(g.box(), TPB), PROBES), TPB, 0, st>>>(g, 0, D.probe);
    STG_LAUNCH_CK();
    STG_TRY(op64(st, g, vol, D.probe, m, P64, nullptr, D.image, 0, nullptr, nullptr, false, PROBES));
    k_scatter<<<dim3(grid_for(nd, TPB), PROBES), TPB, 0, st>>>(g, 0, nd, D.slot_of, D.comp_of, D.dense_of, D.image, D.A);
    STG_LAUNCH_CK();
    if (closed) {
        k_closed<<<grid_for((long long)nd * nd, TPB), TPB, 0, st>>>(nd, D.comp_of, D.A);
        STG_LAUNCH_CK();
    }
    return invert ? gj_invert(st, nd, D.A, D.Ainv, D.info, &D.inv) : STG_OK;
}

int gj_invert(cudaStream_t st, int nd, double* a, double* b, int* info, const double** inv, bool coop) {
    STG_CK(cudaMemsetAsync(info, 0, sizeof(int), st));
    if (coop) {
        // one block per SM at most (fewer blocks, a cheaper grid barrier), within what can
        // be co-resident
        int dev = 0, sms = 0, per_sm = 0;
        STG_CK(cudaGetDevice(&dev));
        STG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        STG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gj_all, TPB, 0));
        if (per_sm >= 1 && sms >= 1) {
            const int g = nd < sms ? nd : sms;
            void* args[] = {&nd, &a, &b, &info};
            STG_CK(cudaLaunchCooperativeKernel((const void*)k_gj_all, dim3((unsigned)g), dim3(TPB), args, 0, st));
            add_launches(1);
            *inv = (nd & 1) ? b + nd : a + nd;  // step nd-1 wrote buffer nd mod 2
            return STG_OK;
        }
    }
    for (int k = 0; k < nd; k++) {
        k_gj_step<<<nd, TPB, 0, st>>>(nd, k, a, b, info);
        STG_LAUNCH_CK();
        double* t = a;
        a = b;
        b = t;
    }
    *inv = a + nd;  // right half of the final buffer, row stride 2 nd
    return STG_OK;
}

// Elimination order of k_inv_blocks: every axis's faces padded to whole tiles, fillers, the
// cells and l at the end.
static int inv_tile(int nd) { return nd <= 512 ? 16 : 32; }

int inv_order(InvOrder& O, const std::vector<std::vector<int>>& faces, const std::vector<int>& cells) {
    int nd = (int)cells.size(), most = 0;
    for (auto& f : faces) {
        nd += (int)f.size();
        most = std::max(most, (int)f.size());
    }
    const int B = inv_tile(nd);
    O.S = (int)faces.size();
    O.TF = (most + B - 1) / B;
    std::vector<int> perm;
    for (int d = 0; d < O.S; d++) {
        perm.insert(perm.end(), faces[d].begin(), faces[d].end());
        perm.resize((size_t)(d + 1) * O.TF * B, -1);
    }
    const size_t c = (cells.size() + 1 + B - 1) / B * B;
    perm.resize(perm.size() + c - 1 - cells.size(), -1);
    perm.insert(perm.end(), cells.begin(), cells.end());
    perm.push_back(-2);
    O.N = (int)perm.size();
    STG_CK(cudaMalloc(&O.perm, sizeof(int) * O.N));
    STG_CK(cudaMemcpy(O.perm, perm.data(), sizeof(int) * O.N, cudaMemcpyHostToDevice));
    return STG_OK;
}

void inv_order_free(InvOrder& O) {
    cudaFree(O.perm);
    O = InvOrder();
}

int inv_blocks(cudaStream_t st, int nd, const InvOrder& O, int closed, double* a, double* b, int* info, const double** inv) {
    const int B = inv_tile(nd);
    int dev = 0, sms = 0, per_sm = 0, N = O.N, TF = O.TF;
    STG_CK(cudaGetDevice(&dev));
    STG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const void* fn = O.S == 3 ? (B == 16 ? (const void*)k_inv_blocks<16, 3> : (const void*)k_inv_blocks<32, 3>)
                              : (B == 16 ? (const void*)k_inv_blocks<16, 2> : (const void*)k_inv_blocks<32, 2>);
    const size_t smem = O.S == 3 ? (B == 16 ? InvShared<16, 3>::dynamic() : InvShared<32, 3>::dynamic())
                                 : (B == 16 ? InvShared<16, 2>::dynamic() : InvShared<32, 2>::dynamic());
    if (smem) STG_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    STG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TPB, smem));
    // the pivoted elimination leaves its result in the first buffer for an even nd (the cells
    // and padded faces of a grid whose size is a multiple of 4 are always even in number)
    const bool fits = (long long)N * N + 3ll * O.S * B * N <= 2ll * nd * nd && (nd & 1) == 0;
    if (!fits || per_sm < 1 || sms < 1 || O.S < 2 || O.S > 3) return gj_invert(st, nd, a, b, info, inv, true);
    STG_CK(cudaMemsetAsync(info, 0, sizeof(int), st));
    const int T = N / B, tiles = T * (T + 1) / 2, g = tiles < sms ? tiles : sms;
    const int* perm = O.perm;
    void* args[] = {&nd, &N, &TF, &perm, &closed, &a, &b, &info};
    STG_CK(cudaLaunchCooperativeKernel(fn, dim3((unsigned)g), dim3(TPB), args, smem, st));
    add_launches(1);
    *inv = a + nd;
    return STG_OK;
}

int dense_apply32(cudaStream_t st, const DenseCoarse& D, const Geom& g, const float4* r, float4* x) {
    double* rd = D.rd;
    k_gather<float4><<<grid_for(D.nd, TPB), TPB, 0, st>>>(D.nd, D.slot_of, D.comp_of, r, rd);
    STG_LAUNCH_CK();
    STG_CK(cudaMemsetAsync(x, 0, sizeof(float4) * g.nslot, st));
    k_gemv<float><<<grid_for(32ll * D.nd, TPB), TPB, 0, st>>>(D.nd, D.inv, 2 * D.nd, rd, D.slot_of, D.comp_of,
                                                              reinterpret_cast<float*>(x));
    STG_LAUNCH_CK();
    return STG_OK;
}

int dense_apply64(cudaStream_t st, const DenseCoarse& D, const Geom& g, const d4* r, d4* x) {
    double* rd = D.rd;
    k_gather<d4><<<grid_for(D.nd, TPB), TPB, 0, st>>>(D.nd, D.slot_of, D.comp_of, r, rd);
    STG_LAUNCH_CK();
    STG_CK(cudaMemsetAsync(x, 0, sizeof(d4) * g.nslot, st));
    k_gemv<double><<<grid_for(32ll * D.nd, TPB), TPB, 0, st>>>(D.nd, D.inv, 2 * D.nd, rd, D.slot_of, D.comp_of,
                                                                reinterpret_cast<double*>(x));
    STG_LAUNCH_CK();
    return STG_OK;
}

}  // namespace stg
