// Batched inverse of small dense matrices, one warp per matrix: FP64
// Gauss-Jordan in registers for n <= 48 (the stencil systems among them), FP64
// LU in shared memory for any other n <= 64, and FP32 inverse or factors with
// FP64 residual refinement.
//
// Replaces linalg::batched_matrix_inverse (linalg/batched_matrix_inverse.cuh:
// 325-397), which hands slices of the batch to cuBLAS getrfBatched +
// getriBatched on an executor thread per device (:121-282).
#include "warp_lu.cuh"
#include "scene_dev.hpp"

#include <algorithm>

namespace naga {

namespace {

size_t smem_limit() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v > 0 ? (size_t)v : 48 * 1024;
}

__global__ void inverse_f64_kernel(const double* __restrict__ A, double* __restrict__ Ainv, int n, int64_t batch,
                                   int* __restrict__ info, int warps_per_block) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    const size_t per_warp = (size_t)16 * n * n + 16 * ((n + 3) / 4);
    double* LU = reinterpret_cast<double*>(smem + per_warp * w);
    double* X = LU + n * n;
    int* piv = reinterpret_cast<int*>(X + n * n);
    const int64_t nw = (int64_t)gridDim.x * warps_per_block;
    for (int64_t b = (int64_t)blockIdx.x * warps_per_block + w; b < batch; b += nw) {
        const double* a = A + b * (int64_t)n * n;
        for (int e = lane; e < n * n; e += 32) LU[e] = a[e];
        __syncwarp();
        int inf = warp_lu(LU, n, piv);
        warp_lu_inverse(LU, n, piv, X);
        double* o = Ainv + b * (int64_t)n * n;
        for (int e = lane; e < n * n; e += 32) o[e] = X[(e % n) * n + e / n];
        if (info && lane == 0) info[b] = inf;
        __syncwarp();
    }
}

// Register-resident Gauss-Jordan inverse of systems of up to 48 rows (the
// stencil systems have n = k + D + 1: 19 / 20 for k = 16, 35 / 36 for k = 32).
// N is the size the registers are laid out for: the system's own (n = N), or
// with PAD the next of a few sizes. Lane l holds rows l and l + 32 in
// registers. Each elimination step publishes the pivot row in shared memory
// and every lane updates its rows from it, so the n^3 multiply-adds are
// independent register FMAs rather than a chain of shared-memory
// read-modify-writes.
//
// Pivoting is virtual: every row carries its getrf position (the row order
// after the swaps so far). The pivot of step k is the first row, in that
// order, of maximal |a| among positions k .. n - 1. That is getrf's choice, so
// the pivot sequence and info match the LU kernel. With B = P A the matrix in
// pivot order, the in-place sweep (pivot row scaled by p = 1 / a_kk, a_kk
// replaced by p; every other row i: a_ij -= a_ik a_kj, a_ik = -a_ik p) leaves
// row k of B^-1 in the row pivoted at step k. Since A^-1 = B^-1 P, the store
// un-permutes: A^-1(k, r_m) = B^-1(k, m), with r_m the row pivoted at step m.
//
// Register columns rotate by one each step: at step k register j holds column
// (k + j) mod N, so the pivot column is always register 0 and the new inverse
// column enters at register N - 1; after N steps the order is the identity
// again, after n steps column c is in register c + N - n. The step loop
// therefore indexes no register by k.
//
// PAD: n steps over n rows. The rows past n never leave position N, whatever
// the values (a NaN or an infinity that a pivot row holds reaches them), so no
// pivot and no store is ever one of theirs. The pivot row is published
// unscaled and the rows are scaled by their reciprocal pivots at the end: the
// multipliers a_ik p and the rows below the pivot are then the LU's own
// values, with its range (a pivot row scaled first overflows where the
// columns' scales differ by 1e155) and its exact zeros.
//
// Padded sizes against the LU in shared memory they had before: 100,000
// systems of 24 x 24 2.20 -> 0.61 ms; 20,000 of 9 x 9 0.092 -> 0.045 ms, of
// 33 x 33 2.02 -> 0.63, of 45 x 45 4.29 -> 0.84, of 48 x 48 5.75 -> 0.90; the
// errors on RBF systems of 24 to 45 rows agree to 1 % (median 7.4e-15 both at
// 24, 4.8e-13 at 45), info on singular integer matrices everywhere.
// Measured alternatives, all slower or equal (10^6 systems of 36 x 36 on
// B200, 18.6 ms for this form): per-row scales instead of rescaling the pivot
// row (19.6 ms), the next pivot searched while the current step's columns
// update (19.6-19.9 ms), a vote-and-shuffle fast path for a unique maximum
// (19.3 ms), the step loop fully unrolled without rotation (25.3 ms at 228
// registers), per-row scales with the next pivot searched beside the update
// (23 to 26 ms: 10 warps/SM, or spills at 12), the four rows past the lanes
// laid across the warp by column instead of as second rows (31 ms: fewer
// multiply-adds, twice the instructions around them).
constexpr int kGjWarps = 2;

template <int N, bool PAD>
__global__ void __launch_bounds__(32 * kGjWarps, (N > 36 ? 4 : N > 32 ? 5 : 8))
    inverse_gj_kernel(const double* __restrict__ A, double* __restrict__ Ainv, int n_, int64_t batch,
                      int* __restrict__ info) {
    constexpr int S = (N + 31) / 32;
    constexpr int NP = (N + 1) & ~1;
    static_assert(!PAD || N % 2 == 0, "a padded pivot row is published whole");
    const int n = PAD ? n_ : N;
    // per warp: the published pivot row (double-buffered by step parity) and
    // the physical row pivoted at each step
    __shared__ __align__(16) double prow[kGjWarps][2][NP];
    __shared__ int rowk[kGjWarps][N];
    const int w = threadIdx.x >> 5, lane = lane_id();
    const int64_t nw = (int64_t)gridDim.x * kGjWarps;
    for (int64_t b = (int64_t)blockIdx.x * kGjWarps + w; b < batch; b += nw) {
        const double* ai = A + b * (int64_t)(n * n);
        double a[S][N], scale[S];
        int pos[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int r = lane + 32 * s;
            pos[s] = r < n ? r : N;  // N marks a padding row
            scale[s] = 0.0;
#pragma unroll
            for (int c = 0; c < N; ++c) a[s][c] = r < n && c < n ? ai[r + n * c] : 0.0;
        }
        int inf = 0;
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            // pivot: max |a| over positions >= k, ties to the lowest position.
            // |a| >= 0, so its bits order like unsigned integers.
            unsigned hi = 0, lo = 0;
            int bp = N;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(a[s][0]));
                const unsigned h = (unsigned)(v >> 32), l = (unsigned)v;
                const bool better = h > hi || (h == hi && (l > lo || (l == lo && pos[s] < bp)));
                if (pos[s] >= k && pos[s] < N && better) {
                    hi = h;
                    lo = l;
                    bp = pos[s];
                }
            }
            const unsigned mh = __reduce_max_sync(kFull, hi);
            const unsigned ml = __reduce_max_sync(kFull, hi == mh ? lo : 0u);
            const int bpos = __reduce_min_sync(kFull, (hi == mh && lo == ml) ? bp : N);
            const bool zero = (mh | ml) == 0u;
            if (zero && !inf) inf = k + 1;
            bool piv[S];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                piv[s] = pos[s] == bpos;
                pos[s] = pos[s] == k ? bpos : (piv[s] ? k : pos[s]);
            }
            double* pr = prow[w][k & 1];
            double f[S], l[S];
            if constexpr (PAD) {
                // published rotated: pr[m] = a_r(m + 1), the pivot last
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (piv[s]) {
                        rowk[w][k] = lane + 32 * s;
#pragma unroll
                        for (int m = 0; m < N; m += 2)
                            *reinterpret_cast<double2*>(pr + m) = make_double2(a[s][m + 1], a[s][m + 2 < N ? m + 2 : 0]);
                    }
                __syncwarp();
                // f_i = a_ik p, the new column -f_i; the pivot row (f = 0)
                // takes 1 there. A zero pivot's reciprocal leaves NaN.
                const double p = 1.0 / pr[N - 1];
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    f[s] = piv[s] ? 0.0 : a[s][0] * p;
                    l[s] = piv[s] ? 1.0 : -f[s];
                    if (piv[s]) scale[s] = p;
                }
            } else {
                // the pivot row's owner scales it and publishes it rotated:
                // pr[m] = a_r(m + 1) p for m < N - 1, pr[N - 1] = p
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (piv[s]) {
                        rowk[w][k] = lane + 32 * s;
                        const double p = zero ? 0.0 : 1.0 / a[s][0];
                        a[s][0] = p;
#pragma unroll
                        for (int j = 1; j < N; ++j) a[s][j] *= p;
#pragma unroll
                        for (int m = 0; m + 1 < N; m += 2)
                            *reinterpret_cast<double2*>(pr + m) = make_double2(a[s][m + 1], m + 2 < N ? a[s][m + 2] : p);
                        if (N & 1) pr[N - 1] = p;
                    }
                __syncwarp();
                // the new column -f_i p; the pivot row (f = 0) only rotates,
                // keeping p
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    f[s] = piv[s] ? 0.0 : a[s][0];
                    l[s] = piv[s] ? a[s][0] : 0.0;
                }
            }
            // every row: a_i(m) = a_i(m + 1) - f_i pr[m] (rotated)
#pragma unroll
            for (int m = 0; m < N; m += 2) {
                const double2 q = *reinterpret_cast<const double2*>(pr + m);
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    a[s][m] = fma(-f[s], q.x, m + 1 < N ? a[s][m + 1] : l[s]);
                    if (PAD && m + 1 == N - 1)
                        a[s][m + 1] = l[s];
                    else if (m + 1 < N)
                        a[s][m + 1] = fma(-f[s], q.y, m + 2 < N ? a[s][m + 2] : l[s]);
                }
            }
        }
        __syncwarp();
        double* o = Ainv + b * (int64_t)(n * n);
        const int c0 = N - n;  // register of column 0
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < n)
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (j >= c0) o[pos[s] + n * rowk[w][j - c0]] = PAD ? a[s][j] * scale[s] : a[s][j];
        if (info && lane == 0) info[b] = inf;
        __syncwarp();
    }
}

// FP32 inverse of one system by Gauss-Jordan in registers, rows lane and
// lane + 32 of the warp; the scheme of inverse_gj_kernel with the pivot row
// published as it is and scaled at the end. Af: the FP64 system, column-major with
// stride NP, identity past n; out: its inverse, column-major, stride NP.
// prow: NP floats twice; rowk: NP ints. Returns getrf's info.
template <int NP>
__device__ int warp_inverse_f32(const double* Af, int n, float* out, float* prow, int* rowk) {
    constexpr int S = (NP + 31) / 32;
    const int lane = lane_id();
    float a[S][NP], scale[S];
    int pos[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int r = lane + 32 * s;
        pos[s] = r < NP ? r : NP;
        scale[s] = 1.f;
#pragma unroll
        for (int c = 0; c < NP; ++c) a[s][c] = r < NP ? (float)Af[r + NP * c] : 0.f;
    }
    int inf = 0;
#pragma unroll 1
    for (int k = 0; k < NP; ++k) {
        unsigned h = 0u;
        int bp = NP;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned v = __float_as_uint(a[s][0]) & 0x7fffffffu;
            if (pos[s] >= k && pos[s] < NP && (v > h || (v == h && pos[s] < bp))) {
                h = v;
                bp = pos[s];
            }
        }
        const unsigned m = __reduce_max_sync(kFull, h);
        const int bpos = __reduce_min_sync(kFull, h == m ? bp : NP);
        const bool zero = m == 0u;
        if (zero && !inf) inf = k + 1;
        float* const pr = prow + (k & 1) * NP;
        bool piv[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            piv[s] = pos[s] == bpos;
            pos[s] = pos[s] == k ? bpos : (piv[s] ? k : pos[s]);
            if (piv[s]) {
                rowk[k] = lane + 32 * s;
#pragma unroll
                for (int c = 0; c < NP; c += 4)
                    *reinterpret_cast<float4*>(pr + c) = make_float4(a[s][c], a[s][c + 1], a[s][c + 2], a[s][c + 3]);
            }
        }
        __syncwarp();
        const float inv = zero ? 0.f : 1.f / pr[0];
        float f[S], last[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            f[s] = piv[s] ? 0.f : -(a[s][0] * inv);
            last[s] = piv[s] ? 1.f : f[s];
            if (piv[s]) scale[s] = inv;
        }
#pragma unroll
        for (int c = 0; c < NP; c += 4) {
            const float4 q = *reinterpret_cast<const float4*>(pr + c);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (c > 0) a[s][c > 0 ? c - 1 : 0] = fmaf(f[s], q.x, a[s][c]);
                a[s][c] = fmaf(f[s], q.y, a[s][c + 1]);
                a[s][c + 1] = fmaf(f[s], q.z, a[s][c + 2]);
                a[s][c + 2] = fmaf(f[s], q.w, a[s][c + 3]);
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) a[s][NP - 1] = last[s];
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < NP)
#pragma unroll
            for (int c = 0; c < NP; ++c) out[pos[s] + NP * rowk[c]] = a[s][c] * scale[s];
    __syncwarp();
    return inf > n ? 0 : inf;
}

// FP32 LU of one system with getrf's pivoting, rows lane and lane + 32 of the
// warp in registers; virtual pivoting and rotating columns as in
// inverse_gj_kernel, the operations and their order those of warp_lu. Ad: the
// FP64 system, column-major with stride NP; LU: its factors, the same layout,
// rows in pivot order; rowk[i]: the row pivoted at step i; mult: NP x NP floats
// for the multipliers by row as they arise (zeros stand in their place in the
// registers, so the update passes over the eliminated columns); prow: NP
// floats twice. Returns getrf's info; a zero pivot's column is left unreduced.
template <int NP>
__device__ int warp_lu_f32(const double* Ad, int n, float* LU, float* mult, float* prow, int* rowk) {
    constexpr int S = (NP + 31) / 32;
    const int lane = lane_id();
    float a[S][NP];
    int pos[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int r = lane + 32 * s;
        pos[s] = r < n ? r : NP;  // NP: no row of the system, never a pivot
#pragma unroll
        for (int c = 0; c < NP; ++c) a[s][c] = r < n ? (float)Ad[r + NP * c] : 0.f;
    }
    int inf = 0;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        unsigned h = 0u;
        int bp = NP;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned v = __float_as_uint(a[s][0]) & 0x7fffffffu;
            if (pos[s] >= k && pos[s] < NP && (v > h || (v == h && pos[s] < bp))) {
                h = v;
                bp = pos[s];
            }
        }
        const unsigned m = __reduce_max_sync(kFull, h);
        const int bpos = __reduce_min_sync(kFull, h == m ? bp : NP);
        const bool zero = m == 0u;
        if (zero && !inf) inf = k + 1;
        float* const pr = prow + (k & 1) * NP;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const bool piv = pos[s] == bpos;
            pos[s] = pos[s] == k ? bpos : (piv ? k : pos[s]);
            if (piv) {
                rowk[k] = lane + 32 * s;
#pragma unroll
                for (int c = 0; c < NP; c += 4)
                    *reinterpret_cast<float4*>(pr + c) = make_float4(a[s][c], a[s][c + 1], a[s][c + 2], a[s][c + 3]);
            }
        }
        __syncwarp();
        const float inv = 1.f / pr[0];
        float l[S], last[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const bool below = pos[s] > k && !zero;
            l[s] = below ? a[s][0] * inv : 0.f;
            last[s] = pos[s] > k ? 0.f : a[s][0];
            if (lane + 32 * s < n) mult[lane + 32 * s + NP * k] = l[s];
        }
#pragma unroll
        for (int c = 0; c < NP; c += 4) {
            const float4 q = *reinterpret_cast<const float4*>(pr + c);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (c > 0) a[s][c > 0 ? c - 1 : 0] = fmaf(-l[s], q.x, a[s][c]);
                a[s][c] = fmaf(-l[s], q.y, a[s][c + 1]);
                a[s][c + 1] = fmaf(-l[s], q.z, a[s][c + 2]);
                a[s][c + 2] = fmaf(-l[s], q.w, a[s][c + 3]);
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) a[s][NP - 1] = last[s];
    }
    __syncwarp();
    const int c0 = NP - n;  // register of column 0
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < n)
#pragma unroll
            for (int c = 0; c < NP; ++c)
                if (c >= c0)
                    LU[pos[s] + NP * (c - c0)] = c - c0 < pos[s] ? mult[lane + 32 * s + NP * (c - c0)] : a[s][c];
    __syncwarp();
    return inf;
}

// A column's refinement: last correction, the one before, and whether it is
// done -- below the tolerance, no longer contracting, or not finite
struct RefineState {
    double dlast = INFINITY, dprev = INFINITY, xlast = 0;
    bool done, lost = false, slow = false;
    __device__ explicit RefineState(bool idle) : done(idle) {}
    // dm, xm: largest correction and entry (NaN not among them); finite:
    // whether every correction is
    __device__ void update(float dm, double xm, bool finite, double tol) {
        dprev = dlast;
        dlast = (double)dm;
        xlast = xm;
        lost = !finite || !(xm < INFINITY);
        done = lost || dlast <= tol * xm || dlast > 0.5 * dprev;
        slow = slow || (dlast > dprev / 256 && dlast > 1e-10 * xm);
    }
    // last correction within the tolerance, or within 1e-10 of the column
    // when refinement stagnated at the FP64 residual floor
    __device__ bool converged(double tol) const { return !lost && (dlast <= tol * xlast || dlast <= 1e-10 * xlast); }
};

// FP64 residual refinement of every column of the inverse of one system, one
// column a lane, 32 columns at a time. The column's residual and correction
// stay in registers; A, the FP32 matrix M and the column's own entries come
// from shared memory, A and M as broadcasts shared by the warp's columns.
// FACTORS: M holds the factors of warp_lu_f32 and its corrections solve with
// them (one straight run of code a column); X starts from 0. Otherwise M is the
// FP32 inverse, X starts from it and a correction is its product with the
// residual. True when every column of the lane converged -- with the inverse,
// at 256 times a step down to 1e-10 of the column.
template <int NP, bool FACTORS>
__device__ bool refine(const double* Ad, const float* M, const int* rowk, double* X, float* R, int n, int max_iter,
                       double tol) {
    const int lane = lane_id();
    bool conv = true;
    // columns 0 .. 31, one a lane
    {
        const int c = lane;
        const bool has = c < n;
        const int cc = has ? c : 0;  // idle lanes read column 0
        if (!FACTORS && has)
            for (int j = 0; j < NP; ++j) X[j * NP + c] = (double)M[j + NP * c];
        RefineState st(!has);
        for (int it = FACTORS ? -1 : 0; it < 0 || (it < max_iter && !__all_sync(kFull, st.done)); ++it) {
            // residual R = I - A X, to FP32
            double r[NP];
#pragma unroll
            for (int i = 0; i < NP; ++i) r[i] = i == c ? 1.0 : 0.0;
            if (it >= 0) {
#pragma unroll 2
                for (int j = 0; j < n; ++j) {
                    const double xj = -X[j * NP + cc];
                    const double2* col = reinterpret_cast<const double2*>(Ad + NP * j);
#pragma unroll
                    for (int i = 0; i < NP; i += 2) {
                        const double2 v = col[i / 2];
                        r[i] = fma(v.x, xj, r[i]);
                        r[i + 1] = fma(v.y, xj, r[i + 1]);
                    }
                }
            }
            if (has) {
#pragma unroll
                for (int i = 0; i < NP; ++i) R[i * NP + c] = (float)r[i];
            }
            __syncwarp();
            // correction D
            float d[NP];
            if constexpr (FACTORS) {
#pragma unroll
                for (int i = 0; i < NP; ++i) d[i] = i < n ? R[rowk[i] * NP + cc] : 0.f;
#pragma unroll
                for (int j = 0; j < NP; ++j)
                    if (j < n) {
                        const float4* col = reinterpret_cast<const float4*>(M + NP * j);
#pragma unroll
                        for (int i = (j + 1) / 4 * 4; i < NP; i += 4) {
                            const float4 v = col[i / 4];
                            if (i > j) d[i] = fmaf(-v.x, d[j], d[i]);
                            if (i + 1 > j) d[i + 1] = fmaf(-v.y, d[j], d[i + 1]);
                            if (i + 2 > j) d[i + 2] = fmaf(-v.z, d[j], d[i + 2]);
                            if (i + 3 > j) d[i + 3] = fmaf(-v.w, d[j], d[i + 3]);
                        }
                    }
#pragma unroll
                for (int j = NP - 1; j >= 0; --j)
                    if (j < n) {
                        const float4* col = reinterpret_cast<const float4*>(M + NP * j);
                        d[j] = d[j] / M[j + NP * j];
#pragma unroll
                        for (int i = 0; i < j; i += 4) {
                            const float4 v = col[i / 4];
                            d[i] = fmaf(-v.x, d[j], d[i]);
                            if (i + 1 < j) d[i + 1] = fmaf(-v.y, d[j], d[i + 1]);
                            if (i + 2 < j) d[i + 2] = fmaf(-v.z, d[j], d[i + 2]);
                            if (i + 3 < j) d[i + 3] = fmaf(-v.w, d[j], d[i + 3]);
                        }
                    }
            } else {
#pragma unroll
                for (int i = 0; i < NP; ++i) d[i] = 0.f;
#pragma unroll 2
                for (int j = 0; j < n; ++j) {
                    const float rj = R[j * NP + cc];
                    const float4* col = reinterpret_cast<const float4*>(M + NP * j);
#pragma unroll
                    for (int i = 0; i < NP; i += 4) {
                        const float4 v = col[i / 4];
                        d[i] = fmaf(v.x, rj, d[i]);
                        d[i + 1] = fmaf(v.y, rj, d[i + 1]);
                        d[i + 2] = fmaf(v.z, rj, d[i + 2]);
                        d[i + 3] = fmaf(v.w, rj, d[i + 3]);
                    }
                }
            }
            // X += D
            if (it < 0) {
                if (has) {
#pragma unroll
                    for (int i = 0; i < NP; ++i) X[i * NP + c] = (double)d[i];
                }
            } else if (!st.done) {
                float dm = 0.f, nil = 0.f;  // nil: NaN with any infinite or NaN correction
                double xm = 0;
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const double x = X[i * NP + c] + (double)d[i];
                    X[i * NP + c] = x;
                    if (i < n) {
                        dm = fmaxf(dm, fabsf(d[i]));
                        xm = fmax(xm, fabs(x));
                        nil = fmaf(d[i], 0.f, nil);
                    }
                }
                st.update(dm, xm, nil == 0.f, tol);
            }
            __syncwarp();
        }
        if (has) conv = st.converged(tol) && (FACTORS || !st.slow);
    }
    // columns 32 .. n - 1, C at a time, 32 / C lanes a column: lane l takes
    // rows (l / C) RL .. of column c0 + l % C, so the few columns past the
    // lanes do not cost another full pass
    constexpr int C = 4, RL = (NP + 32 / C - 1) / (32 / C);
    for (int c0 = 32; c0 < n; c0 += C) {
        const int c = c0 + lane % C, i0 = lane / C * RL;
        const bool has = c < n;
        const int cc = has ? c : c0;
        int row[RL];
#pragma unroll
        for (int u = 0; u < RL; ++u) row[u] = i0 + u < NP ? i0 + u : NP - 1;
        if (!FACTORS && has)
            for (int u = 0; u < RL; ++u)
                if (i0 + u < NP) X[(i0 + u) * NP + c] = (double)M[i0 + u + NP * c];
        __syncwarp();
        RefineState st(!has);
        for (int it = FACTORS ? -1 : 0; it < 0 || (it < max_iter && !__all_sync(kFull, st.done)); ++it) {
            double r[RL];
            float d[RL];
#pragma unroll
            for (int u = 0; u < RL; ++u) r[u] = row[u] == c ? 1.0 : 0.0;
            if (it >= 0) {
#pragma unroll 4
                for (int j = 0; j < n; ++j) {
                    const double xj = -X[j * NP + cc];
#pragma unroll
                    for (int u = 0; u < RL; ++u) r[u] = fma(Ad[row[u] + NP * j], xj, r[u]);
                }
            }
            __syncwarp();
            if (has) {
#pragma unroll
                for (int u = 0; u < RL; ++u)
                    if (i0 + u < NP) R[row[u] * NP + c] = (float)r[u];
            }
            __syncwarp();
            if constexpr (FACTORS) {
                // x_j goes from its lane to the column's other lanes
#pragma unroll
                for (int u = 0; u < RL; ++u) d[u] = row[u] < n ? R[rowk[row[u]] * NP + cc] : 0.f;
#pragma unroll 1
                for (int o = 0; o < 32 / C; ++o)
#pragma unroll
                    for (int u = 0; u < RL; ++u) {
                        const int j = o * RL + u;
                        if (j >= n) continue;
                        const float xj = __shfl_sync(kFull, d[u], o * C + lane % C);
#pragma unroll
                        for (int v = 0; v < RL; ++v)
                            if (row[v] > j) d[v] = fmaf(-M[row[v] + NP * j], xj, d[v]);
                    }
#pragma unroll 1
                for (int o = 32 / C - 1; o >= 0; --o)
#pragma unroll
                    for (int u = RL - 1; u >= 0; --u) {
                        const int j = o * RL + u;
                        if (j >= n) continue;
                        const float xj = __shfl_sync(kFull, d[u], o * C + lane % C) / M[j + NP * j];
                        if (lane / C == o) d[u] = xj;
#pragma unroll
                        for (int v = 0; v < RL; ++v)
                            if (row[v] < j) d[v] = fmaf(-M[row[v] + NP * j], xj, d[v]);
                    }
            } else {
#pragma unroll
                for (int u = 0; u < RL; ++u) d[u] = 0.f;
#pragma unroll 4
                for (int j = 0; j < n; ++j) {
                    const float rj = R[j * NP + cc];
#pragma unroll
                    for (int u = 0; u < RL; ++u) d[u] = fmaf(M[row[u] + NP * j], rj, d[u]);
                }
            }
            float dm = 0.f, nil = 0.f;
            double xm = 0;
#pragma unroll
            for (int u = 0; u < RL; ++u)
                if (!st.done && i0 + u < n) {
                    const double x = (it < 0 ? 0.0 : X[row[u] * NP + c]) + (double)d[u];
                    X[row[u] * NP + c] = x;
                    dm = fmaxf(dm, fabsf(d[u]));
                    xm = fmax(xm, fabs(x));
                    nil = fmaf(d[u], 0.f, nil);
                }
#pragma unroll
            for (int o = C; o < 32; o <<= 1) {
                dm = fmaxf(dm, __shfl_xor_sync(kFull, dm, o));
                xm = fmax(xm, __shfl_xor_sync(kFull, xm, o));
                nil += __shfl_xor_sync(kFull, nil, o);
            }
            if (it >= 0 && !st.done) st.update(dm, xm, nil == 0.f, tol);
            __syncwarp();
        }
        if (has) conv = conv && st.converged(tol) && (FACTORS || !st.slow);
    }
    __syncwarp();
    return conv;
}

template <int NP>
struct RefineSize {
    static_assert(NP % 4 == 0, "16-B columns");
    // A, X (FP64), M, R (FP32), the published rows and their order
    static constexpr size_t per_warp = (size_t)NP * NP * (8 + 8 + 4 + 4) + NP * (8 + 4) + 32;
    static constexpr size_t stride = (per_warp + 127) / 128 * 128;
};

// Refinement with the factors, for the systems the inverse does not serve.
// Returns getrf's info, -1 when some column did not converge.
template <int NP>
__device__ __forceinline__ int refine_with_factors(const double* Ad, float* LU, double* X, float* R, float* prow, int* rowk,
                                                int n, int max_iter, double tol) {
    for (int e = lane_id(); e < NP * NP; e += 32) LU[e] = 0.f;
    __syncwarp();
    const int inf = warp_lu_f32<NP>(Ad, n, LU, R, prow, rowk);
    const bool conv = refine<NP, true>(Ad, LU, rowk, X, R, n, inf ? 0 : max_iter, tol);
    return inf ? inf : (__all_sync(kFull, conv) ? 0 : -1);
}

template <int NP>
__device__ __noinline__ int refine_with_factors_call(const double* Ad, float* LU, double* X, float* R, float* prow,
                                                     int* rowk, int n, int max_iter, double tol) {
    return refine_with_factors<NP>(Ad, LU, X, R, prow, rowk, n, max_iter, tol);
}

// FP32 inverse or factors, FP64 residual refinement of every column of the
// inverse. Most systems take the FP32 inverse: a correction is then one product
// of independent multiply-adds. At the limit of what the refinement reaches
// the inverse and the factors fail on different systems, about as often (of
// 2000 systems of 2-D stencils with 32 supports, 50 and 41), so a system whose
// corrections do not shrink 256 times a step is done again by solves with the
// factors throughout, and the systems refused are those that these do not
// reach: the same, over 30,000 systems of condition 1e6 and up, as with the
// factors alone. (A bound of 16 reaches 3 to 70 % of those too, some with 1.6
// times the error; 1024 sends random systems of 36 rows to the factors, 1.45 ->
// 1.60 ms.)
// Against triangular solves and residuals read and written in shared memory,
// one dependent chain a lane: 20,000 systems of 36 x 36 9.70 -> 1.26 ms, of 20
// x 20 1.08 -> 0.26; 5,000 of 45 x 45 8.1 -> 0.92, of 49 x 49 10.1 -> 2.5;
// 3,000 of 64 x 64 18.0 -> 2.3 (solves with the factors for all of them:
// 36 x 36 1.98, 45 x 45 2.5, 64 x 64 7.7). Bound by the latency of the
// shared-memory operands: 7 warps/SM (31 KB a system), a third of the issue
// slots. Up to 20 rows one warp a block: at 128 registers 14 fit an SM, and
// small batches spread evenly (7 warps a block 0.28, 4 0.28 ms of 20 x 20).
// Up to 8 and 4 rows registers of their own, or the smallest systems would be
// slower than by a chain a lane: 20,000 of 2 x 2 0.047 (by chains) and 0.129
// (padded to 20) -> 0.032 ms, of 8 x 8 0.22 and 0.18 -> 0.073.
template <int NP>
__global__ void __launch_bounds__(NP > 36 ? 128 : NP > 20 ? 224 : 32, NP > 20 ? 1 : NP > 8 ? 14 : 24)
    inverse_f32r_kernel(const double* __restrict__ A, double* __restrict__ Ainv, int n, int64_t batch, int max_iter,
                        double tol, int* __restrict__ info, int warps_per_block) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    double* Ad = reinterpret_cast<double*>(smem + RefineSize<NP>::stride * w);
    double* X = Ad + NP * NP;  // X[j NP + c]: row j of column c
    float* M = reinterpret_cast<float*>(X + NP * NP);
    float* R = M + NP * NP;    // as X
    float* prow = R + NP * NP;
    int* rowk = reinterpret_cast<int*>(prow + 2 * NP);
    const int64_t nw = (int64_t)gridDim.x * warps_per_block;
    for (int64_t b = (int64_t)blockIdx.x * warps_per_block + w; b < batch; b += nw) {
        const double* a = A + b * (int64_t)n * n;
        for (int e = lane; e < NP * NP; e += 32) {
            const int r = e % NP, c = e / NP;
            Ad[e] = r < n && c < n ? a[r + (int64_t)n * c] : (r == c ? 1.0 : 0.0);
        }
        __syncwarp();
        int inf = warp_inverse_f32<NP>(Ad, n, M, prow, rowk);
        if (inf || !__all_sync(kFull, refine<NP, false>(Ad, M, rowk, X, R, n, max_iter, tol)))
            // inlined where that keeps the path above from spilling around
            // the call (5,000 of 45 x 45 0.96 -> 0.91 ms; 64 x 64 2.31 -> 2.39)
            inf = NP == 48 ? refine_with_factors<NP>(Ad, M, X, R, prow, rowk, n, max_iter, tol)
                           : refine_with_factors_call<NP>(Ad, M, X, R, prow, rowk, n, max_iter, tol);
        double* o = Ainv + b * (int64_t)n * n;
        for (int e = lane; e < n * n; e += 32) o[e] = X[(e % n) * NP + e / n];
        if (info && lane == 0) info[b] = inf;
        __syncwarp();
    }
}

template <int NP>
int launch_f32r(const double* A, double* Ainv, int n, int64_t batch, int max_iter, double tol, int* info,
                cudaStream_t st) {
    const size_t stride = RefineSize<NP>::stride;
    const int wpb = (int)std::min<size_t>(NP > 36 ? 4 : NP > 20 ? 7 : 1, smem_limit() / stride);
    if (wpb < 1) return set_error(NAGA_EINVAL, "batched inverse: matrix too large for shared memory");
    const size_t smem = stride * wpb;
    NAGA_CUDA_TRY(cudaFuncSetAttribute(inverse_f32r_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = (int)std::min<int64_t>((batch + wpb - 1) / wpb, (int64_t)sm_count() * 32);
    inverse_f32r_kernel<NP><<<blocks, 32 * wpb, smem, st>>>(A, Ainv, n, batch, max_iter, tol, info, wpb);
    NAGA_CUDA_TRY(cudaGetLastError());
    return NAGA_OK;
}

template <int N, bool PAD>
int launch_gj(const double* A, double* Ainv, int n, int64_t batch, int* info, cudaStream_t st) {
    static int per_sm = 0;
    auto kern = inverse_gj_kernel<N, PAD>;
    if (per_sm < 1) {
        NAGA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kGjWarps, 0));
        per_sm = std::max(per_sm, 1);
    }
    const int64_t need = (batch + kGjWarps - 1) / kGjWarps;
    const int blocks = (int)std::min<int64_t>(need, (int64_t)sm_count() * per_sm);
    kern<<<blocks, 32 * kGjWarps, 0, st>>>(A, Ainv, n, batch, info);
    NAGA_CUDA_TRY(cudaGetLastError());
    return NAGA_OK;
}

}  // namespace

int batched_inverse(const double* A, double* Ainv, int n, int64_t batch, int* info, bool refined, int max_iter,
                    double tol, cudaStream_t st) {
    if (n < 1 || n > 64) return set_error(NAGA_EINVAL, "batched inverse: n must be in [1, 64]");
    if (batch < 0) return set_error(NAGA_EINVAL, "batched inverse: negative batch");
    if (batch == 0) return NAGA_OK;
    if (!A || !Ainv) return set_error(NAGA_EINVAL, "batched inverse: null pointer");
    // up to 48 rows in registers: the stencil systems at their own size, the
    // others rounded up to the next of a few; larger ones by LU in shared
    // memory
    if (!refined && n <= 48) {
        switch (n) {
            case 19: return launch_gj<19, false>(A, Ainv, n, batch, info, st);
            case 20: return launch_gj<20, false>(A, Ainv, n, batch, info, st);
            case 35: return launch_gj<35, false>(A, Ainv, n, batch, info, st);
            case 36: return launch_gj<36, false>(A, Ainv, n, batch, info, st);
            default: break;
        }
        if (n <= 8) return launch_gj<8, true>(A, Ainv, n, batch, info, st);
        if (n <= 16) return launch_gj<16, true>(A, Ainv, n, batch, info, st);
        if (n <= 24) return launch_gj<24, true>(A, Ainv, n, batch, info, st);
        if (n <= 32) return launch_gj<32, true>(A, Ainv, n, batch, info, st);
        return launch_gj<48, true>(A, Ainv, n, batch, info, st);
    }
    if (refined) {
        if (n <= 4) return launch_f32r<4>(A, Ainv, n, batch, max_iter, tol, info, st);
        if (n <= 8) return launch_f32r<8>(A, Ainv, n, batch, max_iter, tol, info, st);
        if (n <= 20) return launch_f32r<20>(A, Ainv, n, batch, max_iter, tol, info, st);
        if (n <= 28) return launch_f32r<28>(A, Ainv, n, batch, max_iter, tol, info, st);
        if (n <= 36) return launch_f32r<36>(A, Ainv, n, batch, max_iter, tol, info, st);
        if (n <= 48) return launch_f32r<48>(A, Ainv, n, batch, max_iter, tol, info, st);
        return launch_f32r<64>(A, Ainv, n, batch, max_iter, tol, info, st);
    }
    const size_t per_warp = (size_t)16 * n * n + 16 * ((n + 3) / 4);
    const int wpb = (int)std::min<size_t>(8, smem_limit() / per_warp);
    if (wpb < 1) return set_error(NAGA_EINVAL, "batched inverse: matrix too large for shared memory");
    const size_t smem = per_warp * wpb;
    const int64_t blocks_needed = (batch + wpb - 1) / wpb;
    const int blocks = (int)std::min<int64_t>(blocks_needed, (int64_t)sm_count() * 32);
    NAGA_CUDA_TRY(cudaFuncSetAttribute(inverse_f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    inverse_f64_kernel<<<blocks, 32 * wpb, smem, st>>>(A, Ainv, n, batch, info, wpb);
    NAGA_CUDA_TRY(cudaGetLastError());
    return NAGA_OK;
}

}  // namespace naga

extern "C" int naga_batched_inverse_f64(const double* A, double* A_inv, int n, int64_t batch, int* info,
                                        void* stream) {
    return naga::batched_inverse(A, A_inv, n, batch, info, false, 0, 0.0, (cudaStream_t)stream);
}

extern "C" int naga_batched_inverse_f32r(const double* A, double* A_inv, int n, int64_t batch, int max_iter,
                                         double rel_tol, int* info, void* stream) {
    if (max_iter < 0 || !(rel_tol >= 0)) return naga::set_error(NAGA_EINVAL, "naga_batched_inverse_f32r: bad tolerance");
    return naga::batched_inverse(A, A_inv, n, batch, info, true, max_iter, rel_tol, (cudaStream_t)stream);
}
