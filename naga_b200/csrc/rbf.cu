// Radial-point-interpolation weights and the nonlocal divergence stencil,
// built on the GPU in FP64 (or FP32 LU + FP64-residual refinement).
//
// NAGA builds the augmented moment matrix G0 = [[Phi, P], [P^T, 0]] per
// support set, inverts it with cuBLAS and contracts the inverse with G_x
// (interpolation/detail/radial_point_method.cuh:349-453). Here one warp
// owns one support set: it assembles G0 in shared memory, factors it with
// partial pivoting and solves for the right-hand sides directly (the
// contraction W = G0^-T G_x equals G0^-1 G_x because G0 is symmetric).
//
// Coordinates are shifted to the group's centre and divided by the spacing
// parameter before assembly. Both shape functions are radial, so this
// leaves the interpolation weights unchanged in exact arithmetic (the RBF
// block scales by a constant and span{1, x} is shift- and scale-invariant)
// while it removes most of the ill-conditioning of the absolute-coordinate
// system.
#include "warp_gj.cuh"
#include "warp_lu.cuh"
#include "scene_dev.hpp"
#include "scratch.hpp"

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

namespace naga {

// systems whose FP32 refinement failed in the last refined call (per thread)
static thread_local int64_t g_fallbacks = 0;

namespace {

// multiquadric (r^2 + (0.1 h)^2)^0.5 in units of h (radial_point_method.cuh:
// 44-66 with q = 0.5, alpha_c = 0.1), or the cubic polyharmonic spline r^3
__device__ __forceinline__ double shape_fn(double r2, int shape) {
    if (shape == 0) return sqrt(r2 + 0.01);
    double r = sqrt(r2);
    return r * r * r;
}

template <int D>
__device__ void build_G0(const double* xs, int k, int shape, double* G) {
    const int n = k + D + 1;
    for (int e = lane_id(); e < n * n; e += 32) {
        const int i = e % n, j = e / n;
        double v;
        if (i >= k && j >= k)
            v = 0.0;
        else if (i >= k)
            v = (i == k) ? 1.0 : xs[j * D + (i - k - 1)];
        else if (j >= k)
            v = (j == k) ? 1.0 : xs[i * D + (j - k - 1)];
        else {
            double r2 = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                double t = xs[i * D + d] - xs[j * D + d];
                r2 += t * t;
            }
            v = shape_fn(r2, shape);
        }
        G[e] = v;
    }
    __syncwarp();
}

// G_x row r for the scaled query point x
template <int D>
__device__ __forceinline__ double gx_row(const double* xs, int k, int shape, const double* x, int r) {
    if (r < k) {
        double r2 = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            double t = xs[r * D + d] - x[d];
            r2 += t * t;
        }
        return shape_fn(r2, shape);
    }
    if (r == k) return 1.0;
    return x[r - k - 1];
}

// y = A x for x distributed over the warp (rows r = lane, lane + 32)
__device__ void warp_matvec(const double* A, int n, double x0, double x1, double& y0, double& y1) {
    const int lane = lane_id();
    y0 = 0;
    y1 = 0;
    for (int j = 0; j < n; ++j) {
        double xj = warp_get(x0, x1, j);
        if (lane < n) y0 += A[lane + n * j] * xj;
        if (lane + 32 < n) y1 += A[lane + 32 + n * j] * xj;
    }
}

// Solves G0 x = b for the distributed right-hand side (x0, x1) in place:
// precision 0: FP64 LU (factors in G); precision 1: FP32 LU in Gf with
// FP64-residual refinement against G (unfactored). Refinement stops when
// the correction falls below 1e-14 of the solution or stops shrinking; it
// has converged when the last correction is below 1e-10 of the solution
// (the relative weight error the FP64 path is held to). Returns false when
// it has not.
__device__ bool solve_rhs(const double* G, const float* Gf, const int* piv, int n, int precision, double& x0,
                          double& x1) {
    if (precision == 0) {
        warp_lu_solve_reg(G, n, piv, x0, x1);
        return true;
    }
    const double b0 = x0, b1 = x1;
    float f0 = (float)b0, f1 = (float)b1;
    warp_lu_solve_reg(Gf, n, piv, f0, f1);
    x0 = f0;
    x1 = f1;
    double prev = INFINITY, dm = INFINITY, xm = 0;
    for (int it = 0; it < 30; ++it) {
        double y0, y1;
        warp_matvec(G, n, x0, x1, y0, y1);
        float r0 = (float)(b0 - y0), r1 = (float)(b1 - y1);
        warp_lu_solve_reg(Gf, n, piv, r0, r1);
        x0 += r0;
        x1 += r1;
        dm = fmax(fabs((double)r0), fabs((double)r1));
        xm = fmax(fabs(x0), fabs(x1));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dm = fmax(dm, __shfl_xor_sync(kFull, dm, o));
            xm = fmax(xm, __shfl_xor_sync(kFull, xm, o));
        }
        if (dm <= 1e-14 * xm || dm > 0.5 * prev) break;
        prev = dm;
    }
    return dm <= 1e-10 * xm;
}

__device__ __forceinline__ size_t rbf_smem_per_warp(int n, int k, int D, int precision) {
    size_t s = (size_t)8 * n * n + (size_t)8 * k * D + 16 * ((n + 3) / 4);
    if (precision) s += (size_t)4 * n * n + 16;
    return (s + 15) / 16 * 16;
}
size_t rbf_smem_per_warp_h(int n, int k, int D, int precision) {
    size_t s = (size_t)8 * n * n + (size_t)8 * k * D + 16 * ((n + 3) / 4);
    if (precision) s += (size_t)4 * n * n + 16;
    return (s + 15) / 16 * 16;
}

struct WarpSmem {
    double* G;
    double* xs;
    int* piv;
    float* Gf;
};
__device__ WarpSmem carve(unsigned char* base, int n, int k, int D, int precision) {
    WarpSmem w;
    w.G = reinterpret_cast<double*>(base);
    w.xs = w.G + n * n;
    w.piv = reinterpret_cast<int*>(w.xs + k * D);
    w.Gf = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(w.piv) + 16 * ((n + 3) / 4));
    return w;
}

// Factor G (and its FP32 copy when refining); returns the LU info.
__device__ int factor(WarpSmem& s, int n, int precision) {
    if (precision == 0) return warp_lu(s.G, n, s.piv);
    for (int e = lane_id(); e < n * n; e += 32) s.Gf[e] = (float)s.G[e];
    __syncwarp();
    return warp_lu(s.Gf, n, s.piv);
}

template <int D>
__global__ void rbf_weights_kernel(const float* __restrict__ src, int64_t nsrc, const uint32_t* __restrict__ support,
                                   int k, const double* __restrict__ qry, int64_t ngroups, int group, double spacing,
                                   int shape, int precision, double* __restrict__ weights, int* __restrict__ status,
                                   int wpb) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    const int n = k + D + 1;
    WarpSmem s = carve(smem + rbf_smem_per_warp(n, k, D, precision) * w, n, k, D, precision);
    for (int64_t g = (int64_t)blockIdx.x * wpb + w; g < ngroups; g += (int64_t)gridDim.x * wpb) {
        double o[D];
#pragma unroll
        for (int d = 0; d < D; ++d) o[d] = qry[(g * group) * D + d];
        for (int t = lane; t < k; t += 32) {
            uint32_t j = support[g * k + t];
            if ((int64_t)j >= nsrc) {
                atomicOr(status, 1);
                j = 0;
            }
#pragma unroll
            for (int d = 0; d < D; ++d) s.xs[t * D + d] = ((double)src[(int64_t)j * D + d] - o[d]) / spacing;
        }
        __syncwarp();
        build_G0<D>(s.xs, k, shape, s.G);
        int prec = precision;
        int info = factor(s, n, prec);
        if (info) atomicOr(status, 2);
        for (int q = 0; q < group; ++q) {
            double x[D];
#pragma unroll
            for (int d = 0; d < D; ++d) x[d] = (qry[(g * group + q) * D + d] - o[d]) / spacing;
            double x0 = lane < n ? gx_row<D>(s.xs, k, shape, x, lane) : 0.0;
            double x1 = lane + 32 < n ? gx_row<D>(s.xs, k, shape, x, lane + 32) : 0.0;
            if (!solve_rhs(s.G, s.Gf, s.piv, n, prec, x0, x1)) {
                // FP32 refinement failed: factor in FP64 and redo the group
                prec = 0;
                if (lane == 0) atomicAdd(status + 1, 1);
                if (warp_lu(s.G, n, s.piv)) atomicOr(status, 2);
                q = -1;
                continue;
            }
            double* out = weights + (g * group + q) * k;
            if (lane < k) out[lane] = x0;
            if (lane + 32 < k) out[lane + 32] = x1;
        }
        __syncwarp();
    }
}

// ------------------------------------------------- divergence stencil build
// 4-point Gauss-Legendre nodes/weights with the six-digit values NAGA uses
// (nonlocal_calculus/detail/quadrature_points.cuh:49-61).
__constant__ double c_gl_w[4] = {0.652145, 0.652145, 0.347855, 0.347855};
__constant__ double c_gl_x[4] = {0.339981, -0.339981, 0.861136, -0.861136};

// unit quadrature offset q (quadrature_points.cuh:74-157): radius
// (x_gl + 1) / 2; theta = t pi / 2; phi = p pi / 4 + pi / 8.
template <int D>
__device__ __forceinline__ void unit_quad(int q, double* u) {
    const double r = (c_gl_x[q & 3] + 1.0) / 2.0;
    const int t = (q >> 2) & 3;
    double st, ct;
    sincospi(0.5 * t, &st, &ct);
    if (D == 2) {
        u[0] = r * ct;
        u[1] = r * st;
    } else {
        const int p = q >> 4;
        double sp, cp;
        sincospi((2.0 * p + 1.0) / 8.0, &sp, &cp);
        u[0] = r * sp * ct;
        u[1] = r * sp * st;
        u[2] = r * cp;
    }
}

// antisymmetric w4 B-spline kernel (nonlocal_calculus/detail/divergence.inl:
// 55-133) and the quadrature weight of divergence.inl:171-197
template <int D>
__device__ __forceinline__ void kernel_and_weight(double delta, const double* xy, int q, double* a, double& wq) {
    const double pi = 3.141592653589793;
    double r2 = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) r2 += xy[d] * xy[d];
    const double r = sqrt(r2);
    double m;
    if (2.0 * r / delta < 1)
        m = (D == 2 ? 240.0 / 7.0 : 48.0) * r * (2.0 * delta - 3.0 * r);
    else if (2.0 * r / delta < 2)
        m = (D == 2 ? 240.0 / 7.0 : 48.0) * (delta - r) * (delta - r);
    else
        m = 0;
    wq = c_gl_w[q & 3] * delta / 2.0 * (2.0 * pi / 4.0);
    if (D == 2) {
        const double den = pi * delta * delta * delta * delta * delta;
        a[0] = m * (xy[0] / r) / den;
        a[1] = m * (xy[1] / r) / den;
        wq *= r;
    } else {
        const double rxy = sqrt(xy[0] * xy[0] + xy[1] * xy[1]);
        const double den = pi * delta * delta * delta * delta * delta * delta;
        const double sp = rxy / r, cp = xy[2] / r;
        const double ct = rxy != 0 ? xy[0] / rxy : 0, st = rxy != 0 ? xy[1] / rxy : 0;
        a[0] = m * sp * ct / den;
        a[1] = m * sp * st / den;
        a[2] = m * cp / den;
        wq *= pi / 4.0;
        wq *= r * rxy;
    }
}

// The quadrature of the stencil build depends on the node only through
// delta: xy = delta u_q, and the product a_d(xy) w_q scales exactly as
// 1 / delta (3-D: a ~ delta^2 / delta^6, w ~ delta^3; 2-D: a ~ delta^2 /
// delta^5, w ~ delta^2). One launch tabulates u_q and K_qd = a_d w_q at
// delta = 1 with the functions above; the per-node loop scales them.
struct QuadTable {
    double u[64][3];
    double K[64][3];
    double ksum[3];   // sum_q K_qd
    double mom[3][3];  // sum_q K_qd u_qe: [d][e]
    double len2[4];    // |u_q|^2 of the four radii
};
__device__ QuadTable g_quad[2];    // D2Q9, D3Q27 (filled once per device)
__constant__ QuadTable c_quad[2];  // copy of g_quad for the warp-uniform reads of quad_row

template <int D>
__global__ void quad_table_kernel() {
    QuadTable& g_q = g_quad[D - 2];
    constexpr int nq = D == 2 ? 16 : 64;
    const int q = threadIdx.x;
    if (q < nq) {
        double u[D], a[D], wq;
        unit_quad<D>(q, u);
        kernel_and_weight<D>(1.0, u, q, a, wq);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            g_q.u[q][d] = d < D ? u[d] : 0.0;
            g_q.K[q][d] = d < D ? a[d] * wq : 0.0;
        }
    }
    if (q < 4) {
        const double r = (c_gl_x[q] + 1.0) / 2.0;
        g_q.len2[q] = r * r;
    }
    __syncthreads();
    if (q < 3) {
        double sum = 0;
        for (int t = 0; t < nq; ++t) sum += g_q.K[t][q];  // fixed order
        g_q.ksum[q] = sum;
        for (int e = 0; e < 3; ++e) {
            sum = 0;
            for (int t = 0; t < nq; ++t) sum += g_q.K[t][q] * g_q.u[t][e];
            g_q.mom[q][e] = sum;
        }
    }
}

// nearest-neighbour distance |x_i - x_{idx[i][1]}| in FP64
template <int D>
__global__ void nn_kernel(const float* __restrict__ pts, const uint32_t* __restrict__ idx, int k, int64_t n,
                          double* __restrict__ nn) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t j = idx[i * k + 1];
        double s = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            double t = (double)pts[i * D + d] - (double)pts[(int64_t)j * D + d];
            s += t * t;
        }
        nn[i] = sqrt(s);
    }
}

// mean nearest-neighbour distance per batch of `batch` consecutive nodes
__global__ void batch_mean_kernel(const double* __restrict__ nn, int64_t n, int64_t batch, double* __restrict__ out) {
    __shared__ double red[32];
    const int64_t b = blockIdx.x;
    const int64_t s = b * batch, e = min(n, s + batch);
    double acc = 0;
    for (int64_t i = s + threadIdx.x; i < e; i += blockDim.x) acc += nn[i];
    acc = warp_sum(acc);
    if (lane_id() == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) out[b] = v / (double)(e - s);
    }
}

}  // namespace

namespace {

// Per-node pieces shared by the two build kernels. One warp per node i:
// the support coordinates, shifted to x_i and divided by the spacing, go to
// xs (shared); lane t keeps support index t (and t + 32) and its squared
// distance; delta is the interaction radius 0.05 |x_i - x_nn|
// (operators.cuh:84-117). A support index outside [0, n) (a kNN sentinel)
// is replaced by i and reported in bad (warp-uniform).
template <int D>
struct NodeStencil {
    uint32_t jl[2];
    double r2own[2];
    double delta, sp;
    bool bad;
};
template <int D>
__device__ __forceinline__ NodeStencil<D> load_node(const float* __restrict__ pts, int64_t n,
                                                    const uint32_t* __restrict__ idx, int k, int64_t i, double sp,
                                                    double* xs) {
    const int lane = lane_id();
    NodeStencil<D> ns;
    ns.sp = sp;
    double xi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) xi[d] = (double)pts[i * D + d];
    ns.jl[0] = ns.jl[1] = 0;
    ns.r2own[0] = ns.r2own[1] = 0;
    bool bad = false;
    for (int t = lane, r = 0; t < k; t += 32, ++r) {
        const uint32_t jr = idx[i * k + t];
        bad = bad || (int64_t)jr >= n;
        const uint32_t j = (int64_t)jr < n ? jr : (uint32_t)i;
        ns.jl[r] = j;
        double rr = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double xj = (double)pts[(int64_t)j * D + d];
            xs[t * D + d] = (xj - xi[d]) / sp;
            rr += (xj - xi[d]) * (xj - xi[d]);
        }
        ns.r2own[r] = rr;
    }
    ns.delta = 0.05 * sqrt(__shfl_sync(kFull, ns.r2own[0], 1));
    ns.bad = __any_sync(kFull, bad);
    __syncwarp();
    return ns;
}

// right-hand sides b_d = sum_q alpha_d(q) w_q G_x(q), rows lane / lane + 32,
// from the delta = 1 table: x_q = delta u_q / h, alpha_d w_q = K_qd / delta;
// cself_d = sum_q alpha_d w_q (the [s = 0] term of the weight)
template <int D>
__device__ __forceinline__ void quad_rhs(const double* xs, int k, int nsys, int shape, const NodeStencil<D>& ns,
                                         double* b0, double* b1, double* cself) {
    constexpr int nq = D == 2 ? 16 : 64;
    const int lane = lane_id();
    const QuadTable& tq = g_quad[D - 2];
    const double rdel = 1.0 / ns.delta, us = ns.delta / ns.sp;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        b0[d] = b1[d] = 0;
        cself[d] = tq.ksum[d] * rdel;
    }
    // rows lane and lane + 32: support coordinates kept in registers (RBF
    // rows), the table read through the read-only path; same arithmetic as
    // gx_row
    const int r0 = lane, r1 = lane + 32;
    double x0[D], x1[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        x0[d] = r0 < k ? xs[r0 * D + d] : 0.0;
        x1[d] = r1 < k ? xs[r1 * D + d] : 0.0;
    }
    const double* tu = &tq.u[0][0];
    const double* tk = &tq.K[0][0];
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
        double xq[D];
#pragma unroll
        for (int d = 0; d < D; ++d) xq[d] = us * __ldg(tu + 3 * q + d);
        auto row = [&](int r, const double* xr) -> double {
            if (r >= nsys) return 0.0;
            if (r < k) {
                double r2 = 0;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    const double t = xr[d] - xq[d];
                    r2 += t * t;
                }
                return shape_fn(r2, shape);
            }
            if (r == k) return 1.0;
            double v = xq[0];
#pragma unroll
            for (int d = 1; d < D; ++d)
                if (r - k - 1 == d) v = xq[d];
            return v;
        };
        const double g0 = row(r0, x0), g1 = row(r1, x1);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double aw = __ldg(tk + 3 * q + d) * rdel;
            b0[d] += aw * g0;
            b1[d] += aw * g1;
        }
    }
}

// filter weights and the stencil records of node i (weights W0: support
// lane, W1: support lane + 32)
template <int D>
__device__ __forceinline__ void write_node(const StencilOut& out, int64_t i, int k, const NodeStencil<D>& ns,
                                           const double* W0, const double* W1) {
    const int lane = lane_id();
    // selective-filter weights: normalised Gaussian of the distance
    // (detail/simulation_engine.cuh:1233-1323), computed once
    double fw0 = 0, fw1 = 0;
    if (out.Ff || (D == 2 && out.Wf)) {
        const double inv2s2 = 0.5 / (out.filter_sigma * out.filter_sigma);
        fw0 = lane < k ? exp(-ns.r2own[0] * inv2s2) : 0.0;
        fw1 = lane + 32 < k ? exp(-ns.r2own[1] * inv2s2) : 0.0;
        const double tot = warp_sum(fw0 + fw1);
        fw0 /= tot;
        fw1 /= tot;
    }
    for (int r = 0; r < 2; ++r) {
        const int t = lane + 32 * r;
        if (t >= k) break;
        const double* Wt = r == 0 ? W0 : W1;
        if (out.W64)
#pragma unroll
            for (int d = 0; d < D; ++d) out.W64[(i * k + t) * D + d] = Wt[d];
        if (out.W32)
#pragma unroll
            for (int d = 0; d < D; ++d) out.W32[(i * k + t) * D + d] = (float)Wt[d];
        const int64_t at = out.npb > 0 ? pass_record(i, t, k, out.split, out.n_total, out.npb) : i * k + t;
        if (out.Wf) {
            const float fz = D == 3 ? (float)Wt[D - 1] : (float)(r == 0 ? fw0 : fw1);
            out.Wf[at] = make_float4((float)Wt[0], (float)Wt[1], fz, __uint_as_float(ns.jl[r]));
        }
        if (out.Ff) out.Ff[at] = make_float2((float)(r == 0 ? fw0 : fw1), __uint_as_float(ns.jl[r]));
    }
    if (out.delta && lane == 0) out.delta[i] = ns.delta;
    if (out.delta32 && lane == 0) out.delta32[i] = (float)ns.delta;
}

// Any k and both precisions: G0 column-major, factored by warp_lu, the D
// right-hand sides solved one after the other.
template <int D>
__global__ void divergence_build_kernel(const float* __restrict__ pts, int64_t n, const uint32_t* __restrict__ idx,
                                        int k, const double* __restrict__ spacing, int64_t spacing_batch,
                                        int shape, int precision, StencilOut out, int* __restrict__ status,
                                        int wpb) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    const int nsys = k + D + 1;
    WarpSmem s = carve(smem + rbf_smem_per_warp(nsys, k, D, precision) * w, nsys, k, D, precision);
    for (int64_t i = (int64_t)blockIdx.x * wpb + w; i < n; i += (int64_t)gridDim.x * wpb) {
        const NodeStencil<D> ns = load_node<D>(pts, n, idx, k, i, spacing[i / spacing_batch], s.xs);
        if (ns.bad && lane == 0) atomicOr(status, 1);
        build_G0<D>(s.xs, k, shape, s.G);
        double b0[D], b1[D], cself[D];
        quad_rhs<D>(s.xs, k, nsys, shape, ns, b0, b1, cself);
        const int info = factor(s, nsys, precision);
        if (info) atomicOr(status, 2);
        double W0[D], W1[D];
        bool ok = true;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            double x0 = b0[d], x1 = b1[d];
            ok = ok && solve_rhs(s.G, s.Gf, s.piv, nsys, precision, x0, x1);
            W0[d] = x0 + (lane == 0 ? cself[d] : 0.0);
            W1[d] = x1;
        }
        if (!ok) {
            // FP32 refinement failed for this system: solve it in FP64
            if (lane == 0) atomicAdd(status + 1, 1);
            if (warp_lu(s.G, nsys, s.piv)) atomicOr(status, 2);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                double x0 = b0[d], x1 = b1[d];
                warp_lu_solve_reg(s.G, nsys, s.piv, x0, x1);
                W0[d] = x0 + (lane == 0 ? cself[d] : 0.0);
                W1[d] = x1;
            }
        }
        write_node<D>(out, i, k, ns, W0, W1);
        __syncwarp();
    }
}

// ---- stencils of up to 32 supports in FP64: the register Gauss-Jordan solve
// of warp_gj.cuh. KC is the stencil size rounded up (16, 24, 32); the rows and
// columns past k are those of the identity.

// The support rows of the moment matrix into sys.a (right-hand sides not
// touched) from the scaled support coordinates xs. The RBF block by symmetry:
// lane l evaluates the pairs (l, l + t mod KC), t = 0 .. KC / 2, and writes
// both mirror entries to the assembly rows, of which it then reads its own.
// shift, if given: a_l to take from row and column l of the RBF block.
template <int D, int KC, int NR>
__device__ __forceinline__ void assemble(GjSystem<KC, D, NR>& sys, const double* xs, int k, int shape, double* rows,
                                         const double* shift = nullptr) {
    using S = GjSystem<KC, D, NR>;
    const int l = lane_id();
    double xl[D];
#pragma unroll
    for (int d = 0; d < D; ++d) xl[d] = l < k ? xs[l * D + d] : 0.0;
    const double al = shift && l < k ? shift[l] : 0.0;
    if (l < KC) {
#pragma unroll 3
        for (int t = 0; t <= KC / 2; ++t) {
            const int c = l + t < KC ? l + t : l + t - KC;
            double r2 = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const double u = xl[d] - (c < k ? xs[c * D + d] : 0.0);
                r2 += u * u;
            }
            double v = l == c ? 1.0 : 0.0;
            if (l < k && c < k) {
                v = shape_fn(r2, shape);
                if (shift) v -= al + shift[c];
            }
            rows[l * S::LD + c] = v;
            rows[c * S::LD + l] = v;
        }
    }
    __syncwarp();
    const double* row = rows + (l < KC ? l : 0) * S::LD;
    sys.a[0] = l < k ? 1.0 : 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) sys.a[1 + d] = xl[d];
#pragma unroll
    for (int m = 0; m < KC; m += 2) {
        const double2 v = *reinterpret_cast<const double2*>(row + m);
        sys.a[S::E + m] = v.x;
        sys.a[S::E + m + 1] = v.y;
    }
#pragma unroll
    for (int m = S::E + KC + NR; m < S::W; ++m) sys.a[m] = 0.0;
    __syncwarp();  // the rows are read: solve() puts the solution there
}

// Right-hand side of support row lane: b_d = sum_q alpha_d(q) w_q phi(|x - x_q|)
// from the delta = 1 table (x_q = delta u_q / h, alpha_d w_q = K_qd / delta).
// The four angles theta of a radius and polar angle are (+-s, 0), (0, +-s) with
// one s, z and one kernel value each way, so they share their part of |x -
// x_q|^2 and enter b as differences and one sum.
template <int D>
__device__ __forceinline__ void quad_row(const double* xl, int shape, double us, double rdel, double* b) {
    const QuadTable& tq = c_quad[D - 2];
    double x2 = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        b[d] = 0;
        x2 = fma(xl[d], xl[d], x2);
    }
    const double us2 = us * us, m0 = -2.0 * us * xl[0], m1 = -2.0 * us * xl[1], m2 = D == 3 ? -2.0 * us * xl[D - 1] : 0.0;
#pragma unroll 1
    for (int p = 0; p < (D == 2 ? 1 : 4); ++p)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int q = 16 * p + r;  // theta = 0
            const double s = tq.u[q][0], z = tq.u[q][2];
            double base = fma(us2, tq.len2[r], x2);
            if (D == 3) base = fma(m2, z, base);
            // |x - x_q|^2 >= 0: the expanded form may round below for a
            // support at the node
            const double g0 = shape_fn(fmax(fma(m0, s, base), 0.0), shape);
            const double g2 = shape_fn(fmax(fma(-m0, s, base), 0.0), shape);
            const double g1 = shape_fn(fmax(fma(m1, s, base), 0.0), shape);
            const double g3 = shape_fn(fmax(fma(-m1, s, base), 0.0), shape);
            const double ks = tq.K[q][0];
            b[0] = fma(ks, g0 - g2, b[0]);
            b[1] = fma(ks, g1 - g3, b[1]);
            if (D == 3) b[D - 1] = fma(tq.K[q][2], (g0 + g2) + (g1 + g3), b[D - 1]);
        }
#pragma unroll
    for (int d = 0; d < D; ++d) b[d] *= rdel;
}

constexpr int kGjBlockWarps = 4;

// Measured against the LU in shared memory that it replaces (every
// multiply-add a shared-memory read-modify-write, 9 wavefronts per two columns
// of a row): 250k nodes, k = 32: 8.6 -> 2.9 ms (100k nodes 3.7 -> 1.2 ms);
// 50k weights 1.70 -> 0.47 ms. Bound by instruction issue at 16 warps/SM (128
// registers): half the issue slots, the FP64 pipe 28 % (the square roots of the
// quadrature and the elimination in about equal parts). Relative error of the
// stencil's weights against 80-bit solves, mean over nodes: 3-D, k = 32,
// multiquadric 5.8e-14, the LU 10.3e-14; 2-D, k = 16, cubic 1.42e-13, the LU
// 1.51e-13.
template <int D, int KC>
__global__ void __launch_bounds__(32 * kGjBlockWarps, 4)
    divergence_build_gj_kernel(const float* __restrict__ pts, int64_t n, const uint32_t* __restrict__ idx, int k,
                               const double* __restrict__ spacing, int64_t spacing_batch, int shape, StencilOut out,
                               int* __restrict__ status) {
    using S = GjSystem<KC, D, D>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    double* rows = reinterpret_cast<double*>(smem) + (size_t)S::doubles * w;
    double* pr = rows + S::kAsm;
    double* rhs = pr + S::kRow;
    double* xs = rhs + S::kRhs;
    for (int64_t i = (int64_t)blockIdx.x * kGjBlockWarps + w; i < n; i += (int64_t)gridDim.x * kGjBlockWarps) {
        const NodeStencil<D> ns = load_node<D>(pts, n, idx, k, i, spacing[i / spacing_batch], xs);
        if (ns.bad && lane == 0) atomicOr(status, 1);
        const double rdel = 1.0 / ns.delta, us = ns.delta / ns.sp;
        const QuadTable& tq = c_quad[D - 2];
        double xl[D], b[D];
#pragma unroll
        for (int d = 0; d < D; ++d) xl[d] = lane < k ? xs[lane * D + d] : 0.0;
        quad_row<D>(xl, shape, us, rdel, b);
        S sys;
        assemble<D, KC, D>(sys, xs, k, shape, rows);
#pragma unroll
        for (int d = 0; d < D; ++d) sys.a[S::E + KC + d] = lane < k ? b[d] : 0.0;
        // the constraints' right-hand sides: sum_q alpha_d w_q (1, x_q)
        if (lane < S::kRhs) {
            const int r = lane / D, d = lane % D;
            rhs[lane] = r == 0 ? tq.ksum[d] * rdel : tq.mom[d][r - 1] * us * rdel;
        }
        __syncwarp();
        if (sys.solve(k, xs, rhs, pr, rows) && lane == 0) atomicOr(status, 2);
        double W0[D], W1[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            // the node's own support also carries the [s = 0] term
            W0[d] = lane < k ? rows[lane * D + d] + (lane == 0 ? tq.ksum[d] * rdel : 0.0) : 0.0;
            W1[d] = 0.0;
        }
        write_node<D>(out, i, k, ns, W0, W1);
        __syncwarp();
    }
}

// Weights of up to NR queries of a group per solve (the elimination is run
// again for every NR of them: the caller takes it for groups of at most NR).
// T: type of the queries and the weights.
//
// The RBF block enters shifted, Phi_rc - a_r - a_c, and the right-hand sides
// less a_r: the weights sum to 1 and the constant column takes up the rest, so
// they are the same. With a_r = phi(|x_r - x|), x the first query, what is left
// of a row is small, and the elimination of the polynomial columns rounds it
// that much less (relative error of the weights in 3-D, k = 32, multiquadric:
// 2.4e-15 unshifted, 1.7e-15 shifted, 1.9e-15 by an LU with the support columns
// first; cubic in 2-D, k = 16: 1.13, 1.03 and 1.05e-14). A query outside its
// support (nearer to none than 0.6 of the farthest) would make a_r the larger
// part: x is then the nearest support (30 spacings off, cubic: 1.3e-12, the
// LU 2.5e-12). a_r is rounded to FP32, within its range, so that the sum of two
// is exact.
template <int D, int KC, int NR, class T>
__global__ void __launch_bounds__(32 * kGjBlockWarps, 4)
    rbf_weights_gj_kernel(const float* __restrict__ src, int64_t nsrc, const uint32_t* __restrict__ support, int k,
                          const T* __restrict__ qry, int64_t ngroups, int group, double spacing, int shape,
                          T* __restrict__ weights, int* __restrict__ status) {
    using S = GjSystem<KC, D, NR>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = lane_id();
    double* rows = reinterpret_cast<double*>(smem) + (size_t)S::doubles * w;
    double* pr = rows + S::kAsm;
    double* rhs = pr + S::kRow;
    double* xs = rhs + S::kRhs;
    for (int64_t g = (int64_t)blockIdx.x * kGjBlockWarps + w; g < ngroups; g += (int64_t)gridDim.x * kGjBlockWarps) {
        double o[D], xl[D], r2o = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            o[d] = (double)qry[(g * group) * D + d];
            xl[d] = 0.0;
        }
        if (lane < k) {
            uint32_t j = support[g * k + lane];
            if ((int64_t)j >= nsrc) {
                atomicOr(status, 1);
                j = 0;
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
                xl[d] = ((double)src[(int64_t)j * D + d] - o[d]) / spacing;
                xs[lane * D + d] = xl[d];
                r2o += xl[d] * xl[d];
            }
        }
        __syncwarp();
        // the shift's centre; squared distances compared by their upper words,
        // the nearest support's lane in the low bits
        const unsigned far = __reduce_max_sync(kFull, lane < k ? (unsigned)__double2hiint(0.36 * r2o) : 0u);
        const unsigned near =
            __reduce_min_sync(kFull, lane < k ? ((unsigned)__double2hiint(r2o) & ~31u) | (unsigned)lane : ~0u);
        const double phi_o = shape_fn(r2o, shape);  // the first query is the origin
        double c = phi_o;
        if ((near & ~31u) > far) {
            r2o = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const double t = xl[d] - xs[(near & 31u) * D + d];
                r2o += t * t;
            }
            c = shape_fn(r2o, shape);
        }
        const double al = c < 1e30 ? (double)(float)c : c;
        if (lane < k) pr[lane] = al;  // solve() publishes its rows there later
        __syncwarp();
        S sys;
        assemble<D, KC, NR>(sys, xs, k, shape, rows, pr);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            double x[D], r2 = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                x[d] = q < group ? ((double)qry[(g * group + q) * D + d] - o[d]) / spacing : 0.0;
                const double t = xl[d] - x[d];
                r2 += t * t;
            }
            sys.a[S::E + KC + q] = lane < k ? (q == 0 ? phi_o : shape_fn(r2, shape)) - al : 0.0;
            if (lane == 0) {
                rhs[q] = 1.0;
#pragma unroll
                for (int d = 0; d < D; ++d) rhs[(1 + d) * NR + q] = x[d];
            }
        }
        __syncwarp();
        if (sys.solve(k, xs, rhs, pr, rows) && lane == 0) atomicOr(status, 2);
        if (lane < k)
            for (int q = 0; q < NR && q < group; ++q) weights[(g * group + q) * k + lane] = (T)rows[lane * NR + q];
        __syncwarp();
    }
}

// launches kern over `count` warps' worth of systems with the per-warp shared
// memory of S
template <class S, class Kern, class... Args>
int launch_gj_systems(Kern kern, int64_t count, cudaStream_t st, Args... args) {
    const size_t smem = sizeof(double) * S::doubles * kGjBlockWarps;
    NAGA_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = (int)std::min<int64_t>((count + kGjBlockWarps - 1) / kGjBlockWarps, (int64_t)sm_count() * 32);
    kern<<<blocks, 32 * kGjBlockWarps, smem, st>>>(args...);
    NAGA_CUDA_TRY(cudaGetLastError());
    return NAGA_OK;
}

// fn(KC as std::integral_constant) for the padded size of a stencil of k <= 32
template <class Fn>
int with_padded_size(int k, Fn&& fn) {
    if (k <= 16) return fn(std::integral_constant<int, 16>{});
    if (k <= 24) return fn(std::integral_constant<int, 24>{});
    return fn(std::integral_constant<int, 32>{});
}

// the register solve serves FP64 systems of up to 32 supports, and groups of
// up to four queries (beyond that the general kernel's one factorisation
// serves all of a group)
bool gj_serves(int k, int group, int precision) { return precision == 0 && k <= 32 && group <= 4; }

template <class T>
int rbf_weights_gj(const float* src, int64_t nsrc, int dim, const uint32_t* support, int k, const T* qry,
                   int64_t ngroups, int group, double spacing, int shape, T* weights, int* status, cudaStream_t st) {
    return with_padded_size(k, [&](auto kc) -> int {
        constexpr int KC = decltype(kc)::value;
        auto go = [&](auto d, auto nr) -> int {
            constexpr int D = decltype(d)::value, NR = decltype(nr)::value;
            return launch_gj_systems<GjSystem<KC, D, NR>>(rbf_weights_gj_kernel<D, KC, NR, T>, ngroups, st, src, nsrc,
                                                          support, k, qry, ngroups, group, spacing, shape, weights,
                                                          status);
        };
        using std::integral_constant;
        if (dim == 2)
            return group == 1 ? go(integral_constant<int, 2>{}, integral_constant<int, 1>{})
                              : go(integral_constant<int, 2>{}, integral_constant<int, 4>{});
        return group == 1 ? go(integral_constant<int, 3>{}, integral_constant<int, 1>{})
                          : go(integral_constant<int, 3>{}, integral_constant<int, 4>{});
    });
}

__global__ void widen_kernel(const float* __restrict__ in, double* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)in[i];
}
__global__ void narrow_kernel(const double* __restrict__ in, float* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

int warps_per_block_for(size_t per_warp) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    size_t lim = v > 0 ? (size_t)v : 48 * 1024;
    return (int)std::min<size_t>(8, lim / per_warp);
}

}  // namespace

// RBF weights on the device; status bits: 1 bad index, 2 singular, 4 no convergence.
// T: type of the queries and the weights; the general kernel takes doubles only.
template <class T>
static int rbf_weights_typed(const float* src, int64_t nsrc, int dim, const uint32_t* support, int k, const T* qry,
                             int64_t ngroups, int group, double spacing, int shape, int precision, T* weights,
                             cudaStream_t st) {
    const int n = k + dim + 1;
    if (dim != 2 && dim != 3) return set_error(NAGA_EINVAL, "naga_rbf_weights: dim must be 2 or 3");
    if (k < dim + 1 || n > 64) return set_error(NAGA_EINVAL, "naga_rbf_weights: need dim + 1 <= k <= 60");
    if (group < 1 || ngroups < 0) return set_error(NAGA_EINVAL, "naga_rbf_weights: bad group size");
    if (!(spacing > 0)) return set_error(NAGA_EINVAL, "naga_rbf_weights: spacing must be > 0");
    if (shape != 0 && shape != 1) return set_error(NAGA_EINVAL, "naga_rbf_weights: unknown shape");
    if (precision != 0 && precision != 1) return set_error(NAGA_EINVAL, "naga_rbf_weights: unknown precision");
    if (ngroups == 0) return NAGA_OK;
    const size_t per_warp = rbf_smem_per_warp_h(n, k, dim, precision);
    const int wpb = warps_per_block_for(per_warp);
    if (wpb < 1) return set_error(NAGA_EINVAL, "naga_rbf_weights: system too large");
    int* d_status = nullptr;
    NAGA_CUDA_TRY(scratch_malloc(&d_status, 2 * sizeof(int), st));
    NAGA_CUDA_TRY(cudaMemsetAsync(d_status, 0, 2 * sizeof(int), st));
    if (gj_serves(k, group, precision)) {
        const int rc = rbf_weights_gj<T>(src, nsrc, dim, support, k, qry, ngroups, group, spacing, shape, weights,
                                         d_status, st);
        if (rc) {
            cudaFreeAsync(d_status, st);
            return rc;
        }
    } else if constexpr (std::is_same<T, double>::value) {
        const int blocks = (int)std::min<int64_t>((ngroups + wpb - 1) / wpb, (int64_t)sm_count() * 32);
        const size_t smem = per_warp * wpb;
        auto kern = dim == 2 ? rbf_weights_kernel<2> : rbf_weights_kernel<3>;
        NAGA_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<blocks, 32 * wpb, smem, st>>>(src, nsrc, support, k, qry, ngroups, group, spacing, shape, precision,
                                             weights, d_status, wpb);
    }
    NAGA_CUDA_TRY(cudaGetLastError());
    int h_st[2] = {0, 0};
    NAGA_CUDA_TRY(cudaMemcpyAsync(h_st, d_status, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    NAGA_CUDA_TRY(cudaFreeAsync(d_status, st));
    NAGA_CUDA_TRY(cudaStreamSynchronize(st));
    const int h_status = h_st[0];
    g_fallbacks = h_st[1];
    if (h_status & 1) return set_error(NAGA_EINVAL, "naga_rbf_weights: support index out of range");
    if (h_status & 2) return set_error(NAGA_ESINGULAR, "naga_rbf_weights: singular moment matrix");
    return NAGA_OK;
}

int rbf_weights_device(const float* src, int64_t nsrc, int dim, const uint32_t* support, int k, const double* qry,
                       int64_t ngroups, int group, double spacing, int shape, int precision, double* weights,
                       cudaStream_t st) {
    return rbf_weights_typed<double>(src, nsrc, dim, support, k, qry, ngroups, group, spacing, shape, precision,
                                     weights, st);
}

// FP32 queries and weights: read and written by the register solve itself,
// through FP64 copies for the systems it does not serve
int rbf_weights_f32_device(const float* src, int64_t nsrc, int dim, const uint32_t* support, int k, const float* qry,
                           int64_t ngroups, int group, double spacing, int shape, int precision, float* weights,
                           cudaStream_t st) {
    if (gj_serves(k, group, precision))
        return rbf_weights_typed<float>(src, nsrc, dim, support, k, qry, ngroups, group, spacing, shape, precision,
                                        weights, st);
    const int64_t nq = ngroups * group;
    double *q64 = nullptr, *w64 = nullptr;
    NAGA_CUDA_TRY(scratch_malloc(&q64, sizeof(double) * nq * dim, st));
    NAGA_CUDA_TRY(scratch_malloc(&w64, sizeof(double) * nq * k, st));
    const int b1 = (int)std::min<int64_t>((nq * dim + 255) / 256, (int64_t)sm_count() * 8);
    widen_kernel<<<b1, 256, 0, st>>>(qry, q64, nq * dim);
    NAGA_CUDA_TRY(cudaGetLastError());
    int rc = rbf_weights_device(src, nsrc, dim, support, k, q64, ngroups, group, spacing, shape, precision, w64, st);
    if (rc == NAGA_OK) {
        const int b2 = (int)std::min<int64_t>((nq * k + 255) / 256, (int64_t)sm_count() * 8);
        narrow_kernel<<<b2, 256, 0, st>>>(w64, weights, nq * k);
        if (cudaGetLastError() != cudaSuccess) rc = set_error(NAGA_ECUDA, "naga_rbf_weights_f32: narrow kernel");
    }
    cudaFreeAsync(q64, st);
    cudaFreeAsync(w64, st);
    return rc;
}

// kNN + interaction radii + MQ spacing + stencil weights for pts[0, n)
int divergence_build_device(const float* pts, int64_t n, int dim, int k, int shape, int precision, uint32_t* idx,
                            StencilOut out, cudaStream_t st) {
    const int nsys = k + dim + 1;
    if (dim != 2 && dim != 3) return set_error(NAGA_EINVAL, "divergence build: dim must be 2 or 3");
    if (k < dim + 2 || nsys > 64) return set_error(NAGA_EINVAL, "divergence build: need dim + 2 <= k <= 60");
    if (n < k) return set_error(NAGA_EINVAL, "divergence build: fewer points than k");
    {
        // the quadrature table of this lattice, once per device
        static std::mutex mu;
        static bool filled[64][2] = {};
        int dev = 0;
        NAGA_CUDA_TRY(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        if (dev >= 0 && dev < 64 && !filled[dev][dim - 2]) {
            if (dim == 2)
                quad_table_kernel<2><<<1, 64, 0, st>>>();
            else
                quad_table_kernel<3><<<1, 64, 0, st>>>();
            NAGA_CUDA_TRY(cudaGetLastError());
            void* table = nullptr;
            NAGA_CUDA_TRY(cudaGetSymbolAddress(&table, g_quad));
            NAGA_CUDA_TRY(cudaMemcpyToSymbolAsync(c_quad, static_cast<QuadTable*>(table) + (dim - 2), sizeof(QuadTable),
                                                  sizeof(QuadTable) * (dim - 2), cudaMemcpyDeviceToDevice, st));
            NAGA_CUDA_TRY(cudaStreamSynchronize(st));
            filled[dev][dim - 2] = true;
        }
    }
    float* d2 = nullptr;
    double* nn = nullptr;
    double* sp = nullptr;
    int* d_status = nullptr;
    const int64_t batch = 16384;
    const int64_t nb = (n + batch - 1) / batch;
    NAGA_CUDA_TRY(scratch_malloc(&d2, sizeof(float) * n * k, st));
    int rc = knn_device(pts, n, pts, n, dim, k, idx, d2, st);
    if (rc) {
        cudaFreeAsync(d2, st);
        return rc;
    }
    NAGA_CUDA_TRY(scratch_malloc(&nn, sizeof(double) * n, st));
    NAGA_CUDA_TRY(scratch_malloc(&sp, sizeof(double) * nb, st));
    NAGA_CUDA_TRY(scratch_malloc(&d_status, 2 * sizeof(int), st));
    NAGA_CUDA_TRY(cudaMemsetAsync(d_status, 0, 2 * sizeof(int), st));
    {
        const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 8);
        if (dim == 2)
            nn_kernel<2><<<blocks, 256, 0, st>>>(pts, idx, k, n, nn);
        else
            nn_kernel<3><<<blocks, 256, 0, st>>>(pts, idx, k, n, nn);
        batch_mean_kernel<<<(unsigned)nb, 256, 0, st>>>(nn, n, batch, sp);
        NAGA_CUDA_TRY(cudaGetLastError());
    }
    const size_t per_warp = rbf_smem_per_warp_h(nsys, k, dim, precision);
    const int wpb = warps_per_block_for(per_warp);
    const size_t smem = per_warp * wpb;
    const int blocks = (int)std::min<int64_t>((n + wpb - 1) / wpb, (int64_t)sm_count() * 32);
    int lrc = NAGA_OK;
    if (gj_serves(k, 1, precision)) {
        lrc = with_padded_size(k, [&](auto kc) -> int {
            constexpr int KC = decltype(kc)::value;
            if (dim == 2)
                return launch_gj_systems<GjSystem<KC, 2, 2>>(divergence_build_gj_kernel<2, KC>, n, st, pts, n, idx, k,
                                                             sp, batch, shape, out, d_status);
            return launch_gj_systems<GjSystem<KC, 3, 3>>(divergence_build_gj_kernel<3, KC>, n, st, pts, n, idx, k, sp,
                                                         batch, shape, out, d_status);
        });
    } else if (dim == 2) {
        NAGA_CUDA_TRY(cudaFuncSetAttribute(divergence_build_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        divergence_build_kernel<2><<<blocks, 32 * wpb, smem, st>>>(pts, n, idx, k, sp, batch, shape, precision, out,
                                                                   d_status, wpb);
    } else {
        NAGA_CUDA_TRY(cudaFuncSetAttribute(divergence_build_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        divergence_build_kernel<3><<<blocks, 32 * wpb, smem, st>>>(pts, n, idx, k, sp, batch, shape, precision, out,
                                                                   d_status, wpb);
    }
    if (lrc) return lrc;
    NAGA_CUDA_TRY(cudaGetLastError());
    int h_st[2] = {0, 0};
    NAGA_CUDA_TRY(cudaMemcpyAsync(h_st, d_status, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    NAGA_CUDA_TRY(cudaStreamSynchronize(st));
    const int h_status = h_st[0];
    g_fallbacks = h_st[1];
    cudaFreeAsync(d2, st);
    cudaFreeAsync(nn, st);
    cudaFreeAsync(sp, st);
    cudaFreeAsync(d_status, st);
    if (h_status & 1) return set_error(NAGA_EINVAL, "divergence build: support index out of range");
    if (h_status & 2) return set_error(NAGA_ESINGULAR, "divergence build: singular moment matrix");
    return NAGA_OK;
}

}  // namespace naga

using namespace naga;

extern "C" int64_t naga_refinement_fallbacks(void) { return naga::g_fallbacks; }

extern "C" int naga_rbf_weights(const float* src, int64_t n, int dim, const uint32_t* support, int k,
                                const double* qry, int64_t ngroups, int group, double spacing, int shape,
                                int precision, double* weights, void* stream) {
    if (ngroups > 0 && (!src || !support || !qry || !weights))
        return set_error(NAGA_EINVAL, "naga_rbf_weights: null pointer");
    return rbf_weights_device(src, n, dim, support, k, qry, ngroups, group, spacing, shape, precision, weights,
                              (cudaStream_t)stream);
}

extern "C" int naga_divergence_build(const float* pts, int64_t n, int dim, int k, int shape, int precision,
                                     uint32_t* idx, double* W, double* delta, void* stream) {
    if (!pts || !idx) return set_error(NAGA_EINVAL, "naga_divergence_build: null pointer");
    StencilOut out{};
    out.W64 = W;
    out.delta = delta;
    return divergence_build_device(pts, n, dim, k, shape, precision, idx, out, (cudaStream_t)stream);
}

extern "C" int naga_divergence_build_f32(const float* pts, int64_t n, int dim, int k, int shape, int precision,
                                         uint32_t* idx, float* W, float* delta, void* stream) {
    if (!pts || !idx) return set_error(NAGA_EINVAL, "naga_divergence_build_f32: null pointer");
    StencilOut out{};
    out.W32 = W;
    out.delta32 = delta;
    return divergence_build_device(pts, n, dim, k, shape, precision, idx, out, (cudaStream_t)stream);
}
