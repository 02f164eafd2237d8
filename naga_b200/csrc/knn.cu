// Exact k-nearest-neighbour search for point clouds on the GPU.
//
// Contract: for every query, the k source points that are smallest under the
// lexicographic order (dist^2, index), with dist^2 the FP32 value of NAGA's
// euclidean_squared (distance_functions.hpp:138-161). NAGA's own search
// (segmentation/nearest_neighbors.cuh:181-440) visits cells in a randomised
// order, breaks ties by visit order and stops one ring after k points are
// found; this search is exact instead, so results are reproducible and
// bit-identical to any exact implementation of the same order.
//
// Layout: each cloud is binned on a uniform grid (about two points per
// cell); the points are counting-sorted by cell into float4 records
// (x, y, z, local index). One warp serves one query. It gathers candidates
// from contiguous row segments (cells along x are adjacent in the sorted
// array): all rows its search ball touches, in query_kernel and, where the
// first ball does not suit, query_again; or Chebyshev shells of cells until no
// closer point can remain, in query_shells.
#include "common.cuh"
#include "scene_dev.hpp"
#include "scratch.hpp"

#include <cstring>

#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

namespace naga {

namespace {

struct CloudGrid {
    double lo[3];
    double w, inv_w;
    int dims[3];
    float r0;           // query_kernel's first radius in cells (0: it leaves the cloud to query_shells)
    int64_t cell_base;  // first cell of this cloud in the global cell array
    int64_t pt_base;    // first point of this cloud (in the input arrays)
    int64_t n;          // points in the cloud
};

// The cell width, and query_kernel's first radius: the ball that holds 1.4 k
// points (at least 8 more than k) at the cloud's mean count per cell. 0 where
// an axis met its cap of 2^20 cells (points past it share the last cell, whose
// place then says nothing of theirs) or the cloud has fewer points than k.
void set_radius(CloudGrid& g, double w, int64_t n, int dim, int k) {
    g.w = w;
    g.inv_w = 1.0 / w;
    double cells = 1;
    bool capped = false;
    for (int d = 0; d < dim; ++d) {
        cells *= g.dims[d];
        capped = capped || g.dims[d] >= 1 << 20;
    }
    const double v = std::max(1.4 * k, k + 8.0) * cells / (double)std::max<int64_t>(n, 1);
    g.r0 = capped || n < k ? 0.f : (float)(dim == 2 ? std::sqrt(v / 3.141592653589793) : std::cbrt(v / 4.18879020478639));
}

__device__ __forceinline__ int find_cloud(const int64_t* offsets, int nclouds, int64_t p) {
    int lo = 0, hi = nclouds - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (offsets[mid] <= p)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// order-preserving float <-> int encoding for atomic min / max
__device__ __forceinline__ int f2ord(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__host__ __device__ inline float ord2f(int i) {
#ifdef __CUDA_ARCH__
    return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
#else
    int j = i >= 0 ? i : i ^ 0x7fffffff;
    float f;
    std::memcpy(&f, &j, 4);
    return f;
#endif
}

// Bounding boxes, `per` consecutive blocks a cloud. Each thread reduces its
// points in registers and a warp publishes one atomic per bound; one atomic
// per point and bound serialises on the few addresses of a cloud (64 clouds,
// 3.2 M points: 7.4 ms -> 0.023 ms).
template <int D>
__global__ void bbox_kernel(const float* pts, const int64_t* offsets, int per,
                            int* bbox /* [nclouds][2][3] ordered ints */) {
    const int c = blockIdx.x / per;
    const int64_t b = offsets[c], e = offsets[c + 1];
    int lo[D], hi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        lo[d] = 0x7fffffff;
        hi[d] = (int)0x80000000;
    }
    for (int64_t p = b + (int64_t)(blockIdx.x % per) * blockDim.x + threadIdx.x; p < e; p += (int64_t)per * blockDim.x) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const int v = f2ord(pts[p * D + d]);
            lo[d] = min(lo[d], v);
            hi[d] = max(hi[d], v);
        }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        lo[d] = __reduce_min_sync(kFull, lo[d]);
        hi[d] = __reduce_max_sync(kFull, hi[d]);
        if (lane_id() == 0 && lo[d] <= hi[d]) {
            atomicMin(&bbox[c * 6 + d], lo[d]);
            atomicMax(&bbox[c * 6 + 3 + d], hi[d]);
        }
    }
}

// blocks per cloud of bbox_kernel: about 4096 points a block, at most eight
// blocks an SM over all clouds
int bbox_blocks_per_cloud(int64_t total, int nclouds) {
    const int64_t want = total / nclouds / 4096 + 1;
    const int64_t cap = std::max<int64_t>(1, (int64_t)sm_count() * 8 / nclouds);
    return (int)std::min(want, cap);
}

template <int D>
__device__ __forceinline__ void cell_of(const CloudGrid& g, const float* x, int* c) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        double v = floor(((double)x[d] - g.lo[d]) / g.w);
        long long iv = (long long)v;
        c[d] = (int)min(max(iv, 0LL), (long long)g.dims[d] - 1);
    }
}

template <int D>
__device__ __forceinline__ int64_t cell_id(const CloudGrid& g, const int* c) {
    int64_t id = c[0];
    if (D > 1) id += (int64_t)g.dims[0] * c[1];
    if (D > 2) id += (int64_t)g.dims[0] * g.dims[1] * c[2];
    return id;
}

template <int D>
__global__ void count_kernel(const float* pts, const int64_t* offsets, int nclouds, int64_t total,
                             const CloudGrid* grids, unsigned* counts) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total;
         p += (int64_t)gridDim.x * blockDim.x) {
        int cl = find_cloud(offsets, nclouds, p);
        CloudGrid g = grids[cl];
        int c[3];
        cell_of<D>(g, pts + p * D, c);
        atomicAdd(&counts[g.cell_base + cell_id<D>(g, c)], 1u);
    }
}

template <int D>
__global__ void scatter_kernel(const float* pts, const int64_t* offsets, int nclouds, int64_t total,
                               const CloudGrid* grids, const unsigned* start, unsigned* fill,
                               float4* sorted) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total;
         p += (int64_t)gridDim.x * blockDim.x) {
        int cl = find_cloud(offsets, nclouds, p);
        CloudGrid g = grids[cl];
        int c[3];
        cell_of<D>(g, pts + p * D, c);
        int64_t cid = g.cell_base + cell_id<D>(g, c);
        unsigned pos = start[cid] + atomicAdd(&fill[cid], 1u);
        float4 r;
        r.x = pts[p * D + 0];
        r.y = D > 1 ? pts[p * D + 1] : 0.f;
        r.z = D > 2 ? pts[p * D + 2] : 0.f;
        r.w = __uint_as_float((unsigned)(p - g.pt_base));
        sorted[pos] = r;
    }
}

__device__ __forceinline__ bool cand_less(float ad, unsigned ai, float bd, unsigned bi) {
    return ad < bd || (ad == bd && ai < bi);
}

// General exact search of one query by its warp, for any cloud and any k <=
// 32 R: Chebyshev shells of cells around the query's cell, the k best
// candidates kept sorted over the lanes by insertion (entry e in lane e % 32,
// register e / 32). The walk stops once the k-th candidate is strictly closer
// than the nearest face of the searched block that does not already touch
// the edge of the grid. query_kernel takes it where its radius search does
// not settle.
template <int D, int R>
__device__ __noinline__ void query_shells(float x0, float x1, float x2, const CloudGrid* grid,
                                          const unsigned* cell_start, const float4* sorted, int k, uint32_t* out_idx,
                                          float* out_d2) {
    const int lane = lane_id();
    const CloudGrid g = *grid;
    const float x[3] = {x0, x1, x2};
    int c0[3] = {0, 0, 0};
    cell_of<D>(g, x, c0);

    float ld[R];
    unsigned li[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        ld[r] = INFINITY;
        li[r] = 0xffffffffu;
    }
    const int kl = (k - 1) & 31, kr = (k - 1) >> 5;

    for (int rad = 0;; ++rad) {
        // rows of the shell along x that lie in the grid, each giving at most
        // two segments (the full row, or its two end cells): a long or flat
        // grid has few of the (2 rad + 1)^(D-1), and a walk over all of them
        // would not end in a useful time
        const int y0 = max(-rad, -c0[1]), y1 = min(rad, g.dims[1] - 1 - c0[1]);
        const int z0 = D == 3 ? max(-rad, -c0[2]) : 0, z1 = D == 3 ? min(rad, g.dims[2] - 1 - c0[2]) : 0;
        const int side = y1 - y0 + 1;
        const int64_t nseg = 2 * (int64_t)side * (z1 - z0 + 1);
        for (int64_t s0 = 0; s0 < nseg; s0 += 32) {
            const int64_t sid = s0 + lane;
            unsigned sb = 0, se = 0;
            if (sid < nseg) {
                const int64_t row = sid >> 1;
                const int half = (int)(sid & 1);
                const int dz = D == 3 ? z0 + (int)(row / side) : 0;
                const int dy = y0 + (int)(D == 3 ? row % side : row);
                const int cy = c0[1] + dy, cz = c0[2] + dz;
                const bool full = (dy == -rad || dy == rad) || (D == 3 && (dz == -rad || dz == rad));
                int xa, xb;
                if (full) {
                    xa = half ? 1 : c0[0] - rad;
                    xb = half ? 0 : c0[0] + rad;
                } else {
                    xa = xb = half ? c0[0] + rad : c0[0] - rad;
                }
                // an end cell outside the grid is no cell of it
                if (full || (xa >= 0 && xa < g.dims[0])) {
                    xa = max(xa, 0);
                    xb = min(xb, g.dims[0] - 1);
                    if (xa <= xb) {
                        int ca[3] = {xa, cy, cz}, cb[3] = {xb, cy, cz};
                        int64_t ia = g.cell_base + cell_id<D>(g, ca);
                        int64_t ib = g.cell_base + cell_id<D>(g, cb);
                        sb = cell_start[ia];
                        se = cell_start[ib + 1];
                    }
                }
            }
            unsigned len = se - sb;
            // inclusive scan of segment lengths across the warp
            unsigned incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                unsigned t = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += t;
            }
            unsigned excl = incl - len;
            unsigned total = __shfl_sync(kFull, incl, 31);
            for (unsigned base = 0; base < total; base += 32) {
                unsigned t = base + lane;
                float cd = INFINITY;
                unsigned ci = 0xffffffffu;
                // find the segment holding item t: largest lane j with excl_j <= t
                int j = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    unsigned e = __shfl_sync(kFull, excl, j + step);
                    if (j + step < 32 && e <= t) j += step;
                }
                unsigned sbj = __shfl_sync(kFull, sb, j);
                unsigned exj = __shfl_sync(kFull, excl, j);
                if (t < total) {
                    float4 p = sorted[sbj + (t - exj)];
                    float pv[3] = {p.x, p.y, p.z};
                    cd = dist2_ref<D>(x, pv);
                    ci = __float_as_uint(p.w);
                }
                float kd = __shfl_sync(kFull, ld[kr], kl);
                unsigned ki = __shfl_sync(kFull, li[kr], kl);
                unsigned mask = __ballot_sync(kFull, cand_less(cd, ci, kd, ki));
                while (mask) {
                    int b = __ffs(mask) - 1;
                    mask &= mask - 1;
                    float bd = __shfl_sync(kFull, cd, b);
                    unsigned bi = __shfl_sync(kFull, ci, b);
                    kd = __shfl_sync(kFull, ld[kr], kl);
                    ki = __shfl_sync(kFull, li[kr], kl);
                    if (!cand_less(bd, bi, kd, ki)) continue;
                    int pos = 0;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        pos += __popc(__ballot_sync(kFull, cand_less(ld[r], li[r], bd, bi)));
                    // shift entries >= pos up by one and drop the last
                    float carry_d = INFINITY;
                    unsigned carry_i = 0xffffffffu;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float upd = __shfl_up_sync(kFull, ld[r], 1);
                        unsigned upi = __shfl_up_sync(kFull, li[r], 1);
                        float topd = __shfl_sync(kFull, ld[r], 31);
                        unsigned topi = __shfl_sync(kFull, li[r], 31);
                        float prevd = lane == 0 ? carry_d : upd;
                        unsigned previ = lane == 0 ? carry_i : upi;
                        int e = 32 * r + lane;
                        if (e == pos) {
                            ld[r] = bd;
                            li[r] = bi;
                        } else if (e > pos) {
                            ld[r] = prevd;
                            li[r] = previ;
                        }
                        carry_d = topd;
                        carry_i = topi;
                    }
                }
            }
        }
        // stopping test after the full shell
        double bound = INFINITY;
        bool covered = true;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            if (c0[d] - rad > 0) {
                covered = false;
                bound = fmin(bound, (double)x[d] - (g.lo[d] + (double)(c0[d] - rad) * g.w));
            }
            if (c0[d] + rad < g.dims[d] - 1) {
                covered = false;
                bound = fmin(bound, (g.lo[d] + (double)(c0[d] + rad + 1) * g.w) - (double)x[d]);
            }
        }
        if (covered) break;
        float kd = __shfl_sync(kFull, ld[kr], kl);
        if (kd < INFINITY && bound > 0 && (double)kd < bound * bound * (1.0 - 1e-5)) break;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int e = 32 * r + lane;
        if (e < k) {
            out_idx[e] = li[r];
            out_d2[e] = ld[r];
        }
    }
}

// Ranks of the first cnt (dist^2, index) keys among themselves; lane l holds
// keys l, l + 32, ... By dist^2 alone, four comparisons a read; ranks that are
// not all different (tied distances) are counted again with the index.
// key has room for four entries past cnt.
template <int PER>
__device__ __forceinline__ void rank_keys(float* key, const unsigned* id, int cnt, float* mine, unsigned* who,
                                          int* rank) {
    const int lane = lane_id();
    if (lane < 4) key[cnt + lane] = INFINITY;
    __syncwarp();
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int e = lane + 32 * u;
        mine[u] = e < cnt ? key[e] : INFINITY;
        who[u] = e < cnt ? id[e] : 0xffffffffu;
        rank[u] = 0;
    }
    for (int i = 0; i < cnt; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(key + i);
#pragma unroll
        for (int u = 0; u < PER; ++u)
            rank[u] += (v.x < mine[u]) + (v.y < mine[u]) + (v.z < mine[u]) + (v.w < mine[u]);
    }
    int distinct = 0;
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        unsigned bits = 0;
#pragma unroll
        for (int u = 0; u < PER; ++u)
            if (lane + 32 * u < cnt && rank[u] >> 5 == h) bits |= 1u << (rank[u] & 31);
        distinct += __popc(__reduce_or_sync(kFull, bits));
    }
    if (distinct != cnt) {
#pragma unroll
        for (int u = 0; u < PER; ++u) rank[u] = 0;
        for (int i = 0; i < cnt; ++i) {
            const float kd = key[i];
            const unsigned ki = id[i];
#pragma unroll
            for (int u = 0; u < PER; ++u) rank[u] += cand_less(kd, ki, mine[u], who[u]);
        }
    }
}

// Keeps the k nearest of cnt >= k keys, in order; the k-th one's dist^2.
template <int PER>
__device__ __forceinline__ float keep_nearest(float* key, unsigned* id, int cnt, int k) {
    float mine[PER];
    unsigned who[PER];
    int rank[PER];
    rank_keys<PER>(key, id, cnt, mine, who, rank);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (lane_id() + 32 * u < cnt && rank[u] < k) {
            key[rank[u]] = mine[u];
            id[rank[u]] = who[u];
        }
    __syncwarp();
    return key[k - 1];
}

// a query in cells of its cloud's grid: cell c0 and the place f in [0, 1)
// inside it
struct QueryCell {
    int c0[3];
    float f[3];
};
// a warp's shared memory: collected keys and the non-empty rows of a chunk
struct QueryScratch {
    float* key;
    unsigned *id, *row_off;
};
struct Collected {
    int cnt, rows;  // keys collected (-1: no search of this radius), rows read
    unsigned seen;  // points of the rows read
};

// Collects every point within rad cells of a query. The cells of the ball are
// walked by rows along x, one row a lane, clipped to the ball.
// BOUNDED: where more than CAP points turn up, the k nearest so far are kept
// and the bound falls to the k-th of them; nothing is collected (cnt 0) from
// rows of more than `most` points. Otherwise the walk ends there, with a count
// above CAP.
template <int D, int CAP, bool BOUNDED>
__device__ __forceinline__ Collected collect_ball(const CloudGrid& g, const unsigned* cell_start, const float4* sorted,
                                                  const float* x, const QueryCell& q, float rad, int k,
                                                  const QueryScratch& s, unsigned most = 0) {
    const int lane = lane_id();
    const unsigned below = (1u << lane) - 1u;
    const float w = (float)g.w;
    float T = (rad * w) * (rad * w);
    unsigned Ti = 0xffffffffu;  // index bound of points at T itself
    // the ball in cells, with room for the rounding of T, dist^2 and f
    const float rho = fmaf(rad, 1.f + 2e-5f, 1e-5f);
    // T beyond FP32: distances that overflow tie at infinity, and only the
    // shell walk sees all of them
    if (!(rho < 1e4f && T < INFINITY)) return {-1, 0, 0u};
    int a[3] = {0, 0, 0}, m[3] = {1, 1, 1};
#pragma unroll
    for (int d = 1; d < D; ++d) {
        const int lo = max(q.c0[d] + (int)floorf(q.f[d] - rho), 0);
        const int hi = min(q.c0[d] + (int)floorf(q.f[d] + rho), g.dims[d] - 1);
        a[d] = lo;
        m[d] = hi - lo + 1;
    }
    const int nrows = m[1] > 0 && m[2] > 0 ? m[1] * m[2] : 0;
    if (nrows > 1024) return {-1, 0, 0u};
    int cnt = 0;
    unsigned seen = 0;
    for (int t0 = 0; t0 < nrows && (BOUNDED || cnt <= CAP); t0 += 32) {
        unsigned sb = 0, len = 0;
        const int t = t0 + lane;
        if (t < nrows) {
            const int rz = D == 3 ? t / m[1] : 0, ry = t - rz * m[1];
            const int cy = a[1] + ry, cz = a[2] + rz;
            // squared distance of the row's slab in y (and z)
            const float oy = (float)(cy - q.c0[1]) - q.f[1];
            float e = fmaxf(0.f, fmaxf(oy, -1.f - oy));
            float rem = fmaf(-e, e, rho * rho);
            if (D == 3) {
                const float oz = (float)(cz - q.c0[2]) - q.f[2];
                e = fmaxf(0.f, fmaxf(oz, -1.f - oz));
                rem = fmaf(-e, e, rem);
            }
            if (rem >= 0.f) {
                const float hx = fmaf(sqrtf(rem), 1.f + 1e-5f, 1e-5f);
                const int xa = max(q.c0[0] + (int)floorf(q.f[0] - hx), 0);
                const int xb = min(q.c0[0] + (int)floorf(q.f[0] + hx), g.dims[0] - 1);
                if (xa <= xb) {
                    const int ca[3] = {xa, cy, cz};
                    const int64_t ia = g.cell_base + cell_id<D>(g, ca);
                    sb = cell_start[ia];
                    len = cell_start[ia + (xb - xa) + 1] - sb;
                }
            }
        }
        unsigned incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        const unsigned excl = incl - len, total = __shfl_sync(kFull, incl, 31);
        if (BOUNDED) {
            seen += total;
            if (seen > most) return {0, nrows, seen};
        }
        // the non-empty rows in order: item i of the chunk is point
        // row_off[rank of its row] + i
        const unsigned some = __ballot_sync(kFull, len > 0);
        if (len > 0) s.row_off[__popc(some & below)] = sb - excl;
        __syncwarp();
        int before = 0;  // rows begun in earlier batches
        for (unsigned base = 0; base < total && (BOUNDED || cnt <= CAP); base += 32) {
            const bool head = len > 0 && excl - base < 32u;
            const unsigned heads = __reduce_or_sync(kFull, head ? 1u << (excl - base) : 0u);
            const unsigned i = base + lane;
            const int j = before + __popc(heads & (below | 1u << lane)) - 1;
            before += __popc(heads);
            float cd = INFINITY;
            unsigned ci = 0xffffffffu;
            if (i < total) {
                const float4 v = sorted[s.row_off[j] + i];
                const float sv[3] = {v.x, v.y, v.z};
                cd = dist2_ref<D>(x, sv);
                ci = __float_as_uint(v.w);
            }
            bool take = BOUNDED ? cand_less(cd, ci, T, Ti) : cd <= T;
            unsigned mask = __ballot_sync(kFull, take);
            if (BOUNDED && cnt + __popc(mask) > CAP) {
                __syncwarp();
                T = keep_nearest<CAP / 32>(s.key, s.id, cnt, k);
                Ti = s.id[k - 1];
                cnt = k;
                take = cand_less(cd, ci, T, Ti);
                mask = __ballot_sync(kFull, take);
            }
            const int pos = cnt + __popc(mask & below);
            if (take && pos < CAP) {
                s.key[pos] = cd;
                s.id[pos] = ci;
            }
            cnt += __popc(mask);
        }
        __syncwarp();
    }
    return {cnt, nrows, seen};
}

// the k nearest of cnt >= k collected keys
template <int PER>
__device__ __forceinline__ void write_nearest(const QueryScratch& s, int cnt, int k, uint32_t* out_idx, float* out_d2) {
    float mine[PER];
    unsigned who[PER];
    int rank[PER];
    rank_keys<PER>(s.key, s.id, cnt, mine, who, rank);
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (lane_id() + 32 * u < cnt && rank[u] < k) {
            out_idx[rank[u]] = who[u];
            out_d2[rank[u]] = mine[u];
        }
    __syncwarp();
}

template <int R>
struct QueryCap {
    static constexpr int cap = 64 * R;  // keys collected at most: 32 R to keep, and a warp's more
};

// The search of a query whose first ball, of rad cells, held fewer than k
// points or more than can be collected (rad 0: no first ball). A ball whose
// rows hold far too many is shrunk before they are read (the first ones, and
// one that grew well past a radius with too few); one with fewer than k grows.
// A query that does not settle in kTries rounds or kRowsRead rows (an empty
// neighbourhood, fewer points than k, a non-finite query) takes query_shells.
constexpr int kTries = 8, kRowsRead = 4096;
constexpr int kShrinks = 1;      // first rounds that may shrink the ball unread
constexpr int kFarTooMany = 10;  // from this many times CAP points in its rows
template <int D, int R>
__device__ __noinline__ void query_again(float x0, float x1, float x2, const CloudGrid* grid, const unsigned* cell_start,
                                         const float4* sorted, int k, float rad, QueryCell q, QueryScratch s,
                                         uint32_t* out_idx, float* out_d2) {
    constexpr int CAP = QueryCap<R>::cap;
    const CloudGrid g = *grid;
    const float x[3] = {x0, x1, x2};
    float rad_lo = 0.f;  // the largest radius with too few
    int rows = 0;
    for (int tries = 0; rad > 0.f && tries < kTries && rows <= kRowsRead; ++tries) {
        const bool may_shrink = tries < kShrinks || (rad_lo > 0.f && rad_lo < 0.6f * rad);
        const unsigned most = may_shrink ? kFarTooMany * CAP : ~0u;
        const Collected c = collect_ball<D, CAP, true>(g, cell_start, sorted, x, q, rad, k, s, most);
        if (c.cnt < 0) break;
        if (c.cnt >= k) {
            write_nearest<CAP / 32>(s, c.cnt, k, out_idx, out_d2);
            return;
        }
        rows += c.rows;
        // to 1.4 k points by the count found, to 8 k or so by the rows' points
        // (two fifths of them lie in the ball), halfway to a radius with too few
        const bool shrink = c.seen > most;
        const float r = (float)k * (shrink ? 20.f / (float)c.seen : 1.4f / fmaxf((float)c.cnt, 1.f));
        const float step = D == 2 ? sqrtf(r) : cbrtf(r);
        if (!shrink) rad_lo = rad;
        rad = shrink ? fmaxf(rad * step, sqrtf(rad * rad_lo)) : rad * fminf(2.f, fmaxf(1.05f, step));
    }
    query_shells<D, R>(x0, x1, x2, grid, cell_start, sorted, k, out_idx, out_d2);
}

// Warp-per-query exact search by radius. R = 1 for k <= 32, 2 for k <= 64.
//
// The warp collects every point with dist^2 <= T in shared memory, T chosen
// so that about 1.4 k points are expected, and ranks the collected (dist^2,
// index) keys against each other: the k of lowest rank are the answer, since
// no point outside the collection is closer than one inside. T comes from the
// cloud's mean density, corrected for the part of the ball outside the
// bounding box; a query that it does not suit goes on in query_again.
//
// A query reads ~2.5 k candidates instead of the ~8 k of full cell shells, and
// ranking costs ~1.4 k broadcast reads instead of one dependent insertion per
// improvement (64 clouds, 3.2 M points, k = 32: 12.9 -> 4.2 ms; 250k points
// 0.98 -> 0.33 ms; 1 to 6 points a cell take the same time within 10 %). Bound
// by instruction issue: ~1000 warp instructions a query, 74 % of the issue
// slots, L1 38 %.
// Clouds of uneven density, 30,000 points, all as queries: coordinates cubed
// from a normal distribution, k = 8, 32, 64: 1.8, 1.7, 2.8 ms (searched again
// wherever too many points turned up, with nothing kept: 3.0, 3.6, 4.7; shells
// of cells with sorted insertion: 1.7, 1.8, 2.6).
// The rare searches stand in a function of their own: in line they cost the
// common one 5 to 7 %. 5 blocks/SM at 48 registers (4 at 64: 4.28 ms on the 64
// clouds against 4.16, 3 at 80 4.74, 6 at 40 4.5).
//
// SELF: the queries are the sources; query q is the point at place q of the
// cell order, so that a block's queries share cells.
template <int D, int R, bool SELF>
__global__ void __launch_bounds__(256, 5) query_kernel(const float* qry, int64_t nq, const int64_t* q_offsets,
                                                       int q_nclouds, const CloudGrid* grids,
                                                       const unsigned* cell_start, const float4* sorted,
                                                       int k, uint32_t* out_idx, float* out_d2) {
    constexpr int CAP = QueryCap<R>::cap;
    __shared__ __align__(16) float key_s[8][CAP + 4];
    __shared__ unsigned id_s[8][CAP];
    __shared__ unsigned row_s[8][32];
    const int wid = threadIdx.x >> 5;
    const QueryScratch scratch{key_s[wid], id_s[wid], row_s[wid]};
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t p = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; p < nq; p += warps) {
        const int cl = q_offsets ? find_cloud(q_offsets, q_nclouds, p) : 0;
        const CloudGrid g = grids[cl];
        float x[3] = {0.f, 0.f, 0.f};
        int64_t q = p;
        if constexpr (SELF) {
            const float4 r = sorted[p];
            x[0] = r.x;
            x[1] = r.y;
            x[2] = r.z;
            q = g.pt_base + __float_as_uint(r.w);
        } else {
#pragma unroll
            for (int d = 0; d < D; ++d) x[d] = qry[q * D + d];
        }
        QueryCell c = {{0, 0, 0}, {0.f, 0.f, 0.f}};
        float out2 = 0.f;   // squared distance to the grid's box
        float inside = 1.f;  // part of the ball's box inside the grid's box
        const float r0 = g.r0;
        bool ok = r0 > 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double u = ((double)x[d] - g.lo[d]) * g.inv_w;
            ok = ok && fabs(u) < 1e9;
            const double fl = floor(u);
            c.c0[d] = ok ? (int)fl : 0;
            c.f[d] = (float)(u - fl);
            const float uf = (float)u, hi = (float)g.dims[d];
            const float o = fmaxf(0.f, fmaxf(-uf, uf - hi));
            out2 = fmaf(o, o, out2);
            inside *= fmaxf(0.3f, (fminf(uf + r0, hi) - fmaxf(uf - r0, 0.f)) / (2.f * r0));
        }
        // radius in cells; past the box, the distance to it comes on top
        const float rad = fmaf(r0, exp2f((-1.f / D) * __log2f(inside)), sqrtf(out2));
        int cnt = -1;
        if (ok) cnt = collect_ball<D, CAP, false>(g, cell_start, sorted, x, c, rad, k, scratch).cnt;
        if (cnt >= k && cnt <= CAP)
            write_nearest<CAP / 32>(scratch, cnt, k, out_idx + q * k, out_d2 + q * k);
        else
            query_again<D, R>(x[0], x[1], x[2], grids + cl, cell_start, sorted, k, cnt < 0 ? 0.f : rad, c, scratch,
                              out_idx + q * k, out_d2 + q * k);
    }
}

template <int D>
void launch_query(const float* qry, int64_t nq, const int64_t* d_qoff, int nclouds, const CloudGrid* grids,
                  const unsigned* start, const float4* sorted, int k, bool self, uint32_t* idx, float* d2,
                  cudaStream_t st) {
    const int blocks = (int)std::min<int64_t>((nq + 7) / 8, (int64_t)sm_count() * 32);
    auto go = [&](auto kern) {
        kern<<<blocks, 256, 0, st>>>(qry, nq, d_qoff, nclouds, grids, start, sorted, k, idx, d2);
    };
    if (k <= 32)
        self ? go(query_kernel<D, 1, true>) : go(query_kernel<D, 1, false>);
    else
        self ? go(query_kernel<D, 2, true>) : go(query_kernel<D, 2, false>);
}

template <int D>
int knn_run(const float* src, const int64_t* h_src_off, int nclouds, const float* qry, int64_t nq,
            const int64_t* h_q_off, int k, uint32_t* idx, float* d2, cudaStream_t st) {
    const int64_t total = h_src_off[nclouds];
    int64_t* d_off = nullptr;
    int64_t* d_qoff = nullptr;
    int* d_bbox = nullptr;
    CloudGrid* d_grids = nullptr;
    unsigned *d_counts = nullptr, *d_start = nullptr, *d_fill = nullptr;
    float4* d_sorted = nullptr;
    void* d_tmp = nullptr;
    int rc = NAGA_OK;
    std::vector<int> hb(6 * nclouds);
    std::vector<CloudGrid> grids(nclouds);
    int64_t ncell = 0;
    size_t tmp_bytes = 0;
    auto fail = [&](cudaError_t e, const char* what) {
        rc = set_error(NAGA_ECUDA, std::string("naga_knn: ") + what + ": " + cudaGetErrorString(e));
    };
    cudaError_t e;
#define KTRY(x, what)          \
    if ((e = (x)) != cudaSuccess) { \
        fail(e, what);         \
        goto done;             \
    }
    KTRY(scratch_malloc(&d_off, sizeof(int64_t) * (nclouds + 1), st), "alloc");
    KTRY(cudaMemcpyAsync(d_off, h_src_off, sizeof(int64_t) * (nclouds + 1), cudaMemcpyHostToDevice, st), "copy");
    if (h_q_off) {
        KTRY(scratch_malloc(&d_qoff, sizeof(int64_t) * (nclouds + 1), st), "alloc");
        KTRY(cudaMemcpyAsync(d_qoff, h_q_off, sizeof(int64_t) * (nclouds + 1), cudaMemcpyHostToDevice, st), "copy");
    }
    for (int c = 0; c < nclouds; ++c)
        for (int d = 0; d < 3; ++d) {
            hb[c * 6 + d] = 0x7fffffff;
            hb[c * 6 + 3 + d] = (int)0x80000000;
        }
    KTRY(scratch_malloc(&d_bbox, sizeof(int) * 6 * nclouds, st), "alloc");
    KTRY(cudaMemcpyAsync(d_bbox, hb.data(), sizeof(int) * 6 * nclouds, cudaMemcpyHostToDevice, st), "copy");
    if (total > 0) {
        const int per = bbox_blocks_per_cloud(total, nclouds);
        bbox_kernel<D><<<(unsigned)(per * nclouds), 256, 0, st>>>(src, d_off, per, d_bbox);
        KTRY(cudaGetLastError(), "bbox kernel");
    }
    KTRY(cudaMemcpyAsync(hb.data(), d_bbox, sizeof(int) * 6 * nclouds, cudaMemcpyDeviceToHost, st), "copy");
    KTRY(cudaStreamSynchronize(st), "sync");
    for (int c = 0; c < nclouds; ++c) {
        CloudGrid& g = grids[c];
        int64_t n = h_src_off[c + 1] - h_src_off[c];
        double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, vol = 1;
        for (int d = 0; d < D; ++d) {
            lo[d] = n > 0 ? (double)ord2f(hb[c * 6 + d]) : 0.0;
            hi[d] = n > 0 ? (double)ord2f(hb[c * 6 + 3 + d]) : 1.0;
            // a NaN or infinite coordinate always lands in a bound (the
            // ordered-integer min / max puts NaN at one end)
            if (!std::isfinite(lo[d]) || !std::isfinite(hi[d])) {
                rc = set_error(NAGA_EINVAL, "naga_knn: non-finite point coordinates in cloud " + std::to_string(c));
                goto done;
            }
            if (hi[d] - lo[d] < 1e-6) hi[d] = lo[d] + 1e-6;
            vol *= hi[d] - lo[d];
        }
        double w = std::pow(2.0 * vol / (double)std::max<int64_t>(n, 1), 1.0 / D);
        int64_t cells = 1;
        for (int d = 0; d < 3; ++d) {
            g.lo[d] = lo[d];
            int64_t dd = d < D ? std::max<int64_t>(1, (int64_t)std::ceil((hi[d] - lo[d]) / w)) : 1;
            dd = std::min<int64_t>(dd, 1 << 20);
            g.dims[d] = (int)dd;
            cells *= dd;
        }
        set_radius(g, w, n, D, k);
        g.cell_base = ncell;
        g.pt_base = h_src_off[c];
        g.n = n;
        ncell += cells;
    }
    KTRY(scratch_malloc(&d_grids, sizeof(CloudGrid) * nclouds, st), "alloc");
    KTRY(cudaMemcpyAsync(d_grids, grids.data(), sizeof(CloudGrid) * nclouds, cudaMemcpyHostToDevice, st), "copy");
    KTRY(scratch_malloc(&d_counts, sizeof(unsigned) * (ncell + 1), st), "alloc");
    KTRY(scratch_malloc(&d_start, sizeof(unsigned) * (ncell + 1), st), "alloc");
    KTRY(scratch_malloc(&d_fill, sizeof(unsigned) * (ncell + 1), st), "alloc");
    KTRY(cudaMemsetAsync(d_counts, 0, sizeof(unsigned) * (ncell + 1), st), "memset");
    KTRY(cudaMemsetAsync(d_fill, 0, sizeof(unsigned) * (ncell + 1), st), "memset");
    KTRY(scratch_malloc(&d_sorted, sizeof(float4) * std::max<int64_t>(total, 1), st), "alloc");
    if (total > 0) {
        int blocks = (int)std::min<int64_t>((total + 255) / 256, 4 * 148 * 8);
        count_kernel<D><<<blocks, 256, 0, st>>>(src, d_off, nclouds, total, d_grids, d_counts);
        KTRY(cudaGetLastError(), "count kernel");
    }
    KTRY(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, d_counts, d_start, ncell + 1, st), "scan size");
    KTRY(scratch_malloc(&d_tmp, tmp_bytes, st), "alloc");
    KTRY(cub::DeviceScan::ExclusiveSum(d_tmp, tmp_bytes, d_counts, d_start, ncell + 1, st), "scan");
    if (total > 0) {
        int blocks = (int)std::min<int64_t>((total + 255) / 256, 4 * 148 * 8);
        scatter_kernel<D><<<blocks, 256, 0, st>>>(src, d_off, nclouds, total, d_grids, d_start, d_fill,
                                                  d_sorted);
        KTRY(cudaGetLastError(), "scatter kernel");
    }
    if (nq > 0) {
        // the queries are the sources themselves (same array, same clouds)
        const bool self = qry == src && nq == total && (nclouds == 1 || h_q_off == h_src_off);
        launch_query<D>(qry, nq, d_qoff, nclouds, d_grids, d_start, d_sorted, k, self, idx, d2, st);
        KTRY(cudaGetLastError(), "query kernel");
    }
done:
#undef KTRY
    cudaFreeAsync(d_off, st);
    if (d_qoff) cudaFreeAsync(d_qoff, st);
    cudaFreeAsync(d_bbox, st);
    if (d_grids) cudaFreeAsync(d_grids, st);
    if (d_counts) cudaFreeAsync(d_counts, st);
    if (d_start) cudaFreeAsync(d_start, st);
    if (d_fill) cudaFreeAsync(d_fill, st);
    if (d_sorted) cudaFreeAsync(d_sorted, st);
    if (d_tmp) cudaFreeAsync(d_tmp, st);
    return rc;
}

}  // namespace

// internal entry used by the scene set-up (src and queries on the device)
int knn_device(const float* src, int64_t n, const float* qry, int64_t nq, int dim, int k, uint32_t* idx,
               float* d2, cudaStream_t st) {
    if (dim != 2 && dim != 3) return set_error(NAGA_EINVAL, "naga_knn: dim must be 2 or 3");
    if (k < 1 || k > 64) return set_error(NAGA_EINVAL, "naga_knn: k must be in [1, 64]");
    if (n < 0 || nq < 0 || n > (int64_t)0xfffffffe) return set_error(NAGA_EINVAL, "naga_knn: bad sizes");
    int64_t off[2] = {0, n};
    return dim == 2 ? knn_run<2>(src, off, 1, qry, nq, nullptr, k, idx, d2, st)
                    : knn_run<3>(src, off, 1, qry, nq, nullptr, k, idx, d2, st);
}

// ----------------------------------------------- allocation-free variant
// Some callers cannot call cudaMalloc once they are running: processes that
// hand all free device memory to their own caching allocator at start-up
// and run on a fixed budget, and latency-critical serving paths, where
// cudaMalloc / cudaFree may synchronise the device and stall every other
// stream. naga_knn_noalloc serves them: its scratch (cell grid, counting
// sort, sorted point records) lives in one file-scope device array that every
// GPU loading this library holds until the process exits. The array's
// host-side name is only a stand-in; its device address is looked up once
// per device with cudaGetSymbolAddress.
namespace {

constexpr int64_t kNoAllocMaxPoints = 65536;  // largest source cloud
constexpr int64_t kNoAllocMaxCells = 65536;   // cap on the cell grid

struct NoAllocScratch {
    int bbox[8];
    int64_t offsets[2];
    CloudGrid grid;
    unsigned counts[kNoAllocMaxCells + 1];
    unsigned start[kNoAllocMaxCells + 1];
    unsigned fill[kNoAllocMaxCells + 1];
    float4 sorted[kNoAllocMaxPoints];
};

static __device__ __align__(256) unsigned char g_knn_scratch[sizeof(NoAllocScratch)];

// device address of g_knn_scratch in the current context: looked up once
// per device and context, and again when the device's context changed (a
// cudaDeviceReset or a host framework resetting the primary context loads
// the module anew, and the array may move); without a context id the
// lookup is made on every call
int noalloc_scratch(NoAllocScratch** out) {
    static std::mutex mu;
    static void* addr[64] = {nullptr};
    static unsigned long long ctx_of[64] = {0};
    int dev = 0;
    NAGA_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_error(NAGA_EINVAL, "naga_knn_noalloc: device ordinal above 63");
    unsigned long long ctx = 0;
    const bool known = current_context_id(&ctx);
    std::lock_guard<std::mutex> lk(mu);
    if (!known || !addr[dev] || ctx_of[dev] != ctx) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_knn_scratch);
        if (e != cudaSuccess)
            return set_error(NAGA_ECUDA, std::string("naga_knn_noalloc: cudaGetSymbolAddress: ") +
                                             cudaGetErrorString(e));
        addr[dev] = known ? p : nullptr;
        ctx_of[dev] = ctx;
        *out = reinterpret_cast<NoAllocScratch*>(p);
        return NAGA_OK;
    }
    *out = reinterpret_cast<NoAllocScratch*>(addr[dev]);
    return NAGA_OK;
}

// resets what must start at zero and the bounding box of a new call
__global__ void noalloc_init_kernel(NoAllocScratch* s, int64_t n) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t t = t0; t <= kNoAllocMaxCells; t += (int64_t)gridDim.x * blockDim.x) {
        s->counts[t] = 0u;
        s->fill[t] = 0u;
    }
    if (t0 < 3) {
        s->bbox[t0] = 0x7fffffff;
        s->bbox[3 + t0] = (int)0x80000000;
    }
    if (t0 == 0) {
        s->offsets[0] = 0;
        s->offsets[1] = n;
    }
}

__global__ void noalloc_set_grid_kernel(NoAllocScratch* s, CloudGrid g) { s->grid = g; }

// exclusive scan of counts[0, m) into start[0, m) by one block
__global__ void noalloc_scan_kernel(NoAllocScratch* s, int m) {
    __shared__ unsigned part[1024];
    const int t = threadIdx.x;
    const int per = (m + blockDim.x - 1) / blockDim.x;
    const int b = t * per, e = min(m, b + per);
    unsigned acc = 0;
    for (int i = b; i < e; ++i) acc += s->counts[i];
    part[t] = acc;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {
        unsigned v = t >= o ? part[t - o] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    unsigned run = part[t] - acc;
    for (int i = b; i < e; ++i) {
        s->start[i] = run;
        run += s->counts[i];
    }
}

template <int D>
int knn_noalloc_run(const float* src, int64_t n, const float* qry, int64_t nq, int k, uint32_t* idx, float* d2,
                    cudaStream_t st) {
    NoAllocScratch* scr = nullptr;
    int rc = noalloc_scratch(&scr);
    if (rc) return rc;
    noalloc_init_kernel<<<64, 256, 0, st>>>(scr, n);
    NAGA_CUDA_TRY(cudaGetLastError());
    if (n > 0) {
        const int per = bbox_blocks_per_cloud(n, 1);
        bbox_kernel<D><<<(unsigned)per, 256, 0, st>>>(src, scr->offsets, per, scr->bbox);
        NAGA_CUDA_TRY(cudaGetLastError());
    }
    int hb[6];
    NAGA_CUDA_TRY(cudaMemcpyAsync(hb, scr->bbox, sizeof(hb), cudaMemcpyDeviceToHost, st));
    NAGA_CUDA_TRY(cudaStreamSynchronize(st));
    CloudGrid g{};
    double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, vol = 1;
    for (int d = 0; d < D; ++d) {
        lo[d] = n > 0 ? (double)ord2f(hb[d]) : 0.0;
        hi[d] = n > 0 ? (double)ord2f(hb[3 + d]) : 1.0;
        if (!std::isfinite(lo[d]) || !std::isfinite(hi[d]))
            return set_error(NAGA_EINVAL, "naga_knn_noalloc: non-finite point coordinates");
        if (hi[d] - lo[d] < 1e-6) hi[d] = lo[d] + 1e-6;
        vol *= hi[d] - lo[d];
    }
    double w = std::pow(2.0 * vol / (double)std::max<int64_t>(n, 1), 1.0 / D);
    int64_t cells = 0;
    for (;;) {
        cells = 1;
        for (int d = 0; d < 3; ++d) {
            const int64_t dd = d < D ? std::max<int64_t>(1, (int64_t)std::ceil((hi[d] - lo[d]) / w)) : 1;
            g.dims[d] = (int)std::min<int64_t>(dd, 1 << 20);
            cells *= g.dims[d];
        }
        if (cells <= kNoAllocMaxCells) break;
        w *= 1.25;  // coarser cells: the search stays exact, only slower
    }
    for (int d = 0; d < 3; ++d) g.lo[d] = lo[d];
    set_radius(g, w, n, D, k);
    g.cell_base = 0;
    g.pt_base = 0;
    g.n = n;
    noalloc_set_grid_kernel<<<1, 1, 0, st>>>(scr, g);
    if (n > 0) {
        const int blocks = (int)std::min<int64_t>((n + 255) / 256, 4 * 148 * 8);
        count_kernel<D><<<blocks, 256, 0, st>>>(src, scr->offsets, 1, n, &scr->grid, scr->counts);
        noalloc_scan_kernel<<<1, 1024, 0, st>>>(scr, (int)cells + 1);
        scatter_kernel<D><<<blocks, 256, 0, st>>>(src, scr->offsets, 1, n, &scr->grid, scr->start, scr->fill,
                                                  scr->sorted);
    } else {
        noalloc_scan_kernel<<<1, 1024, 0, st>>>(scr, (int)cells + 1);
    }
    NAGA_CUDA_TRY(cudaGetLastError());
    if (nq > 0) {
        launch_query<D>(qry, nq, nullptr, 1, &scr->grid, scr->start, scr->sorted, k, qry == src && nq == n, idx, d2,
                        st);
        NAGA_CUDA_TRY(cudaGetLastError());
    }
    return NAGA_OK;
}

}  // namespace

}  // namespace naga

using namespace naga;

extern "C" int naga_knn_noalloc(const float* src, int64_t n, const float* qry, int64_t nq, int dim, int k,
                                uint32_t* idx, float* d2, void* stream) {
    if (dim != 2 && dim != 3) return set_error(NAGA_EINVAL, "naga_knn_noalloc: dim must be 2 or 3");
    if (k < 1 || k > 64) return set_error(NAGA_EINVAL, "naga_knn_noalloc: k must be in [1, 64]");
    if (n < 0 || nq < 0) return set_error(NAGA_EINVAL, "naga_knn_noalloc: negative size");
    if (n > kNoAllocMaxPoints)
        return set_error(NAGA_EINVAL, "naga_knn_noalloc: " + std::to_string(n) +
                                          " source points exceed the fixed scratch of 65536 points; use naga_knn");
    if ((n > 0 && !src) || (nq > 0 && (!qry || !idx || !d2)))
        return set_error(NAGA_EINVAL, "naga_knn_noalloc: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    return dim == 2 ? knn_noalloc_run<2>(src, n, qry, nq, k, idx, d2, st)
                    : knn_noalloc_run<3>(src, n, qry, nq, k, idx, d2, st);
}

extern "C" int naga_knn(const float* src, int64_t n, const float* qry, int64_t nq, int dim, int k,
                        uint32_t* idx, float* d2, void* stream) {
    if ((n > 0 && !src) || (nq > 0 && (!qry || !idx || !d2)))
        return set_error(NAGA_EINVAL, "naga_knn: null pointer");
    return knn_device(src, n, qry, nq, dim, k, idx, d2, (cudaStream_t)stream);
}

extern "C" int naga_knn_clouds(const float* pts, const int64_t* offsets, int n_clouds, int dim, int k,
                               uint32_t* idx, float* d2, void* stream) {
    if (!offsets || n_clouds < 1) return set_error(NAGA_EINVAL, "naga_knn_clouds: bad offsets");
    if (dim != 2 && dim != 3) return set_error(NAGA_EINVAL, "naga_knn_clouds: dim must be 2 or 3");
    if (k < 1 || k > 64) return set_error(NAGA_EINVAL, "naga_knn_clouds: k must be in [1, 64]");
    for (int c = 0; c < n_clouds; ++c)
        if (offsets[c + 1] < offsets[c]) return set_error(NAGA_EINVAL, "naga_knn_clouds: offsets decrease");
    if (offsets[0] != 0) return set_error(NAGA_EINVAL, "naga_knn_clouds: offsets[0] must be 0");
    int64_t total = offsets[n_clouds];
    if (total > 0 && (!pts || !idx || !d2)) return set_error(NAGA_EINVAL, "naga_knn_clouds: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    return dim == 2 ? knn_run<2>(pts, offsets, n_clouds, pts, total, offsets, k, idx, d2, st)
                    : knn_run<3>(pts, offsets, n_clouds, pts, total, offsets, k, idx, d2, st);
}
