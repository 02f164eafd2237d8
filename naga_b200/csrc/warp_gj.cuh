// Gauss-Jordan solve of one augmented RBF moment system per warp, in
// registers.
//
// System: KC support rows [P | Phi] and E = D + 1 constraint rows [0 | P^T]
// (the polynomial columns first), NR right-hand sides. Lane l holds support
// row l. The E polynomial columns are eliminated first, where the constraint
// rows are zero: their E pivot rows then only determine the polynomial
// coefficients, which nobody asks for, so they are dropped and their lanes
// take the constraint rows. The KC support columns follow over exactly KC
// rows. This is LU with partial pivoting of the column-permuted system; no
// second, nearly empty row per lane goes through the elimination. (It rounds
// the RBF block at its full size E times more than an elimination that starts
// with the support columns.)
//
// Step j: the pivot of column j is the row of largest |a| among the rows not
// yet pivoted (magnitudes compared in their upper 15 bits of mantissa, by one
// warp maximum over keys that carry the row's number; rows within that of each
// other are equally good pivots: the error of the solution is the same to four
// digits as with all bits compared). Its owner publishes it in shared memory and
// every other row, pivoted ones too, subtracts its multiple: after the last
// step row r holds b / pivot for the column it was pivoted on, with no back
// substitution. Eliminating the pivoted rows costs no instruction: their lanes
// run the step anyway.
//
// Register columns rotate by one a step (register m holds column j + m), so
// no register is indexed by the step; the loop runs in phases whose width
// shrinks with the columns left. The next step's pivot key is taken as soon
// as its column is up to date, ahead of the rest of the update, so the
// warp-wide maximum overlaps it.
#pragma once
#include "common.cuh"

namespace naga {

template <int KC, int D, int NR>
struct GjSystem {
    static_assert(KC % 8 == 0 && KC <= 32, "one support row a lane, four phases of even width");
    static constexpr int E = D + 1;
    static constexpr int W = (E + KC + NR + 1) / 2 * 2;  // columns with the right-hand sides, even
    static constexpr int LD = KC + 2;                    // row stride of the assembly buffer (16-B rows, distinct banks)
    // per-warp shared memory, in doubles: assembly rows (the solution once
    // they are read); two published rows; the constraints' right-hand sides;
    // the support coordinates
    static constexpr int kAsm = KC * LD, kRow = 2 * W, kRhs = E * NR, kXs = KC * D;
    static constexpr int doubles = (kAsm + kRow + kRhs + kXs + 15) / 16 * 16;

    double a[W];   // this lane's row, rotating
    int mycol;     // column the row was pivoted on, -1 before
    double myinv;  // its reciprocal pivot
    unsigned best; // key of the next pivot (warp-uniform)

    // |column 0| without its lower 37 mantissa bits, then 31 - lane; 0 .. 31:
    // no candidate, or a zero
    __device__ __forceinline__ unsigned key() const {
        const int lane = lane_id();
        return lane < KC && mycol < 0 ? ((unsigned)__double2hiint(a[0]) & 0x7fffffe0u) | (unsigned)(31 - lane) : 0u;
    }

    // STEPS elimination steps from column j0, M registers wide
    template <int M, int STEPS>
    __device__ __forceinline__ bool phase(int j0, double* rows) {
        const int lane = lane_id();
        bool zero = false;
#pragma unroll 1
        for (int j = j0; j < j0 + STEPS; ++j) {
            double* const pr = rows + (j & 1) * W;
            const bool mine = lane == 31 - (int)(best & 31u);
            zero = zero || best < 32u;
            if (mine) {
#pragma unroll
                for (int m = 0; m < M; m += 2) *reinterpret_cast<double2*>(pr + m) = make_double2(a[m], a[m + 1]);
            }
            __syncwarp();
            const double2 p01 = *reinterpret_cast<const double2*>(pr);
            const double inv = 1.0 / p01.x;
            double f = -(a[0] * inv);
            if (mine) {
                f = 0.0;
                mycol = j;
                myinv = inv;
            }
            a[0] = fma(f, p01.y, a[1]);
            best = __reduce_max_sync(kFull, key());
#pragma unroll
            for (int m = 2; m < M; m += 2) {
                const double2 q = *reinterpret_cast<const double2*>(pr + m);
                a[m - 1] = fma(f, q.x, a[m]);
                a[m] = fma(f, q.y, a[m + 1 < M ? m + 1 : m]);
            }
        }
        return zero;
    }

    // The solution of the system whose support rows are in a (polynomial
    // columns, support columns, right-hand sides): sol[c NR + d] in shared
    // memory for the support columns c < KC. xs: the k support coordinates;
    // rhs[r NR + d]: the constraint rows' right-hand sides. True when a pivot
    // was zero.
    __device__ __forceinline__ bool solve(int k, const double* xs, const double* rhs, double* rows, double* sol) {
        mycol = -1;
        myinv = 0.0;
        best = __reduce_max_sync(kFull, key());
        bool zero = phase<W, E>(0, rows);
        if (mycol >= 0) {
            const int r = mycol;
#pragma unroll
            for (int c = 0; c < KC; ++c) a[c] = c < k ? (r == 0 ? 1.0 : xs[c * D + r - 1]) : 0.0;
#pragma unroll
            for (int d = 0; d < NR; ++d) a[KC + d] = rhs[r * NR + d];
            mycol = -1;
        }
        best = __reduce_max_sync(kFull, key());
        constexpr int S = KC / 4, M = (KC + NR + 1) / 2 * 2;
        zero |= phase<M, S>(E, rows);
        zero |= phase<M - S, S>(E + S, rows);
        zero |= phase<M - 2 * S, S>(E + 2 * S, rows);
        zero |= phase<M - 3 * S, S>(E + 3 * S, rows);
        if (mycol >= E) {
#pragma unroll
            for (int d = 0; d < NR; ++d) sol[(mycol - E) * NR + d] = a[d] * myinv;
        }
        __syncwarp();
        return zero;
    }
};

}  // namespace naga
