// column.cuh -- line solves of y and z lines held in columns of threads.
//
// A tile is TL lines that are neighbours in x (one 64- or 128-byte row of the
// field per point along the line).  Thread (l, c) = (tid % TL, tid / TL) owns
// chunk c of line l: it loads its LT points straight into registers (a warp's
// load of one row is coalesced, the addresses step by a constant), eliminates
// its chunk there and stores the solution from there.  Shared memory only
// carries what chunks need from each other: the field values at the chunks'
// ends for the stencils and the boundary rows, and the two end rows of each
// chunk's reduced system, which one warp per line solves with the shuffles of
// reduced_solve.  Against staging whole lines through a transposing layout
// (one warp per line), that leaves out a store and a load per point, all
// per-point index arithmetic and the idle lanes of short lines; the
// arithmetic of every row is the same.
#pragma once

#include "line_solver.cuh"
#include "tile.cuh"

namespace csb {

// Shared-memory slots of one field of a tile: row t of chunk c of line l.  The
// odd chunk stride lets a warp read one line's 32 chunk ends without bank
// conflicts, and threads (l, c) write their rows with at most a 2-way one.
template <int LT, int TL>
struct Column {
    static constexpr int kChunk = TL + 1;
    static constexpr int kRow = 32 * kChunk;
    static constexpr int kField = LT * kRow;
    __device__ __forceinline__ static int at(int t, int c, int l) { return t * kRow + c * kChunk + l; }
    __device__ __forceinline__ static int pos(int j, int l) { return at(j % LT, j / LT, l); }
};

// Threads of a column tile for lines of p chunks (whole warps).
inline int column_threads(int tl, int p) { return (tl * p + 31) / 32 * 32; }

// The boundary rows of the interface closure for every line of a tile of NF
// fields (V: raw field values, all written): rows[(f TL + l) 4 + k] = rows 0,
// 1, n-1, n-2 of the right-hand side (the last two without their sign).  Eight
// neighbouring threads form the eight 8-term sums of one line (interface_sum's
// operations), then two of them are added.  recv != nullptr: the far-end sums
// are received values recv[k F + line] instead.  All threads of the tile call
// it; the caller synchronizes before the rows are read.
template <int LT, int TL, int NF, typename T>
__device__ __forceinline__ void column_closure_rows(const T *V, T *rows, int n, const Coeffs &cf, const T *recv,
                                                    int64_t F, int64_t line0) {
    using C = Column<LT, TL>;
    static_assert(NF * TL * 8 % 32 == 0, "whole warps");
    for (int i = threadIdx.x; i < NF * TL * 8; i += blockDim.x) {
        const int g = i >> 3, d = i & 7, f = g / TL, l = g % TL;
        T dv = T(0);
        if (recv && (d & 2)) {
            if (line0 + l < F) dv = recv[(int64_t)((d >> 1 & 2) | (d & 1)) * F + line0 + l];
        } else {
            const bool bci = d < 2 || d == 4 || d == 5, asc = d < 2 || d >= 6, second = (d & 1) != 0;
            const T *line = V + f * C::kField;
#pragma unroll
            for (int k = 0; k < kLmd; ++k) {
                const double w = bci ? (second ? cf.pbci[kLmd + k] : cf.pbci[k])
                                     : (second ? cf.pbco[kLmd + k] : cf.pbco[k]);
                dv += xmul(T(w), line[C::pos(asc ? k : n - 1 - k, l)]);
            }
        }
        const T x = dv + __shfl_down_sync(0xffffffffu, dv, 2);
        if (!(d & 2)) rows[g * 4 + ((d >> 2) * 2 | (d & 1))] = x;
    }
}

// Right-hand side of the compact derivative for this thread's chunk: d holds
// its field values on entry; the two points on either side come from V.  Rows
// of the physical closure are formed here; rows of the interface closure are
// put in by column_take_rows once column_closure_rows has run.  Slots outside
// the line are read but only reach rows that are replaced.
template <int LT, int TL, typename T>
__device__ __forceinline__ void column_rhs(const T *V, int c, int l, int n, int nstart, int nend, T (&d)[LT]) {
    using C = Column<LT, TL>;
    const int cm = c > 0 ? c - 1 : 0, cp = c < 31 ? c + 1 : 31;
    T w[LT + 4];
    w[0] = V[C::at(LT - 2, cm, l)];
    w[1] = V[C::at(LT - 1, cm, l)];
    w[LT + 2] = V[C::at(0, cp, l)];
    w[LT + 3] = V[C::at(1, cp, l)];
#pragma unroll
    for (int t = 0; t < LT; ++t) w[t + 2] = d[t];
    chunk_rhs<LT, T>(w, c, n, nstart, nend, d);
}

// Put the interface closure rows of line l (rows: its four entries) into d.
template <int LT, typename T>
__device__ __forceinline__ void column_take_rows(const T *rows, int c, int n, int nstart, int nend, T (&d)[LT]) {
    if (nstart && c == 0) {
        d[0] = rows[0];
        d[1] = rows[1];
    }
    if (nend) {
        if (c == (n - 1) / LT) set_at<LT, T>(d, (n - 1) - c * LT, -rows[2]);
        if (c == (n - 2) / LT) set_at<LT, T>(d, (n - 2) - c * LT, -rows[3]);
    }
}

// Write an eliminated chunk's end rows where the line's warp reads them.
template <int LT, int TL, typename T>
__device__ __forceinline__ void column_put_ends(T *V, const T (&d)[LT], int c, int l, int len) {
    using C = Column<LT, TL>;
    if (len == LT) {
        V[C::at(0, c, l)] = d[0];
        V[C::at(LT - 1, c, l)] = d[LT - 1];
    } else if (len > 0) {
        V[C::at(0, c, l)] = d[0];
        if (len >= 2) V[C::at(len - 1, c, l)] = get_at<LT, T>(d, len - 1);
    }
}

// Solve the reduced systems of the tile's lines, one warp per line, in place
// of the chunks' end rows.  beta != nullptr (cyclic systems): the factor of
// the Sherman-Morrison correction per field and line.
template <int LT, int TL, int NF, typename T>
__device__ __forceinline__ void column_reduced(T *V, const DevTables<T> &tab, int64_t F, int64_t line0, T *beta) {
    using C = Column<LT, TL>;
    const int lane = threadIdx.x & 31, len = lane_len(lane, LT, tab.p, tab.last_len);
    for (int l = threadIdx.x >> 5; l < TL; l += blockDim.x >> 5) {
        if (line0 + l >= F) break;
        T y0[NF], y1[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            y0[f] = len >= 1 ? V[f * C::kField + C::at(0, lane, l)] : T(0);
            y1[f] = len >= 2 ? V[f * C::kField + C::at(len - 1, lane, l)] : T(0);
        }
        reduced_solve<NF, T>(tab, y0, y1, lane);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (len >= 1) V[f * C::kField + C::at(0, lane, l)] = y0[f];
            if (len >= 2) V[f * C::kField + C::at(len - 1, lane, l)] = y1[f];
            if (beta) {
                const T ya = __shfl_sync(0xffffffffu, y0[f], 0);
                const T yb = __shfl_sync(0xffffffffu, len >= 2 ? y1[f] : y0[f], tab.p - 1);
                if (lane == 0) beta[f * TL + l] = (ya + tab.cyc_s2 * yb) * tab.cyc_s1;
            }
        }
    }
}

// The solution of this thread's chunk from its end values in V.
template <int LT, int TL, typename T>
__device__ __forceinline__ void column_finish(const T *V, const DevTables<T> &tab, int c, int l, int len, T (&d)[LT]) {
    using C = Column<LT, TL>;
    const T X0 = len >= 1 ? V[C::at(0, c, l)] : T(0);
    const T X1 = len >= 2 ? V[C::at(len - 1, c, l)] : T(0);
    chunk_substitute<LT, T>(tab, d, X0, X1, c, len);
}

}  // namespace csb
