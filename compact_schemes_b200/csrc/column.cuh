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
// P: chunk slots per line (lines of at most P chunks).
template <int LT, int TL, int P = 32>
struct Column {
    static constexpr int kChunk = TL + 1;
    static constexpr int kRow = P * kChunk;
    static constexpr int kSlots = P;
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
// are received values recv[k F + line0 + f TL + l] instead (the fields are then
// TL-line groups of one field).  CT: type the sums are formed in.  All threads of the tile call it; the caller
// synchronizes before the rows are read.
template <int LT, int TL, int NF, typename T, typename CT = T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_closure_rows(const T *V, CT *rows, int n, const Coeffs &cf, const CT *recv,
                                                    int F, int line0) {
    static_assert(NF * TL * 8 % 32 == 0, "whole warps");
    for (int i = threadIdx.x; i < NF * TL * 8; i += blockDim.x) {
        const int g = i >> 3, d = i & 7, f = g / TL, l = g % TL;
        CT dv = CT(0);
        if (recv && (d & 2)) {
            if (line0 + g < F) dv = recv[(int64_t)((d >> 1 & 2) | (d & 1)) * F + line0 + g];
        } else {
            const bool bci = d < 2 || d == 4 || d == 5, asc = d < 2 || d >= 6, second = (d & 1) != 0;
            const T *line = V + f * C::kField;
#pragma unroll
            for (int k = 0; k < kLmd; ++k) {
                const double w = bci ? (second ? cf.pbci[kLmd + k] : cf.pbci[k])
                                     : (second ? cf.pbco[kLmd + k] : cf.pbco[k]);
                dv += xmul(CT(w), CT(line[C::pos(asc ? k : n - 1 - k, l)]));
            }
        }
        const CT x = dv + __shfl_down_sync(0xffffffffu, dv, 2);
        if (!(d & 2)) rows[g * 4 + ((d >> 2) * 2 | (d & 1))] = x;
    }
}

// Write the rows of a chunk that other threads read: the two at either end
// (the neighbours' stencils), all of them near the line's ends (the closure).
template <int LT, int TL, typename T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_put_raw(T *V, const T (&d)[LT], int c, int l, int n) {
    V[C::at(0, c, l)] = d[0];
    V[C::at(1, c, l)] = d[1];
    if (LT > 2) V[C::at(LT - 2, c, l)] = d[LT - 2];
    if (LT > 3) V[C::at(LT - 1, c, l)] = d[LT - 1];
    if (LT > 4 && (c * LT < kLmd || (c + 1) * LT > n - kLmd)) {
#pragma unroll
        for (int t = 2; t < LT - 2; ++t) V[C::at(t, c, l)] = d[t];
    }
}

// Right-hand side of the compact derivative for this thread's chunk (len rows):
// d holds its field values on entry; the two points on either side come from V.
// Rows of the physical closure are formed here; rows of the interface closure
// are put in by column_take_rows once column_closure_rows has run.  Slots
// outside the line are read but only reach rows that are replaced.
template <int LT, int TL, typename T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_rhs(const T *V, int c, int l, int len, int n, int nstart, int nend,
                                           T (&d)[LT]) {
    const int cm = c > 0 ? c - 1 : 0, cp = c < C::kSlots - 1 ? c + 1 : C::kSlots - 1;
    T w[LT + 4];
    w[0] = V[C::at(LT - 2, cm, l)];
    w[1] = V[C::at(LT - 1, cm, l)];
    w[LT + 2] = V[C::at(0, cp, l)];
    w[LT + 3] = V[C::at(1, cp, l)];
#pragma unroll
    for (int t = 0; t < LT; ++t) w[t + 2] = d[t];
    chunk_rhs<LT, T>(w, c, len, n, nstart, nend, d);
}

// Put the interface closure rows of a line (rows: its four entries) into d.
template <int LT, typename T>
__device__ __forceinline__ void column_take_rows(const T *rows, int c, int n, int nstart, int nend, T (&d)[LT]) {
    if (c == 0 || (c + 1) * LT >= n - 1)
        chunk_take_rows<LT, T>(rows[0], rows[1], rows[2], rows[3], c, n, nstart, nend, d);
}

// Write an eliminated chunk's end rows where the line's warp reads them.
template <int LT, int TL, typename T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_put_ends(T *V, const T (&d)[LT], int c, int l, int len) {
    V[C::at(0, c, l)] = d[0];
    if (len == LT) V[C::at(LT - 1, c, l)] = d[LT - 1];
    else if (len >= 2) V[C::at(len - 1, c, l)] = get_at<LT, T>(d, len - 1);
}

// Solve the reduced systems of the tile's lines, one warp per line (all NF
// fields of it together), in place of the chunks' end rows.  beta != nullptr
// (cyclic systems): the factor of the Sherman-Morrison correction per field and
// line.
template <int LT, int TL, int NF, typename T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_reduced(T *V, const DevTables<T> &tab, T *beta = nullptr) {
    const int lane = threadIdx.x & 31, len = lane_len(lane, LT, tab.p, tab.last_len);
    for (int l = threadIdx.x >> 5; l < TL; l += blockDim.x >> 5) {
        T *lo = V + C::at(0, lane, l), *hi = V + C::at(len >= 2 ? len - 1 : 0, lane, l);
        T y0[NF], y1[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            y0[f] = len >= 1 ? lo[f * C::kField] : T(0);
            y1[f] = len >= 2 ? hi[f * C::kField] : T(0);
        }
        reduced_solve<NF, T>(tab, y0, y1, lane);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (len >= 1) lo[f * C::kField] = y0[f];
            if (len >= 2) hi[f * C::kField] = y1[f];
            if (beta) {
                const T ya = __shfl_sync(0xffffffffu, y0[f], 0);
                const T yb = __shfl_sync(0xffffffffu, len >= 2 ? y1[f] : y0[f], tab.p - 1);
                if (lane == 0) beta[f * TL + l] = (ya + tab.cyc_s2 * yb) * tab.cyc_s1;
            }
        }
    }
}

// The solution of this thread's chunk from its end values in V.
template <int LT, int TL, typename T, typename C = Column<LT, TL>>
__device__ __forceinline__ void column_finish(const T *V, const DevTables<T> &tab, int c, int l, int len, T (&d)[LT]) {
    const T X0 = V[C::at(0, c, l)];
    const T X1 = V[C::at(len >= 2 ? len - 1 : 0, c, l)];
    chunk_substitute<LT, T>(tab, d, X0, X1, c, len);
}

// ----------------------------------------------------------------------------
// Lines of 65 to 128 points, one field at a time: four neighbouring lines per
// warp, lane 4 c + l holding chunk c (16 rows, at most 8 chunks) of line l in
// registers.  A row of the tile is one 32-byte sector; neighbours and the
// reduced system go by shuffle, so a warp needs no other warp and no barrier,
// and the reduced system takes 3 steps on an eighth of the rows.
// ----------------------------------------------------------------------------
constexpr int kWarpLines = 4;
constexpr int kWarpChunk = 16;
// Lines that fit it: shorter ones leave too few rows per lane to pay for its
// serial sweeps (64^3: 5.8 us against 4.9 us), longer ones need 32-row chunks, whose
// registers allow only 16 warps per SM (256^3: 83 against 78 us).
__host__ __device__ constexpr bool warp_column(int n) { return n > 64 && n <= 8 * kWarpChunk; }
// ... and whether a launch of `lines` lines of them is faster with it than with the
// column tiles below (two lines a thread, chunks of 4 rows).  The lane's serial
// sweeps take 8 us where the tiles take 5, so it needs half a wave of lines (96 an
// SM: three CTAs of 32) to be busy with.  With the table-driven factors a second
// wave costs as much as the first and pays again once it is full; the interior
// factors (interface closure, full chunks) leave room for it.  FP64 derivatives of
// one field of 72- to 128-point lines, us, column tiles / four lines a warp:
//   lines            2304     6400       9216      16384      35000  166464
//   interior      5.2/5.9  6.3/6.7   11.7/7.4  15.5/13.4  32.2/21.0  116/83
//   table-driven  5.4/8.9  6.3/9.6  11.8/10.0  16.6/17.6  28.0/28.3 120/113
// Single precision gains only from the interior factors on large fields (112-point
// lines: 36864 lines 18.9 / 17.1, 18496 lines 10.3 / 11.5 us).
inline bool warp_column_pays(int n, int nstart, int nend, int64_t lines, int nsm, int bytes) {
    const bool interior = nstart && nend && n % kWarpChunk == 0;
    const int64_t wave = (int64_t)96 * nsm;
    if (!warp_column(n)) return false;
    if (bytes == 4) return interior && lines > 2 * wave;
    return 2 * lines >= wave && (interior || lines <= wave || lines > 2 * wave);
}

// Right-hand side of a lane's chunk from its field values d; ends: this warp's
// [4][17] end points in shared memory; far: the received far-end sum that this
// lane's closure sum uses instead (or null).
template <int LT, typename T>
__device__ __forceinline__ void warp_column_rhs(T (*ends)[2 * kLmd + 1], int lane, int len, int n, int nstart, int nend,
                                                const Coeffs &cf, const T *far, T (&d)[1][LT]) {
    const int c = lane / kWarpLines, l = lane % kWarpLines;
    T rows = T(0);
    if (nstart || nend) {
        chunk_put_ends<LT, 1, T>(ends + l, d, c, len, n);
        __syncwarp();
        rows = ends_closure_row<T>(ends[lane >> 3], lane & 7, cf, far);
    }
    T x[LT + 4];
    x[0] = __shfl_up_sync(0xffffffffu, d[0][LT - 2], kWarpLines);
    x[1] = __shfl_up_sync(0xffffffffu, d[0][LT - 1], kWarpLines);
    x[LT + 2] = __shfl_down_sync(0xffffffffu, d[0][0], kWarpLines);
    x[LT + 3] = __shfl_down_sync(0xffffffffu, d[0][1], kWarpLines);
#pragma unroll
    for (int t = 0; t < LT; ++t) x[t + 2] = d[0][t];
    chunk_rhs<LT, T>(x, c, len, n, nstart, nend, d[0]);
    if (nstart || nend) {
        // all four: a short line's first chunk can hold its last rows too
        const T r0 = __shfl_sync(0xffffffffu, rows, 8 * l), r1 = __shfl_sync(0xffffffffu, rows, 8 * l + 1);
        const T r2 = __shfl_sync(0xffffffffu, rows, 8 * l + 4), r3 = __shfl_sync(0xffffffffu, rows, 8 * l + 5);
        chunk_take_rows<LT, T>(r0, r1, r2, r3, c, n, nstart, nend, d[0]);
    }
}

// Solve the four lines of the warp in place.
template <int LT, typename T>
__device__ __forceinline__ void warp_column_solve(const DevTables<T> &tab, int lane, int len, T (&d)[1][LT]) {
    const int c = lane / kWarpLines;
    chunk_eliminate<LT, 1, T>(tab, d, c);
    T y0[1] = {d[0][0]}, y1[1];
    if (len == LT) y1[0] = d[0][LT - 1];
    else y1[0] = len >= 2 ? get_at<LT, T>(d[0], len - 1) : T(0);
    reduced_solve<1, T, 32, kWarpLines>(tab, y0, y1, c);
    chunk_substitute<LT, T>(tab, d[0], y0[0], y1[0], c, len);
}

}  // namespace csb
