// numerics.cu -- compact derivative / filter line solves and the numerics_*
// C-ABI (replaces src/numerics_base.hpp, src/numerics_pc.hpp,
// src/numerics_rtc.hpp and src/cuda/kernels/numerics_*.hpp of the reference).
//
// Derivatives: along x a warp solves one or two lines, each lane loading its own
// chunks as vectors (k_deriv_row) or, for rows of any length and start and for
// chunks too long for that, the warp staging its lines in shared memory with
// 256-byte coalesced accesses (k_deriv_row_any).  Along y and z threads load their
// chunks of a tile of neighbouring lines straight into registers (k_deriv_col,
// column.cuh), or four lines share a warp (k_deriv_wcol).  blockIdx.y is the field.
// The filter stages a tile of 8 lines in shared memory (LineLayout order), one warp
// solving each line.
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "column.cuh"
#include "context.h"

namespace csb {

static thread_local char g_err[512] = "";

int set_error(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
    return code;
}

int check_cuda(cudaError_t e, const char *what) {
    return set_error(CS_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

TableCache::~TableCache() {
    for (auto &kv : map_) {
        if (kv.second->d64) cudaFree(kv.second->d64);
        if (kv.second->d32) cudaFree(kv.second->d32);
        delete kv.second;
    }
}

// Whether every lane's per-row factors equal the compile-time interior_chunk
// values (exact comparison): the line's chunks are all full and hold only the
// constant interior rows.
template <int LT>
static bool interior_match(const HostTables &h) {
    constexpr InteriorChunk<LT> K = interior_chunk<LT>();
    const std::vector<double> *tabs[6] = {&h.fwd1, &h.fwd2, &h.bwd1, &h.bwd2, &h.rca, &h.rcc};
    const double *ref[6] = {K.fwd1, K.fwd2, K.bwd1, K.bwd2, K.rca, K.rcc};
    for (int k = 0; k < 6; ++k)
        for (int t = 0; t < LT; ++t)
            for (int lane = 0; lane < h.p; ++lane)
                if ((*tabs[k])[(size_t)t * 32 + lane] != ref[k][t]) return false;
    return true;
}
static bool interior_tables(const HostTables &h) {
    if (h.cyclic || h.n != h.p * h.lt || h.p < 2) return false;
    switch (h.lt) {
        case 2: return interior_match<2>(h);
        case 4: return interior_match<4>(h);
        case 8: return interior_match<8>(h);
        case 16: return interior_match<16>(h);
        case 32: return interior_match<32>(h);
    }
    return false;
}

template <typename CT>
static void bind(DevTables<CT> &t, CT *base, const HostTables &h) {
    const size_t tl = (size_t)h.lt * 32;
    t.fwd1 = base;
    t.fwd2 = base + tl;
    t.bwd1 = base + 2 * tl;
    t.bwd2 = base + 3 * tl;
    t.rca = base + 4 * tl;
    t.rcc = base + 5 * tl;
    t.k1 = base + 6 * tl;
    t.k2 = base + 6 * tl + 384;
    t.invb = base + 6 * tl + 768;
    t.cycz = base + 6 * tl + 832;
    t.cyc_s1 = (CT)h.cyc_s1;
    t.cyc_s2 = (CT)h.cyc_s2;
    t.n = h.n;
    t.p = h.p;
    t.last_len = h.last_len;
    t.cyclic = h.cyclic ? 1 : 0;
    t.pcr = sizeof(CT) == 4 ? h.pcr32 : h.pcr64;
    t.interior = interior_tables(h) ? 1 : 0;
}

// Device layout of the tables; fp32 selects the inverse diagonals of the
// FP32 PCR depth.
static std::vector<double> pack(const HostTables &h, bool fp32 = false) {
    std::vector<double> v;
    for (auto *a : {&h.fwd1, &h.fwd2, &h.bwd1, &h.bwd2, &h.rca, &h.rcc, &h.k1, &h.k2, fp32 ? &h.invb32 : &h.invb})
        v.insert(v.end(), a->begin(), a->end());
    if (h.cyclic) v.insert(v.end(), h.cycz.begin(), h.cycz.end());
    else v.insert(v.end(), (size_t)h.lt * 32, 0.0);
    return v;
}

// Whether all lanes of a table set share lane 0's per-row chunk factors
// (every chunk full, no cyclic correction), and those factors in FP32.  The
// comparison is exact, so a line qualifies only when its tables say so.
static void chunk_factors(const HostTables &h, bool &uniform, float *cfu) {
    uniform = !h.cyclic && h.lt <= 32 && h.n == h.p * h.lt && h.p >= 2;
    const std::vector<double> *tabs[6] = {&h.fwd1, &h.fwd2, &h.bwd1, &h.bwd2, &h.rca, &h.rcc};
    for (int k = 0; k < 6 && uniform; ++k)
        for (int t = 0; t < h.lt && uniform; ++t)
            for (int lane = 1; lane < h.p; ++lane)
                if ((*tabs[k])[(size_t)t * 32 + lane] != (*tabs[k])[(size_t)t * 32]) {
                    uniform = false;
                    break;
                }
    if (!uniform) return;
    for (int k = 0; k < 6; ++k)
        for (int t = 0; t < h.lt; ++t) {
            const double v = (*tabs[k])[(size_t)t * 32];
            cfu[k * h.lt + t] = (float)(k >= 4 ? -v : v);
        }
}

static bool host_tables_for(int n, int scheme, int nstart, int nend, double af, HostTables &h, int min_lt = 2) {
    std::vector<double> a(n), b(n), c(n);
    bool cyclic = false;
    if (scheme == kDeriv) {
        deriv_rows(n, nstart, nend, a.data(), b.data(), c.data());
    } else if (scheme == kDerivT) {
        std::vector<double> a0(n), c0(n);
        deriv_rows(n, nstart, nend, a0.data(), b.data(), c0.data());
        for (int i = 0; i < n; ++i) {
            a[i] = i > 0 ? c0[i - 1] : 0.0;
            c[i] = i < n - 1 ? a0[i + 1] : 0.0;
        }
    } else {
        cyclic = nstart && nend;
        filter_rows(n, cyclic, af, a.data(), b.data(), c.data());
        if (scheme == kFilterT && !cyclic) {  // the cyclic filter matrix is symmetric
            std::vector<double> a0(a), c0(c);
            for (int i = 0; i < n; ++i) {
                a[i] = i > 0 ? c0[i - 1] : 0.0;
                c[i] = i < n - 1 ? a0[i + 1] : 0.0;
            }
        }
    }
    return build_tables(n, a.data(), b.data(), c.data(), cyclic, h, min_lt);
}

const DeviceTables *TableCache::get(int n, int scheme, int nstart, int nend, double af, int min_lt) {
    uint64_t bits = 0;
    if (scheme == kFilter || scheme == kFilterT) std::memcpy(&bits, &af, sizeof bits);
    TableKey key{n, scheme, nstart ? 1 : 0, nend ? 1 : 0, bits, min_lt};
    std::lock_guard<std::mutex> lk(mu_);
    auto it = map_.find(key);
    if (it != map_.end()) return it->second;
    auto *dt = new DeviceTables();
    if (!host_tables_for(n, scheme, nstart, nend, af, dt->host, min_lt)) {
        delete dt;
        set_error(CS_ERR_UNSUPPORTED, "line length %d outside [5, %d]", n, kMaxLine);
        return nullptr;
    }
    std::vector<double> v = pack(dt->host);
    const std::vector<double> v32 = pack(dt->host, true);
    std::vector<float> vf(v32.begin(), v32.end());
    if (cudaMalloc(&dt->d64, v.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&dt->d32, vf.size() * sizeof(float)) != cudaSuccess ||
        cudaMemcpy(dt->d64, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dt->d32, vf.data(), vf.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
        if (dt->d64) cudaFree(dt->d64);
        if (dt->d32) cudaFree(dt->d32);
        delete dt;
        set_error(CS_ERR_ALLOC, "line-solver table upload failed");
        return nullptr;
    }
    bind(dt->t64, dt->d64, dt->host);
    bind(dt->t32, dt->d32, dt->host);
    dt->lt = dt->host.lt;
    chunk_factors(dt->host, dt->uniform, dt->cfu);
    map_[key] = dt;
    return dt;
}

// ----------------------------------------------------------------------------
// kernels
// ----------------------------------------------------------------------------
// Stage the tile's lines into shared memory.
template <int LT, int AXIS, typename T>
__device__ __forceinline__ void load_tile(const T *__restrict__ in, T *sm, int64_t line0, int64_t F,
                                          int n, int lxi, int let) {
    using L = LineLayout<LT>;
    const int tid = threadIdx.x;
    if (AXIS == 0) {
        const int w = tid >> 5, lane = tid & 31;
        const int64_t fidx = line0 + w;
        if (fidx < F) {
            const T *src = in + fidx * n;
            for (int j = lane; j < n; j += 32) sm[w * L::kSlot + L::pos(j)] = src[j];
        }
    } else {
        const int l = tid % kTileLines;
        const int64_t fidx = line0 + l;
        if (fidx < F) {
            const int64_t base = line_base<AXIS>(fidx, lxi, let), s = line_stride<AXIS>(lxi, let);
            for (int j = tid / kTileLines; j < n; j += kThreads / kTileLines)
                sm[l * L::kSlot + L::pos(j)] = in[base + j * s];
        }
    }
}

template <int LT, int AXIS, typename T>
__device__ __forceinline__ void store_tile(T *__restrict__ out, const T *sm, int64_t line0, int64_t F,
                                           int n, int lxi, int let) {
    using L = LineLayout<LT>;
    const int tid = threadIdx.x;
    if (AXIS == 0) {
        const int w = tid >> 5, lane = tid & 31;
        const int64_t fidx = line0 + w;
        if (fidx < F) {
            T *dst = out + fidx * n;
            for (int j = lane; j < n; j += 32) dst[j] = sm[w * L::kSlot + L::pos(j)];
        }
    } else {
        const int l = tid % kTileLines;
        const int64_t fidx = line0 + l;
        if (fidx < F) {
            const int64_t base = line_base<AXIS>(fidx, lxi, let), s = line_stride<AXIS>(lxi, let);
            for (int j = tid / kTileLines; j < n; j += kThreads / kTileLines)
                out[base + j * s] = sm[l * L::kSlot + L::pos(j)];
        }
    }
}

template <int LT, typename T>
__device__ __forceinline__ void store_line_regs(T *line, const T (&d)[LT], int lane, int n) {
    using L = LineLayout<LT>;
#pragma unroll
    for (int t = 0; t < LT; ++t)
        if (lane * LT + t < n) line[L::pos_ct(lane, t)] = d[t];
}

// The fields one derivative launch covers (blockIdx.y): field f is
// in[f * in_fs + .] -> out[f * out_fs + .], line-end values at drva + f F and
// received sums at recv + 4 f F (either may be null).
template <typename T>
struct FieldSet {
    const T *in;
    T *out;
    const T *recv;
    T *drva;
    int64_t in_fs, out_fs;
};

// Compact first derivative along x (deriv_kernel_1d/2d,
// src/cuda/kernels/numerics_pc.hpp:124-249) of rows whose length and start are
// multiples of VB bytes: a warp solves NV neighbouring lines, each lane loading
// its own chunks with VB-byte vectors and storing the solution from the same
// registers.  Neighbouring points come by shuffle, and only the eight points
// at either end of a line pass through shared memory (the interface sums).
template <int LT, int NV, int VB, typename T>
__global__ void __launch_bounds__(kThreads, LT <= 8 ? 3 : (LT == 16 ? 2 : 1))
k_deriv_row(FieldSet<T> fs, DevTables<T> tab, int nstart, int nend, int64_t F, Coeffs cf) {
    constexpr int VE = VB / (int)sizeof(T);
    __shared__ T ends[kThreads / 32][NV][2 * kLmd + 1];
    const int n = tab.n, w = threadIdx.x >> 5, lane = threadIdx.x & 31, j0 = lane * LT;
    const int64_t line0 = ((int64_t)blockIdx.x * (kThreads / 32) + w) * NV;
    if (line0 >= F) return;
    const int len = lane_len(lane, LT, tab.p, tab.last_len);
    const T *in = fs.in + blockIdx.y * fs.in_fs + line0 * n + j0;
    T *out = fs.out + blockIdx.y * fs.out_fs + line0 * n + j0;
    T d[NV][LT];
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        // past the last line: the last line again, not stored
        const T *src = in + (line0 + h < F ? h : 0) * (int64_t)n;
#pragma unroll
        for (int t = 0; t < LT; t += VE) {
            if (t < len) {
                load_vec<VB, T>(src + t, &d[h][t]);
            } else {
#pragma unroll
                for (int k = 0; k < VE; ++k) d[h][t + k] = T(0);
            }
        }
    }
    T rows = T(0);  // lane 8 h + {0, 1, 4, 5}: interface rows 0, 1, n-1, n-2 of line h
    if (nstart || nend) {
        chunk_put_ends<LT, NV, T>(ends[w], d, lane, len, n);
        __syncwarp();
        const int h = lane >> 3, k8 = lane & 7;
        T far = T(0);
        if (fs.recv && (k8 & 2) && h < NV && line0 + h < F)
            far = fs.recv[((int64_t)blockIdx.y * 4 + ((k8 >> 1 & 2) | (k8 & 1))) * F + line0 + h];
        rows = ends_closure_row<T>(ends[w][h < NV ? h : 0], k8, cf, fs.recv ? &far : nullptr);
    }
#pragma unroll
    for (int h = 0; h < NV; ++h) chunk_warp_rhs<LT, T>(rows, h, lane, len, n, nstart, nend, d[h]);
    warp_solve<LT, NV, T>(tab, d, lane);
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (line0 + h >= F) break;
        if (fs.drva) {
            T *dr = fs.drva + blockIdx.y * F + line0 + h;
            if (lane == 0) dr[0] = d[h][0];
            if (lane == (n - 1) / LT) dr[5 * F] = get_at<LT, T>(d[h], (n - 1) - j0);
        }
#pragma unroll
        for (int t = 0; t < LT; t += VE)
            if (t < len) store_vec<VB, T>(out + (int64_t)h * n + t, &d[h][t]);
    }
}

// The same for x rows of any length and start: a warp stages NV lines in
// shared memory (LineLayout) with 256-byte coalesced accesses and solves them
// from there.
template <int LT, int NV, typename T>
__global__ void __launch_bounds__(kThreads, LT <= 8 ? 3 : (LT == 16 || sizeof(T) == 4 ? 2 : 1))
k_deriv_row_any(FieldSet<T> fs, DevTables<T> tab, int nstart, int nend, int64_t F, Coeffs cf) {
    using L = LineLayout<LT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = tab.n, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T *sm = reinterpret_cast<T *>(smem_raw) + w * NV * L::kSlot;
    const int64_t line0 = ((int64_t)blockIdx.x * (kThreads / 32) + w) * NV;
    if (line0 >= F) return;
    const T *in = fs.in + blockIdx.y * fs.in_fs + line0 * n;
    T *out = fs.out + blockIdx.y * fs.out_fs + line0 * n;
    const int nl = F - line0 < NV ? (int)(F - line0) : NV;
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (h >= nl) break;
        for (int j = lane; j < n; j += 32) sm[h * L::kSlot + L::pos(j)] = in[(int64_t)h * n + j];
    }
    __syncwarp();
    T d[NV][LT];
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (h < nl) {
            T r4[4];
            const T *rp = nullptr;
            if (fs.recv && (nstart || nend)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) r4[k] = fs.recv[((int64_t)blockIdx.y * 4 + k) * F + line0 + h];
                rp = r4;
            }
            deriv_rhs<LT, T, T>(sm + h * L::kSlot, n, lane, nstart, nend, rp, cf, d[h]);
        } else {
#pragma unroll
            for (int t = 0; t < LT; ++t) d[h][t] = T(0);
        }
    }
    warp_solve<LT, NV, T>(tab, d, lane);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (h >= nl) break;
        if (fs.drva) {
            T *dr = fs.drva + blockIdx.y * F + line0 + h;
            if (lane == 0) dr[0] = d[h][0];
            if (lane == (n - 1) / LT) dr[5 * F] = get_at<LT, T>(d[h], (n - 1) - lane * LT);
        }
        store_line_regs<LT, T>(sm + h * L::kSlot, d[h], lane, n);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        if (h >= nl) break;
        for (int j = lane; j < n; j += 32) out[(int64_t)h * n + j] = sm[h * L::kSlot + L::pos(j)];
    }
}

// The same along y and z for the lines of warp_column (column.cuh): four lines
// per warp.  SUM: also sum[f] = (add0[f] + add1[f]) +
// derivative, the right-hand side of calc_fluxes from its last derivative.
template <int LT, int AXIS, typename T, bool SUM>
__global__ void __launch_bounds__(kThreads, 3)
k_deriv_wcol(FieldSet<T> fs, DevTables<T> tab, int lxi, int let, int nstart, int nend, int F, Coeffs cf,
             DerivSum sum) {
    __shared__ T ends[kThreads / 32][kWarpLines][2 * kLmd + 1];
    const int n = tab.n, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane % kWarpLines, c = lane / kWarpLines;
    const int len = lane_len(c, LT, tab.p, tab.last_len);
    const int line0 = ((int)blockIdx.x * (kThreads / 32) + w) * kWarpLines, s = AXIS == 1 ? lxi : lxi * let;
    if (line0 >= F) return;
    const int fidx = min(line0 + l, F - 1);  // past the last line: the last line again, not stored
    const int base = (AXIS == 1 ? (fidx / lxi) * (lxi * let) + fidx % lxi : fidx) + c * LT * s;
    const T *in = fs.in + blockIdx.y * fs.in_fs;
    T d[1][LT];
#pragma unroll
    for (int t = 0; t < LT; ++t) d[0][t] = t < len ? in[base + t * s] : T(0);
    T far = T(0);
    if (fs.recv && (lane & 2)) {
        const int k = (lane & 7) >> 1 & 2 | (lane & 1), line = line0 + (lane >> 3);
        if (line < F) far = fs.recv[((int64_t)blockIdx.y * 4 + k) * F + line];
    }
    warp_column_rhs<LT, T>(ends[w], lane, len, n, nstart, nend, cf, fs.recv ? &far : nullptr, d);
    warp_column_solve<LT, T>(tab, lane, len, d);
    if (len == 0 || line0 + l >= F) return;
    if (fs.drva) {
        T *dr = fs.drva + (int64_t)blockIdx.y * F + fidx;
        if (c == 0) dr[0] = d[0][0];
        if (c == (n - 1) / LT) dr[5 * (int64_t)F] = get_at<LT, T>(d[0], (n - 1) - c * LT);
    }
    T *out = fs.out + blockIdx.y * fs.out_fs;
    if constexpr (SUM) {
        const double *a0 = sum.add0 + blockIdx.y * sum.add_fs, *a1 = sum.add1 + blockIdx.y * sum.add_fs;
        double *total = sum.sum + blockIdx.y * sum.sum_fs;
        constexpr int B = 8;
#pragma unroll
        for (int t0 = 0; t0 < LT; t0 += B) {
            double r[B];
#pragma unroll
            for (int b = 0; b < B; ++b)
                if (t0 + b < len) r[b] = a0[base + (t0 + b) * s] + a1[base + (t0 + b) * s];
#pragma unroll
            for (int b = 0; b < B; ++b)
                if (t0 + b < len) total[base + (t0 + b) * s] = r[b] + d[0][t0 + b];
        }
    }
#pragma unroll
    for (int t = 0; t < LT; ++t)
        if (t < len) out[base + t * s] = d[0][t];
}

// The same for all other y and z lines: column tiles (column.cuh) of two groups of TL lines,
// thread (l, c) holding chunk c of lines l and l + TL, so that addresses, solver
// constants, table loads and barriers serve two lines (and a row of the tile is
// 128 bytes).  Bound by its instructions and load latency (24 warps per SM): one
// 256^3 field 76 us, 3.5 TB/s, against 80 us with one line per thread, 87 us with
// 16-line tiles, and 105 us staged through a transposing layout.
//
// A CTA also prefetches into L2, a row a thread, the tile `ahead` places on: a
// prefetch holds no register and no load slot of the SM.  One 256^3 field 80 -> 76
// us (distance 4: 78), the batched launches of the call sequence 358 -> 331 us along
// y, 328 -> 296 us along z; with the sum over the axes in the store 774 -> 744 us
// at distance 4 (32: 766).  Single precision, other chunk lengths and
// the x rows do not gain (28.0 -> 28.3, 23.5 -> 24.4, 62.2 -> 64.3 us), nor do
// fields that L2 can still hold; see deriv_ahead.
template <int LT, int AXIS, int TL, int NL, typename T, bool SUM>
__global__ void __launch_bounds__(TL * 32, LT <= 8 ? 768 / (TL * 32) : 2)
k_deriv_col(FieldSet<T> fs, DevTables<T> tab, int lxi, int let, int nstart, int nend, int F, Coeffs cf,
            DerivSum sum, int ahead) {
    using C = Column<LT, TL>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *V = reinterpret_cast<T *>(smem_raw), *rows = V + NL * C::kField;
    const int n = tab.n, l = threadIdx.x % TL, c = threadIdx.x / TL, j0 = c * LT;
    const int len = lane_len(c, LT, tab.p, tab.last_len);
    const int line0 = (int)blockIdx.x * (NL * TL), s = AXIS == 1 ? lxi : lxi * let;
    int base[NL];
#pragma unroll
    for (int h = 0; h < NL; ++h) {
        // past the last line: the last line again, not stored
        const int fidx = min(line0 + h * TL + l, F - 1);
        base[h] = (AXIS == 1 ? (fidx / lxi) * (lxi * let) + fidx % lxi : fidx) + j0 * s;
    }
    const T *in = fs.in + blockIdx.y * fs.in_fs;
    if (LT == 8 && sizeof(T) == 8 && ahead) {
        const int la = line0 + ahead * (NL * TL);
        if (la < F) {
            const T *p = in + (AXIS == 1 ? (la / lxi) * (lxi * let) + la % lxi : la);
            for (int j = threadIdx.x; j < n; j += blockDim.x)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (int64_t)j * s));
        }
    }
    T d[NL][LT];
#pragma unroll
    for (int t = 0; t < LT; ++t)
#pragma unroll
        for (int h = 0; h < NL; ++h) d[h][t] = t < len ? in[base[h] + t * s] : T(0);
#pragma unroll
    for (int h = 0; h < NL; ++h) column_put_raw<LT, TL, T>(V + h * C::kField, d[h], c, l, n);
    __syncthreads();
    if (nstart || nend)
        column_closure_rows<LT, TL, NL, T, T>(V, rows, n, cf, fs.recv ? fs.recv + (int64_t)blockIdx.y * 4 * F : nullptr,
                                           F, line0);
#pragma unroll
    for (int h = 0; h < NL; ++h) column_rhs<LT, TL, T>(V + h * C::kField, c, l, len, n, nstart, nend, d[h]);
    __syncthreads();
    if (nstart || nend) {
#pragma unroll
        for (int h = 0; h < NL; ++h) column_take_rows<LT, T>(rows + 4 * (h * TL + l), c, n, nstart, nend, d[h]);
    }
    chunk_eliminate<LT, NL, T>(tab, d, c);
#pragma unroll
    for (int h = 0; h < NL; ++h) column_put_ends<LT, TL, T>(V + h * C::kField, d[h], c, l, len);
    __syncthreads();
    column_reduced<LT, TL, NL, T>(V, tab);
    __syncthreads();
    if (len == 0) return;
#pragma unroll
    for (int h = 0; h < NL; ++h) column_finish<LT, TL, T>(V + h * C::kField, tab, c, l, len, d[h]);
    T *out = fs.out + blockIdx.y * fs.out_fs;
#pragma unroll
    for (int h = 0; h < NL; ++h) {
        const int fidx = line0 + h * TL + l;
        if (fidx >= F) break;
        if (fs.drva) {
            T *dr = fs.drva + (int64_t)blockIdx.y * F + fidx;
            if (c == 0) dr[0] = d[h][0];
            if (c == (n - 1) / LT) dr[5 * (int64_t)F] = get_at<LT, T>(d[h], (n - 1) - j0);
        }
        if constexpr (SUM) {
            const double *a0 = sum.add0 + blockIdx.y * sum.add_fs, *a1 = sum.add1 + blockIdx.y * sum.add_fs;
            double *total = sum.sum + blockIdx.y * sum.sum_fs;
            double r[LT];
#pragma unroll
            for (int t = 0; t < LT; ++t)
                if (t < len) r[t] = a0[base[h] + t * s] + a1[base[h] + t * s];
#pragma unroll
            for (int t = 0; t < LT; ++t)
                if (t < len) total[base[h] + t * s] = r[t] + d[h][t];
        }
#pragma unroll
        for (int t = 0; t < LT; ++t)
            if (t < len) out[base[h] + t * s] = d[h][t];
    }
}

// Compact filter of one field along AXIS.
template <int LT, int AXIS>
__global__ void __launch_bounds__(kThreads)
k_filter(const double *__restrict__ in, double *__restrict__ out, DevTables<double> tab, int lxi,
         int let, double af, int64_t F) {
    using L = LineLayout<LT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sm = reinterpret_cast<double *>(smem_raw);
    const int n = tab.n;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t line0 = (int64_t)blockIdx.x * kTileLines;
    load_tile<LT, AXIS>(in, sm, line0, F, n, lxi, let);
    if (AXIS == 0) __syncwarp();
    else __syncthreads();
    const int64_t fidx = line0 + w;
    if (fidx < F) {
        double d[1][LT];
        double *line = sm + w * L::kSlot;
        filter_rhs<LT, double, double>(line, n, lane, tab.cyclic != 0, af, d[0]);
        warp_solve<LT, 1, double>(tab, d, lane);
        __syncwarp();
        store_line_regs<LT, double>(line, d[0], lane, n);
    }
    if (AXIS == 0) __syncwarp();
    else __syncthreads();
    store_tile<LT, AXIS>(out, sm, line0, F, n, lxi, let);
}

// Interface sums of one face (fill_gpu_buffer_kernel,
// src/cuda/kernels/numerics_pc.hpp:42-122).
template <int AXIS>
__global__ void k_fill(const double *__restrict__ in, double *__restrict__ send, int lxi, int let,
                       int n, int face, int64_t F, Coeffs cf) {
    const int64_t fidx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (fidx >= F) return;
    const int64_t base = line_base<AXIS>(fidx, lxi, let), s = line_stride<AXIS>(lxi, let);
    const int istart = face * (n - 1), inc = 1 - 2 * face;
    double v0 = 0.0, v1 = 0.0;
#pragma unroll
    for (int i = 0; i < kLmd; ++i) {
        const double f = in[base + (int64_t)(istart + inc * i) * s];
        v0 += cf.pbco[i] * f;
        v1 += cf.pbco[kLmd + i] * f;
    }
    send[fidx] = v0;
    send[F + fidx] = v1;
}

// ----------------------------------------------------------------------------
// launch helpers
// ----------------------------------------------------------------------------
inline int64_t face_size(const cs_dcomp &d, int axis) {
    return axis == 0 ? (int64_t)d.let * d.lze : (axis == 1 ? (int64_t)d.lxi * d.lze : (int64_t)d.lxi * d.let);
}
inline int line_len(const cs_dcomp &d, int axis) { return axis == 0 ? d.lxi : (axis == 1 ? d.let : d.lze); }

template <typename KernelT>
static int prep_smem(KernelT kern, size_t bytes) {
    if (bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute");
    }
    return CS_OK;
}

// Distance, in tiles, of k_deriv_col's prefetch.  None below 96 MB of input: 126 MB
// of L2 keep such a field, and what is already there is only asked for twice.
static int deriv_ahead(const cs_dcomp &d, int nf, bool with_sum) {
    if ((int64_t)nf * d.lmx * (int64_t)sizeof(double) < (int64_t)96 << 20) return 0;
    return with_sum ? 4 : 32;
}

// y and z lines in column tiles (k_deriv_col) of NL groups of eight lines.
template <int LT, int AXIS, int NL, typename T>
static int launch_deriv_col(const FieldSet<T> &fs, int nf, const DevTables<T> &tab, const cs_dcomp &d, int nstart,
                            int nend, const Coeffs &cf, const DerivSum *sum, int nsm, cudaStream_t st) {
    constexpr int TL = 8;
    const int64_t F = face_size(d, AXIS);
    const size_t smem = (size_t)NL * (Column<LT, TL>::kField + 4 * TL) * sizeof(T);
    auto kern = k_deriv_col<LT, AXIS, TL, NL, T, false>;
    if constexpr (AXIS == 2 && sizeof(T) == 8) {
        if (sum) kern = k_deriv_col<LT, AXIS, TL, NL, T, true>;
    }
    if (int rc = prep_smem(kern, smem)) return rc;
    // Where not every SM gets a CTA, eight warps in each solve the reduced systems in
    // one round, whatever the lines' chunks need (24x24x16 along z 5.2 -> 4.0 us).
    const int64_t blocks = (F + NL * TL - 1) / (NL * TL);
    const int threads = blocks * nf < nsm ? TL * 32 : column_threads(TL, tab.p);
    kern<<<dim3((unsigned)blocks, (unsigned)nf), threads, smem, st>>>(
        fs, tab, d.lxi, d.let, nstart, nend, (int)F, cf, sum ? *sum : DerivSum{}, deriv_ahead(d, nf, sum != nullptr));
    CSB_CUDA(cudaGetLastError());
    return CS_OK;
}

template <int LT, int AXIS, typename T>
static int launch_deriv_lt(const FieldSet<T> &fs, int nf, const DevTables<T> &tab, const cs_dcomp &d, int nstart,
                           int nend, const Coeffs &cf, const DerivSum *sum, int nsm, cudaStream_t st) {
    const int64_t F = face_size(d, AXIS);
    if constexpr (AXIS == 0) {
        constexpr int NV = LT <= 8 ? 2 : 1, WARPS = kThreads / 32;
        // A lane's chunk of more than 64 bytes spreads each of its vector loads over
        // 4 KB and more.  With 128 bytes (FP64, lines of 257..512 points) that still
        // pays for the table-driven solve (400x96x96, physical closure 31 -> 25 us;
        // staged 33), not for the faster interior one (512x88x88, interface closure
        // 24.6 against 22.6 us staged), and on lines of more than 512 points only in FP32
        // with fewer CTAs than SMs (FP32 1024x16x16 5.5 against 10.8 us, 1024x64x64 18.5
        // against 14.4; FP64 28.7 against 26.7 us).
        const bool vectors = LT * sizeof(T) <= 64 || (LT == 16 && !tab.interior) ||
                             (LT == 32 && sizeof(T) == 4 && (F + WARPS - 1) / WARPS * nf < nsm);
        const dim3 grid((unsigned)((F + NV * WARPS - 1) / (NV * WARPS)), (unsigned)nf);
        auto aligned = [&](int vb) {
            const int64_t ve = vb / (int)sizeof(T);
            return vectors && LT % ve == 0 && d.lxi % ve == 0 && (nf == 1 || (fs.in_fs % ve == 0 && fs.out_fs % ve == 0)) &&
                   reinterpret_cast<uintptr_t>(fs.in) % vb == 0 && reinterpret_cast<uintptr_t>(fs.out) % vb == 0;
        };
        if constexpr (LT * sizeof(T) >= 32) {
            if (aligned(32)) {
                k_deriv_row<LT, NV, 32, T><<<grid, kThreads, 0, st>>>(fs, tab, nstart, nend, F, cf);
                CSB_CUDA(cudaGetLastError());
                return CS_OK;
            }
        }
        if constexpr (LT * sizeof(T) >= 16) {
            if (aligned(16)) {
                k_deriv_row<LT, NV, 16, T><<<grid, kThreads, 0, st>>>(fs, tab, nstart, nend, F, cf);
                CSB_CUDA(cudaGetLastError());
                return CS_OK;
            }
        }
        const size_t smem = (size_t)NV * WARPS * LineLayout<LT>::kSlot * sizeof(T);
        auto kern = k_deriv_row_any<LT, NV, T>;
        if (int rc = prep_smem(kern, smem)) return rc;
        kern<<<grid, kThreads, smem, st>>>(fs, tab, nstart, nend, F, cf);
    } else {
        const bool with_sum = AXIS == 2 && sizeof(T) == 8 && sum;
        if (LT == kWarpChunk && warp_column(tab.n)) {
            if constexpr (LT == kWarpChunk) {
                constexpr int LINES = kThreads / 32 * kWarpLines;
                auto kern = k_deriv_wcol<LT, AXIS, T, false>;
                if constexpr (AXIS == 2 && sizeof(T) == 8) {
                    if (with_sum) kern = k_deriv_wcol<LT, AXIS, T, true>;
                }
                kern<<<dim3((unsigned)((F + LINES - 1) / LINES), (unsigned)nf), kThreads, 0, st>>>(
                    fs, tab, d.lxi, d.let, nstart, nend, (int)F, cf, with_sum ? *sum : DerivSum{});
            }
        } else {
            // Two lines a thread, but one of 32 rows (two take 147 KB and an SM for
            // themselves: FP64 72x700x72 39 -> 29 us along y), and one of 16 where two
            // would not give every SM a CTA (16x400x16 7.5 -> 5.3 us).
            const DerivSum *s = with_sum ? sum : nullptr;
            if (LT == 16 && (F + 15) / 16 * nf < nsm)
                return launch_deriv_col<LT, AXIS, LT >= 16 ? 1 : 2, T>(fs, nf, tab, d, nstart, nend, cf, s, nsm, st);
            return launch_deriv_col<LT, AXIS, LT == 32 ? 1 : 2, T>(fs, nf, tab, d, nstart, nend, cf, s, nsm, st);
        }
    }
    CSB_CUDA(cudaGetLastError());
    return CS_OK;
}

template <int AXIS, typename T>
static int launch_deriv_axis(int lt, const FieldSet<T> &fs, int nf, const DevTables<T> &tab, const cs_dcomp &d,
                             int nstart, int nend, const Coeffs &cf, const DerivSum *sum, int nsm,
                             cudaStream_t st) {
    switch (lt) {
        case 2: return launch_deriv_lt<2, AXIS, T>(fs, nf, tab, d, nstart, nend, cf, sum, nsm, st);
        case 4: return launch_deriv_lt<4, AXIS, T>(fs, nf, tab, d, nstart, nend, cf, sum, nsm, st);
        case 8: return launch_deriv_lt<8, AXIS, T>(fs, nf, tab, d, nstart, nend, cf, sum, nsm, st);
        case 16: return launch_deriv_lt<16, AXIS, T>(fs, nf, tab, d, nstart, nend, cf, sum, nsm, st);
        case 32: return launch_deriv_lt<32, AXIS, T>(fs, nf, tab, d, nstart, nend, cf, sum, nsm, st);
    }
    return set_error(CS_ERR_UNSUPPORTED, "chunk length %d", lt);
}

template <int LT, int AXIS>
static int launch_filter_lt(const double *in, double *out, const DevTables<double> &tab,
                            const cs_dcomp &d, double af, cudaStream_t st) {
    const int64_t F = face_size(d, AXIS);
    const size_t smem = (size_t)kTileLines * LineLayout<LT>::kSlot * sizeof(double);
    auto kern = k_filter<LT, AXIS>;
    int rc = prep_smem(kern, smem);
    if (rc) return rc;
    const int64_t blocks = (F + kTileLines - 1) / kTileLines;
    kern<<<(unsigned)blocks, kThreads, smem, st>>>(in, out, tab, d.lxi, d.let, af, F);
    CSB_CUDA(cudaGetLastError());
    return CS_OK;
}

template <int AXIS>
static int launch_filter_axis(int lt, const double *in, double *out, const DevTables<double> &tab,
                              const cs_dcomp &d, double af, cudaStream_t st) {
    switch (lt) {
        case 2: return launch_filter_lt<2, AXIS>(in, out, tab, d, af, st);
        case 4: return launch_filter_lt<4, AXIS>(in, out, tab, d, af, st);
        case 8: return launch_filter_lt<8, AXIS>(in, out, tab, d, af, st);
        case 16: return launch_filter_lt<16, AXIS>(in, out, tab, d, af, st);
        case 32: return launch_filter_lt<32, AXIS>(in, out, tab, d, af, st);
    }
    return set_error(CS_ERR_UNSUPPORTED, "chunk length %d", lt);
}

static int check_dims(const cs_dcomp &d) {
    if (d.lxi < 1 || d.let < 1 || d.lze < 1 || (int64_t)d.lxi * d.let * d.lze != (int64_t)d.lmx)
        return set_error(CS_ERR_INVALID, "inconsistent t_dcomp {%d,%d,%d,%d}", d.lmx, d.lxi, d.let, d.lze);
    return CS_OK;
}

static bool same_dims(const cs_dcomp &a, const cs_dcomp &b) {
    return a.lmx == b.lmx && a.lxi == b.lxi && a.let == b.let && a.lze == b.lze;
}

template <typename T>
const DevTables<T> &pick_tables(const DeviceTables &dt);
template <>
const DevTables<double> &pick_tables<double>(const DeviceTables &dt) { return dt.t64; }
template <>
const DevTables<float> &pick_tables<float>(const DeviceTables &dt) { return dt.t32; }

// nf derivatives along `axis` in one launch: field f is in + f in_fs -> out +
// f out_fs, with the numerics object's interface buffers of variable var + f.
template <typename T>
static int deriv_launch(cs_numerics *nm, int axis, const T *in, int64_t in_fs, T *out, int64_t out_fs, int nf,
                        unsigned var, int nstart, int nend, int halo, const DerivSum *sum, cudaStream_t st) {
    const cs_dcomp &d = nm->d;
    const int n = line_len(d, axis);
    const int64_t F = face_size(d, axis);
    if ((nstart || nend) && n < kLmd) return set_error(CS_ERR_UNSUPPORTED, "interface closure needs n >= 8");
    const bool wcol = axis > 0 && warp_column_pays(n, nstart, nend, nf * F, nm->nsm, (int)sizeof(T));
    const DeviceTables *dt = nm->tables.get(n, kDeriv, nstart, nend, 0.0, wcol ? kWarpChunk : 2);
    if (!dt) return CS_ERR_UNSUPPORTED;
    FieldSet<T> fs{in, out, nullptr, nullptr, in_fs, out_fs};
    if (sizeof(T) == sizeof(double)) {
        if (halo == CS_HALO_RECV) fs.recv = reinterpret_cast<const T *>(nm->recv[axis] + (int64_t)var * 4 * F);
        fs.drva = reinterpret_cast<T *>(nm->drva[axis] + (int64_t)var * F);
    } else if (halo == CS_HALO_RECV && (nstart || nend)) {
        return set_error(CS_ERR_UNSUPPORTED, "FP32 derivative supports CS_HALO_SELF only");
    }
    const DevTables<T> &tab = pick_tables<T>(*dt);
    switch (axis) {
        case 0: return launch_deriv_axis<0, T>(dt->lt, fs, nf, tab, d, nstart, nend, nm->cf, nullptr, nm->nsm, st);
        case 1: return launch_deriv_axis<1, T>(dt->lt, fs, nf, tab, d, nstart, nend, nm->cf, nullptr, nm->nsm, st);
        default: return launch_deriv_axis<2, T>(dt->lt, fs, nf, tab, d, nstart, nend, nm->cf, sum, nm->nsm, st);
    }
}

template <typename T>
static int deriv_impl(cs_numerics *nm, int axis, const T *in, T *out, int nstart, int nend,
                      cs_dcomp d, unsigned var, unsigned comp, unsigned slot, int halo,
                      void *stream) {
    if (!nm || !in || !out) return set_error(CS_ERR_INVALID, "null argument");
    if (!nm->setup_done) return set_error(CS_ERR_STATE, "cs_deriv before cs_deriv_setup");
    if (int rc = check_dims(d)) return rc;
    if (!same_dims(d, nm->d)) return set_error(CS_ERR_INVALID, "dims differ from the numerics object");
    if (axis < 0 || axis > 2 || var >= 5 || comp > 14 || slot > 14)
        return set_error(CS_ERR_INVALID, "axis %d var %u comp %u slot %u", axis, var, comp, slot);
    return deriv_launch<T>(nm, axis, in + (int64_t)comp * d.lmx, 0, out + (int64_t)slot * d.lmx, 0, 1, var, nstart,
                           nend, halo, nullptr, (cudaStream_t)stream);
}

int deriv_fields(cs_numerics *nm, int axis, const double *in, int64_t in_fs, double *out, int64_t out_fs, int nf,
                 unsigned var, const DerivSum *sum, cudaStream_t st) {
    if (!nm->setup_done) return set_error(CS_ERR_STATE, "cs_deriv before cs_deriv_setup");
    return deriv_launch<double>(nm, axis, in, in_fs, out, out_fs, nf, var, nm->ndf[0][axis], nm->ndf[1][axis],
                                CS_HALO_RECV, sum, st);
}

// Interface sums of every face of a single-rank block and their exchange
// (fill_buffers, then the copy of cs_halo_exchange_self) for nf variables in
// one launch (34 us for five variables at 256^3; face by face and copy by copy
// it was 30 launches and 30 copies, about 180 us, and all latency on small
// blocks): thread = (face, line), blockIdx.y = variable; the sums of face
// ip go to its send buffer and to the receive buffer of face 1 - ip.
struct ExchangeArgs {
    const double *in;  // variable 0; variables fs apart, axis a's component comp_fs * a further
    int64_t fs, comp_fs;
    double *send[3], *recv[3];
    int64_t F[3];
    int n[3], on[3], lxi, let;
    unsigned var;  // variable of the buffers that blockIdx.y = 0 fills
};
__global__ void k_exchange_self(ExchangeArgs x, Coeffs cf) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int a = 0;
    for (; a < 3; ++a) {
        const int64_t lines = x.on[a] ? 2 * x.F[a] : 0;
        if (i < lines) break;
        i -= lines;
    }
    if (a == 3) return;
    const int64_t F = x.F[a], fidx = i < F ? i : i - F;
    const int ip = i < F ? 0 : 1;
    const int64_t base = a == 0 ? line_base<0>(fidx, x.lxi, x.let)
                                : (a == 1 ? line_base<1>(fidx, x.lxi, x.let) : line_base<2>(fidx, x.lxi, x.let));
    const int64_t s = a == 0 ? 1 : (a == 1 ? (int64_t)x.lxi : (int64_t)x.lxi * x.let);
    const double *in = x.in + blockIdx.y * x.fs + a * x.comp_fs + base + (ip ? (x.n[a] - 1) * s : 0);
    const int64_t inc = ip ? -s : s;
    double v0 = 0.0, v1 = 0.0;
#pragma unroll
    for (int k = 0; k < kLmd; ++k) {
        const double f = in[k * inc];
        v0 += cf.pbco[k] * f;
        v1 += cf.pbco[kLmd + k] * f;
    }
    const int64_t o = (int64_t)(x.var + blockIdx.y) * 4 * F + fidx;
    double *snd = x.send[a] + o + ip * 2 * F, *rcv = x.recv[a] + o + (1 - ip) * 2 * F;
    snd[0] = v0;
    snd[F] = v1;
    rcv[0] = v0;
    rcv[F] = v1;
}

int exchange_self(cs_numerics *nm, const double *in, int64_t fs, int64_t comp_fs, int nf, unsigned var,
                  cudaStream_t st) {
    if (!nm->setup_done) return set_error(CS_ERR_STATE, "cs_fill_buffers before cs_deriv_setup");
    ExchangeArgs x{};
    int64_t total = 0;
    for (int a = 0; a < 3; ++a) {
        x.n[a] = line_len(nm->d, a);
        if ((nm->ndf[0][a] || nm->ndf[1][a]) && x.n[a] < kLmd)
            return set_error(CS_ERR_UNSUPPORTED, "interface face needs n >= 8");
    }
    for (int a = 0; a < 3; ++a) {
        if (nm->ndf[0][a] != nm->ndf[1][a])
            return set_error(CS_ERR_UNSUPPORTED,
                             "axis %d has one interface face: a single rank has no neighbour for it", a);
        x.F[a] = face_size(nm->d, a);
        x.on[a] = nm->ndf[0][a];
        x.send[a] = nm->send[a];
        x.recv[a] = nm->recv[a];
        if (x.on[a]) total += 2 * x.F[a];
    }
    if (total == 0) return CS_OK;
    x.in = in;
    x.fs = fs;
    x.comp_fs = comp_fs;
    x.lxi = nm->d.lxi;
    x.let = nm->d.let;
    x.var = var;
    k_exchange_self<<<dim3((unsigned)((total + 127) / 128), (unsigned)nf), 128, 0, st>>>(x, nm->cf);
    CSB_CUDA(cudaGetLastError());
    return CS_OK;
}

}  // namespace csb

using namespace csb;

extern "C" {

const char *cs_last_error(void) { return csb::g_err; }
int cs_version(void) { return 1; }

int cs_numerics_create(cs_numerics **out, cs_dcomp d, const int nbc[2][3]) {
    if (!out || !nbc) return set_error(CS_ERR_INVALID, "null argument");
    *out = nullptr;
    if (int rc = check_dims(d)) return rc;
    auto *nm = new cs_numerics();
    nm->d = d;
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&nm->nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) nm->nsm = 1;
    for (int f = 0; f < 2; ++f)
        for (int a = 0; a < 3; ++a) {
            const int b = nbc[f][a];
            nm->nbc[f][a] = b;
            if (b == CS_BC_NON_REFLECTIVE || b == CS_BC_WALL_INVISCID || b == CS_BC_WALL_VISCOUS ||
                b == CS_BC_INTER_CURV) nm->ndf[f][a] = 0;
            else if (b == CS_BC_INTER_STRAIGHT || b == CS_BC_INTER_SUBDOMAINS || b == CS_BC_PERIODIC)
                nm->ndf[f][a] = 1;
            else {
                delete nm;
                return set_error(CS_ERR_INVALID, "unknown boundary code %d", b);
            }
        }
    for (int a = 0; a < 3; ++a) {
        const int64_t F = face_size(d, a);
        if (cudaMalloc(&nm->drva[a], 2 * 5 * F * sizeof(double)) != cudaSuccess ||
            cudaMalloc(&nm->send[a], 4 * 5 * F * sizeof(double)) != cudaSuccess ||
            cudaMalloc(&nm->recv[a], 4 * 5 * F * sizeof(double)) != cudaSuccess) {
            cs_numerics_destroy(nm);
            return set_error(CS_ERR_ALLOC, "numerics scratch allocation failed");
        }
        cudaMemset(nm->drva[a], 0, 2 * 5 * F * sizeof(double));
        cudaMemset(nm->send[a], 0, 4 * 5 * F * sizeof(double));
        cudaMemset(nm->recv[a], 0, 4 * 5 * F * sizeof(double));
    }
    *out = nm;
    return CS_OK;
}

int cs_numerics_destroy(cs_numerics *nm) {
    if (!nm) return CS_OK;
    for (int a = 0; a < 3; ++a) {
        if (nm->drva[a]) cudaFree(nm->drva[a]);
        if (nm->send[a]) cudaFree(nm->send[a]);
        if (nm->recv[a]) cudaFree(nm->recv[a]);
    }
    delete nm;
    return CS_OK;
}

int cs_deriv_setup(cs_numerics *nm) {
    if (!nm) return set_error(CS_ERR_INVALID, "null argument");
    compute_interface_coeffs(nm->cf);
    for (int a = 0; a < 3; ++a) {
        const int n = line_len(nm->d, a);
        if (n < 5) continue;  // degenerate axis: derivative along it is rejected at call time
        // the tables of every form that this object's launches (1, 4 or 5 fields) take
        const int64_t F = face_size(nm->d, a);
        bool use[2] = {false, false};  // four lines a warp: no, yes
        for (int nf : {1, 4, 5})
            for (int bytes : {8, 4})
                use[a > 0 && warp_column_pays(n, nm->ndf[0][a], nm->ndf[1][a], nf * F, nm->nsm, bytes)] = true;
        for (int w = 0; w < 2; ++w)
            if (use[w] && !nm->tables.get(n, kDeriv, nm->ndf[0][a], nm->ndf[1][a], 0.0, w ? kWarpChunk : 2))
                return CS_ERR_UNSUPPORTED;
    }
    nm->setup_done = true;
    return CS_OK;
}

int cs_interface_coeffs(double pbco[16], double pbci[16]) {
    if (!pbco || !pbci) return set_error(CS_ERR_INVALID, "null argument");
    Coeffs cf;
    compute_interface_coeffs(cf);
    std::memcpy(pbco, cf.pbco, sizeof cf.pbco);
    std::memcpy(pbci, cf.pbci, sizeof cf.pbci);
    return CS_OK;
}

int cs_get_coeffs(const cs_numerics *nm, double pbco[16], double pbci[16]) {
    if (!nm || !pbco || !pbci) return set_error(CS_ERR_INVALID, "null argument");
    if (!nm->setup_done) return set_error(CS_ERR_STATE, "cs_get_coeffs before cs_deriv_setup");
    std::memcpy(pbco, nm->cf.pbco, sizeof nm->cf.pbco);
    std::memcpy(pbci, nm->cf.pbci, sizeof nm->cf.pbci);
    return CS_OK;
}

int cs_get_ndf(const cs_numerics *nm, int ndf[2][3]) {
    if (!nm || !ndf) return set_error(CS_ERR_INVALID, "null argument");
    std::memcpy(ndf, nm->ndf, sizeof nm->ndf);
    return CS_OK;
}

int cs_get_buffers(cs_numerics *nm, int axis, double **drva, double **send, double **recv) {
    if (!nm || axis < 0 || axis > 2) return set_error(CS_ERR_INVALID, "bad argument");
    if (drva) *drva = nm->drva[axis];
    if (send) *send = nm->send[axis];
    if (recv) *recv = nm->recv[axis];
    return CS_OK;
}

int cs_deriv(cs_numerics *nm, int axis, const double *in, double *out, int nstart, int nend,
             cs_dcomp d, unsigned var, unsigned comp, unsigned slot, int halo, void *stream) {
    return deriv_impl<double>(nm, axis, in, out, nstart, nend, d, var, comp, slot, halo, stream);
}

int cs_deriv_f32(cs_numerics *nm, int axis, const float *in, float *out, int nstart, int nend,
                 cs_dcomp d, unsigned var, unsigned comp, unsigned slot, int halo, void *stream) {
    return deriv_impl<float>(nm, axis, in, out, nstart, nend, d, var, comp, slot, halo, stream);
}

int cs_fill_buffers(cs_numerics *nm, const double *in, int var_lo, int var_hi, int nrt, cs_dcomp d,
                    void *stream) {
    if (!nm || !in) return set_error(CS_ERR_INVALID, "null argument");
    if (!nm->setup_done) return set_error(CS_ERR_STATE, "cs_fill_buffers before cs_deriv_setup");
    if (int rc = check_dims(d)) return rc;
    if (var_lo < 0 || var_hi > 5 || var_lo > var_hi) return set_error(CS_ERR_INVALID, "variable range");
    cudaStream_t st = (cudaStream_t)stream;
    for (int m = var_lo; m < var_hi; ++m)
        for (int nn = 0; nn < 3; ++nn) {
            const int nzk = (1 - nrt) * nn;
            const int64_t F = face_size(d, nn);
            const int n = line_len(d, nn);
            const double *src = in + ((int64_t)nzk + (int64_t)m * 3) * d.lmx;
            for (int ip = 0; ip < 2; ++ip) {
                if (nm->ndf[ip][nn] != 1) continue;
                if (n < kLmd) return set_error(CS_ERR_UNSUPPORTED, "interface face needs n >= 8");
                double *snd = nm->send[nn] + (int64_t)m * 4 * F + (int64_t)ip * 2 * F;
                const unsigned blocks = (unsigned)((F + 255) / 256);
                if (nn == 0) k_fill<0><<<blocks, 256, 0, st>>>(src, snd, d.lxi, d.let, n, ip, F, nm->cf);
                else if (nn == 1) k_fill<1><<<blocks, 256, 0, st>>>(src, snd, d.lxi, d.let, n, ip, F, nm->cf);
                else k_fill<2><<<blocks, 256, 0, st>>>(src, snd, d.lxi, d.let, n, ip, F, nm->cf);
                CSB_CUDA(cudaGetLastError());
            }
        }
    return CS_OK;
}

int cs_halo_exchange_self(cs_numerics *nm, unsigned var, void *stream) {
    if (!nm || var >= 5) return set_error(CS_ERR_INVALID, "bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    for (int nn = 0; nn < 3; ++nn) {
        if (nm->ndf[0][nn] != nm->ndf[1][nn])
            return set_error(CS_ERR_UNSUPPORTED,
                             "axis %d has one interface face: a single rank has no neighbour for it", nn);
        if (nm->ndf[0][nn] != 1) continue;
        const int64_t F = face_size(nm->d, nn);
        double *snd = nm->send[nn] + (int64_t)var * 4 * F;
        double *rcv = nm->recv[nn] + (int64_t)var * 4 * F;
        // face 0 receives face 1's sums, face 1 receives face 0's
        // (tag pairing of src/numerics_base.hpp:161-176).
        CSB_CUDA(cudaMemcpyAsync(rcv, snd + 2 * F, 2 * F * sizeof(double), cudaMemcpyDeviceToDevice, st));
        CSB_CUDA(cudaMemcpyAsync(rcv + 2 * F, snd, 2 * F * sizeof(double), cudaMemcpyDeviceToDevice, st));
    }
    return CS_OK;
}

int cs_filter(cs_numerics *nm, int axis, const double *in, double *out, double alpha_f, cs_dcomp d,
              void *stream) {
    if (!nm || !in || !out) return set_error(CS_ERR_INVALID, "null argument");
    if (int rc = check_dims(d)) return rc;
    if (!same_dims(d, nm->d)) return set_error(CS_ERR_INVALID, "dims differ from the numerics object");
    if (axis < 0 || axis > 2) return set_error(CS_ERR_INVALID, "axis %d", axis);
    if (nm->ndf[0][axis] != nm->ndf[1][axis])
        return set_error(CS_ERR_UNSUPPORTED, "filter needs both faces periodic or both physical");
    if (!(alpha_f > -0.5 && alpha_f <= 0.5)) return set_error(CS_ERR_INVALID, "alpha_f %g", alpha_f);
    const int n = line_len(d, axis);
    if (n < 7) return set_error(CS_ERR_UNSUPPORTED, "filter needs n >= 7");
    const DeviceTables *dt = nm->tables.get(n, kFilter, nm->ndf[0][axis], nm->ndf[1][axis], alpha_f);
    if (!dt) return CS_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    switch (axis) {
        case 0: return launch_filter_axis<0>(dt->lt, in, out, dt->t64, d, alpha_f, st);
        case 1: return launch_filter_axis<1>(dt->lt, in, out, dt->t64, d, alpha_f, st);
        default: return launch_filter_axis<2>(dt->lt, in, out, dt->t64, d, alpha_f, st);
    }
}

int cs_line_tables(int n, int scheme, int nstart, int nend, double alpha_f, int meta[7],
                   double *tables, size_t tables_len) {
    if (!meta) return set_error(CS_ERR_INVALID, "null meta");
    HostTables h;
    if (!host_tables_for(n, scheme, nstart, nend, alpha_f, h))
        return set_error(CS_ERR_UNSUPPORTED, "line length %d", n);
    meta[0] = h.n; meta[1] = h.lt; meta[2] = h.p; meta[3] = h.last_len; meta[4] = h.cyclic;
    meta[5] = h.pcr64; meta[6] = h.pcr32;
    if (tables) {
        std::vector<double> v = pack(h);
        v.push_back(h.cyc_s1);
        v.push_back(h.cyc_s2);
        if (tables_len < v.size()) return set_error(CS_ERR_INVALID, "tables buffer too small (%zu)", v.size());
        std::memcpy(tables, v.data(), v.size() * sizeof(double));
    }
    return CS_OK;
}

}  // extern "C"
