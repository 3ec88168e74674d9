// context.h -- host-side objects behind the opaque C-ABI handles.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <string>
#include <tuple>

#include "cs_common.h"
#include "line_solver.cuh"

namespace csb {

int set_error(int code, const char *fmt, ...);
int check_cuda(cudaError_t e, const char *what);

#define CSB_CUDA(call)                                      \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return check_cuda(e_, #call); \
    } while (0)

// Device copy of the tables of one line configuration, in FP64 and FP32.
struct DeviceTables {
    HostTables host;
    double *d64 = nullptr;
    float *d32 = nullptr;
    DevTables<double> t64{};
    DevTables<float> t32{};
    int lt = 0;
    // every lane's chunk shares lane 0's per-row factors (full chunks, the
    // constant interior rows only: ChunkFactors); cfu holds them in FP32 as
    // [f1, f2, b1, b2, -rca, -rcc][lt]
    bool uniform = false;
    float cfu[6 * 32] = {};
};

// key: n, scheme, nstart, nend, alpha_f bits
using TableKey = std::tuple<int, int, int, int, uint64_t, int>;

// Cache of device tables (one per device/line configuration).
class TableCache {
public:
    ~TableCache();
    // Returns nullptr and sets the error on failure.  min_lt: shortest chunk
    // of the tables (build_tables).
    const DeviceTables *get(int n, int scheme, int nstart, int nend, double alpha_f, int min_lt = 2);

private:
    std::mutex mu_;
    std::map<TableKey, DeviceTables *> map_;
};

}  // namespace csb

struct cs_numerics {
    cs_dcomp d{};
    int nbc[2][3]{};
    int ndf[2][3]{};
    csb::Coeffs cf{};
    bool setup_done = false;
    int nsm = 1;  // SMs of the device
    double *drva[3] = {nullptr, nullptr, nullptr};
    double *send[3] = {nullptr, nullptr, nullptr};
    double *recv[3] = {nullptr, nullptr, nullptr};
    csb::TableCache tables;
};

namespace csb {

// sum[f] = (add0[f] + add1[f]) + the derivative of field f, formed by the
// derivative's own launch (fields f add_fs / sum_fs apart).
struct DerivSum {
    const double *add0 = nullptr, *add1 = nullptr;
    double *sum = nullptr;
    int64_t add_fs = 0, sum_fs = 0;
};

// Several fields of a single-rank block at once (numerics.cu), with the face
// closures, the received sums and the line-end buffers of the numerics object,
// variables var .. var + nf - 1.
// nf derivatives along `axis`: in + f in_fs -> out + f out_fs; sum (z only, may
// be null) adds them up.
int deriv_fields(cs_numerics *nm, int axis, const double *in, int64_t in_fs, double *out, int64_t out_fs, int nf,
                 unsigned var, const DerivSum *sum, cudaStream_t st);
// Interface sums of all faces into the send buffers and, exchanged, into the
// receive buffers: variable f's field for axis a is in + f fs + a comp_fs.
int exchange_self(cs_numerics *nm, const double *in, int64_t fs, int64_t comp_fs, int nf, unsigned var,
                  cudaStream_t st);

}  // namespace csb
