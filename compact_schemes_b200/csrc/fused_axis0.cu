// fused_axis0.cu -- instantiation of the fused passes along axis 0 (one
// translation unit per axis keeps the build parallel).
#include "fused_kernels.cuh"

namespace csb {

template <>
int launch_grad<0>(const PassArgs &a, const double *q, bool dtred, cudaStream_t st) {
    if (a.pl) return launch_grad_pl<0>(a, q, dtred, st);
    return launch_grad_tl<0, 8>(a, q, dtred, st);
}

template <>
int launch_flux<0>(const PassArgs &a, int mode, const double *q, const double *qn, double *qout,
                   double *drva, const RkParams &rk, cudaStream_t st) {
    if (a.pl) return launch_flux_pl<0>(a, mode, q, qn, qout, drva, rk, st);
    return launch_flux_tl<0, 8>(a, mode, q, qn, qout, drva, rk, st);
}

int launch_gradflux_x(const PassArgs &a, const double *q, double *drva, bool dtred, cudaStream_t st) {
    switch (a.tab->lt) {
        case 2: return launch_gradflux_t<2>(a, q, drva, dtred, st);
        case 4: return launch_gradflux_t<4>(a, q, drva, dtred, st);
    }
    return set_error(CS_ERR_UNSUPPORTED, "chunk length");
}

}  // namespace csb
