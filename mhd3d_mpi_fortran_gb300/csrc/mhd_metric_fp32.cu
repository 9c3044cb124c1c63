// FP32 instantiation of the metric-mode (curvilinear) step kernels: FP32
// state, reconstruction and fluxes; metric terms computed in FP64, held in FP32.
// FMA contraction on.
#include "mhd_kernels.cuh"

namespace mhd {
template struct Launch<float, true>;
}
