// gm_stage_f64.cu -- the FP64 stage kernels without pressure.
#include "gm_stage_tma.cuh"

namespace gmk {
GMK_INSTANTIATE_TMA(double, false)
}
