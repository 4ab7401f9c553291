// gm_stage_f64_press.cu -- the FP64 stage kernels with the pressure gradient.
#include "gm_stage_tma.cuh"

namespace gmk {
GMK_INSTANTIATE_TMA(double, true)
}
