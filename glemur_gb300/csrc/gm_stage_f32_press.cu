// gm_stage_f32_press.cu -- the FP32 stage kernels with the pressure gradient.
#include "gm_stage_tma.cuh"

namespace gmk {
GMK_INSTANTIATE_TMA(float, true)
}
