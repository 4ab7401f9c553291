// gm_stage_f32.cu -- the FP32 stage kernels without pressure.
#include "gm_stage_tma.cuh"

namespace gmk {
GMK_INSTANTIATE_TMA(float, false)
}
