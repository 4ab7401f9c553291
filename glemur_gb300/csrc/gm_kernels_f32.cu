// gm_kernels_f32.cu -- FP32-storage instantiation of the relaxation kernels
// (the TMA-fed stage kernels: gm_stage_f32.cu and gm_stage_f32_press.cu).
#include "gm_kernels_impl.cuh"

namespace gmk {
GMK_INSTANTIATE(float)
}
