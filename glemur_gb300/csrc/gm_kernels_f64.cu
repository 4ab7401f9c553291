// gm_kernels_f64.cu -- FP64-storage instantiation of the relaxation kernels
// (the TMA-fed stage kernels: gm_stage_f64.cu and gm_stage_f64_press.cu).
#include "gm_kernels_impl.cuh"

namespace gmk {
GMK_INSTANTIATE(double)
}
