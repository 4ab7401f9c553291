// gm_fields_f32.cu -- the FP32 field kernels.
#include "gm_fields.cuh"

namespace gmk {
GMK_INSTANTIATE_FIELDS(float)
}
