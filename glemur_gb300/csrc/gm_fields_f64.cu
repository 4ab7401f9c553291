// gm_fields_f64.cu -- the FP64 field kernels.
#include "gm_fields.cuh"

namespace gmk {
GMK_INSTANTIATE_FIELDS(double)
}
