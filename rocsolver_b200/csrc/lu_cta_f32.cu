// lu_cta_f32.cu -- the CTA LU variants, FP32.
#include "lu_cta_run.cuh"

namespace rsb {
RSB_LU_CTA_INST(float, true, false)
} // namespace rsb
