// lu_cta_f32_npvt.cu -- the CTA LU variants, FP32 without pivoting.
#include "lu_cta_run.cuh"

namespace rsb {
RSB_LU_CTA_INST(float, false, false)
} // namespace rsb
