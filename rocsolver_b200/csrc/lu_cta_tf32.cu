// lu_cta_tf32.cu -- the CTA LU variants, FP32 with split-TF32 trailing updates.
#include "lu_cta_run.cuh"

namespace rsb {
RSB_LU_CTA_INST(float, true, true)
} // namespace rsb
