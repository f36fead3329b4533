// lu_cta_f64.cu -- the CTA LU variants, FP64.
#include "lu_cta_run.cuh"

namespace rsb {
RSB_LU_CTA_INST(double, true, false)
} // namespace rsb
