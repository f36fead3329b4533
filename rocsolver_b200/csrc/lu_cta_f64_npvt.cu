// lu_cta_f64_npvt.cu -- the CTA LU variants, FP64 without pivoting.
#include "lu_cta_run.cuh"

namespace rsb {
RSB_LU_CTA_INST(double, false, false)
} // namespace rsb
