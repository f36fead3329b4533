// lu_cta_run.h -- host interface of the CTA LU variants (lu_cta.cuh), which are compiled in
// translation units of their own (lu_cta_*.cu: they take minutes each).
#pragma once

#include "launch.h"
#include "tuning.h"

namespace rsb {

inline rocblas_status launch_status()
{
    return cudaGetLastError() == cudaSuccess ? rocblas_status_success
                                             : rocblas_status_internal_error;
}

// Opt in to the dynamic shared memory a launch needs (static shared memory of the kernel
// counts against the same 48 KiB default, so the attribute is always set).
template <typename K>
inline bool set_smem(K kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)bytes)
           == cudaSuccess;
}

// the compiled CTA variant that c names (threads, rows per thread, panel width); *ran = false
// when there is none or it cannot take this size
template <typename T, bool PIVOT, bool TC>
rocblas_status run_getrf_tuned(const LuCfg& c, cudaStream_t s, int m, int n, Batch<T> A, int lda,
                               int* ipiv, int64_t sP, int* info, int bc, Gate g, bool* ran);

} // namespace rsb
