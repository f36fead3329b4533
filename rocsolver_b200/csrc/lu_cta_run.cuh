// lu_cta_run.cuh -- launches of the CTA LU variants (lu_cta.cuh).
#pragma once

#include <algorithm>

#include "logger.h"
#include "lu_cta.cuh"
#include "lu_cta_run.h"

namespace rsb {

// cw: trailing column chunk (multiple of 32); 0 picks the default (FP64: 64, FP32: 128 at
// most, so that two CTAs fit in an SM's shared memory).  *ran = false when the variant
// cannot take this size (more rows than threads x rows per thread, or too much shared
// memory).
template <typename T, int NT, int R, int JB, bool PIVOT, bool TC = false, bool UM = false>
static rocblas_status run_getrf_cta(cudaStream_t s, int m, int n, Batch<T> A, int lda,
                                    int* ipiv, int64_t sP, int* info, int bc, Gate g, int cw,
                                    int fold, bool* ran = nullptr)
{
    if(ran)
        *ran = false;
    if(m > NT * R)
        return rocblas_status_not_implemented;
    const int cwmax = sizeof(T) == 8 ? LU_CW_F64 : LU_CW_F32;
    const int nround = ((n + 31) / 32) * 32;
    if(cw <= 0)
        cw = cwmax;
    cw = ((cw + 31) / 32) * 32;
    if(cw > nround)
        cw = nround;
    if(UM && cw > 256) // one MMA covers at most 256 columns
        cw = 256;
    size_t smem = CtaLuSmem<T, NT, JB>::bytes(m, cw, R);
    if constexpr(UM)
        smem += um_bytes<NT, JB>(cw);
    if(smem > 227 * 1024)
        return rocblas_status_not_implemented;
    auto k = getrf_cta_kernel<T, NT, R, JB, 8, PIVOT, TC, UM>;
    if(!set_smem(k, smem))
        return rocblas_status_internal_error;
    if(ran)
        *ran = true;
    RSB_LOG_KERNEL("getrf_cta_kernel");
    k<<<bc, NT, smem, s>>>(m, n, A, lda, ipiv, sP, info, cw, fold, g);
    return launch_status();
}

// two-level FP32 LU (outer panels of 64 columns, tcgen05 trailing updates with K = 64)
template <int NT, int R, int JB>
static rocblas_status run_getrf_cta2(cudaStream_t s, int m, int n, Batch<float> A, int lda,
                                     int* ipiv, int64_t sP, int* info, int bc, Gate g, int cw,
                                     bool* ran)
{
    *ran = false;
    if(m > NT * R)
        return rocblas_status_not_implemented;
    const int nround = ((n + 31) / 32) * 32;
    if(cw <= 0)
        cw = 128;
    cw = ((cw + 31) / 32) * 32;
    cw = std::min(std::min(cw, 256), std::max(nround, 32));
    const int cwi = LU2_JO;
    const size_t smem = CtaLuSmem<float, NT, JB>::bytes(m, cwi, R) + lu2_bytes(cw);
    if(smem > 227 * 1024)
        return rocblas_status_not_implemented;
    auto k = getrf_cta2_kernel<NT, R, JB>;
    if(!set_smem(k, smem))
        return rocblas_status_internal_error;
    *ran = true;
    RSB_LOG_KERNEL("getrf_cta2_kernel");
    k<<<bc, NT, smem, s>>>(m, n, A, lda, ipiv, sP, info, cw, cwi, g);
    return launch_status();
}

template <typename T, bool PIVOT, bool TC>
rocblas_status run_getrf_tuned(const LuCfg& c, cudaStream_t s, int m, int n, Batch<T> A, int lda,
                               int* ipiv, int64_t sP, int* info, int bc, Gate g, bool* ran)
{
    *ran = false;
    // fold = 2 selects the tcgen05 trailing update (FP32 split-TF32 variants, panel widths
    // that are multiples of 8)
    if constexpr(sizeof(T) == 4 && TC && PIVOT)
    {
        // fold = 3: two-level LU (outer panels of 64 columns on tcgen05)
        if(c.fold == 3)
        {
#define RSB_LU2_VARIANT(NT_, R_, JB_)                                                          \
            if(c.nt == NT_ && c.r == R_ && c.jb == JB_)                                        \
                return run_getrf_cta2<NT_, R_, JB_>(s, m, n, A, lda, ipiv, sP, info, bc, g, c.cw, \
                                                    ran);
            RSB_LU2_VARIANT(256, 2, 32)
            RSB_LU2_VARIANT(256, 2, 16)
            RSB_LU2_VARIANT(256, 4, 16)
            RSB_LU2_VARIANT(256, 4, 8)
            RSB_LU2_VARIANT(256, 8, 8)
#undef RSB_LU2_VARIANT
            return rocblas_status_not_implemented;
        }
        if(c.fold == 2)
        {
#define RSB_LU_UM_VARIANT(NT_, R_, JB_)                                                        \
            if(c.nt == NT_ && c.r == R_ && c.jb == JB_)                                        \
                return run_getrf_cta<T, NT_, R_, JB_, PIVOT, TC, true>(s, m, n, A, lda, ipiv, \
                                                                       sP, info, bc, g, c.cw, 0, \
                                                                       ran);
            RSB_LU_UM_VARIANT(128, 1, 32)
            RSB_LU_UM_VARIANT(128, 2, 32)
            RSB_LU_UM_VARIANT(256, 1, 32)
            RSB_LU_UM_VARIANT(256, 2, 32)
            RSB_LU_UM_VARIANT(256, 2, 16)
            RSB_LU_UM_VARIANT(256, 4, 16)
            RSB_LU_UM_VARIANT(256, 4, 8)
            RSB_LU_UM_VARIANT(256, 8, 8)
#undef RSB_LU_UM_VARIANT
            return rocblas_status_not_implemented;
        }
    }
#define RSB_LU_VARIANT(NT_, R_, JB_)                                                          \
    if(c.nt == NT_ && c.r == R_ && c.jb == JB_)                                                \
        return run_getrf_cta<T, NT_, R_, JB_, PIVOT, TC>(s, m, n, A, lda, ipiv, sP, info, bc, \
                                                         g, c.cw, c.fold, ran);
    RSB_LU_VARIANT(64, 1, 32)
    RSB_LU_VARIANT(128, 1, 32)
    RSB_LU_VARIANT(128, 2, 32)
    RSB_LU_VARIANT(128, 2, 16)
    RSB_LU_VARIANT(128, 4, 16)
    RSB_LU_VARIANT(256, 1, 32)
    RSB_LU_VARIANT(256, 2, 16)
    RSB_LU_VARIANT(256, 2, 32)
    RSB_LU_VARIANT(256, 4, 8)
    RSB_LU_VARIANT(256, 4, 16)
    RSB_LU_VARIANT(256, 8, 4)
    RSB_LU_VARIANT(256, 8, 8)
#undef RSB_LU_VARIANT
    return rocblas_status_not_implemented;
}

#define RSB_LU_CTA_INST(T, PIVOT, TC)                                                          \
    template rocblas_status run_getrf_tuned<T, PIVOT, TC>(                                     \
        const LuCfg&, cudaStream_t, int, int, Batch<T>, int, int*, int64_t, int*, int, Gate,   \
        bool*);

} // namespace rsb
