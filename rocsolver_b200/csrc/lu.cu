// lu.cu -- launchers for getrf / getrs / gesv and the Cholesky pair.
//
// Kernel selection by size replaces the reference's compile-time tuning tables
// (library/src/include/ideal_sizes.hpp:208-240 getrf, :166-180 potrf;
// roclapack_getf2.hpp:181-276 select_spkernel): the CTA LU configuration comes from the
// run-time tuning table (tuning.h) when it has an entry, else from the built-in choice
// between them and the blocked LU (lu_blk.cuh).
#include <algorithm>

#include "chol.cuh"
#include "chol_blk.cuh"
#include "launch.h"
#include "logger.h"
#include "lu_blk.h"
#include "lu_cta_run.h"
#include "lu_small.cuh"
#include "trsv.cuh"
#include "tuning.h"

namespace rsb {

__global__ void reset_info_kernel(int* info, int bc)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < bc)
        info[i] = 0;
}

rocblas_status launch_reset_info(cudaStream_t s, int* info, int bc)
{
    if(bc <= 0)
        return rocblas_status_success;
    reset_info_kernel<<<(bc + 255) / 256, 256, 0, s>>>(info, bc);
    return launch_status();
}

__global__ void reset_info2_kernel(int* a, int* b, int bc)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < bc)
    {
        a[i] = 0;
        b[i] = 0;
    }
}

rocblas_status launch_reset_info2(cudaStream_t s, int* a, int* b, int bc)
{
    if(bc <= 0)
        return rocblas_status_success;
    reset_info2_kernel<<<(bc + 255) / 256, 256, 0, s>>>(a, b, bc);
    return launch_status();
}

// ------------------------------------------------------------------------------ getrf
template <typename T, int NMAX, bool PIVOT>
static void run_getrf_warp(cudaStream_t s, int m, int n, Batch<T> A, int lda, int* ipiv,
                           int64_t sP, int* info, int bc, Gate g)
{
    dim3 grid((bc + SMALL_WPB - 1) / SMALL_WPB);
    RSB_LOG_KERNEL("getrf_warp_kernel");
    getrf_warp_kernel<T, NMAX, PIVOT><<<grid, 32 * SMALL_WPB, 0, s>>>(m, n, A, lda, ipiv, sP,
                                                                       info, bc, g);
}

// Without a table entry: whether the one-launch CTA kernels (one CTA holds a member from first
// to last panel) take a call, or the blocked LU in separate launches.
//
// FP64 up to 512 rows: the CTA kernels, always.  These factors feed inverses and adjoints of
// matrices whose condition nothing bounds (uniform + 4 I, 16384 members of n = 64, hold one of
// 1e7 now and then), where another order of rounding shows: with the blocked LU such outputs
// moved by 1e-9 to 4e-9 (relative, 2-norm) in one of ten to one of four batches of n = 64 ..
// 256, beyond the 5e-10 that they are held to, at the same error against 64-bit results.  The
// blocked LU is no clear gain there either (getrf alone, ms, blocked / CTA): n = 64 x 16384
// 1.06 / 1.63, n = 65 x 16384 3.08 / 2.64, n = 128 x 8178 2.52 / 3.04, n = 129 x 8052 5.65 /
// 4.52, n = 200 x 3350 4.80 / 4.06, n = 256 x 2044 3.52 / 3.79, n = 512 x 592 6.95 / 7.12.
//
// Else the faster one.  The blocked LU pays for a whole 64-column panel, and for rows up to 64,
// 128, 256 or a cluster of 2, 4 or 8 CTAs of 256, whatever part of them a member fills; a
// cluster's CTA has an SM to itself, so clusters of 2 take 74 members at a time where the CTA
// kernels take 148; and the CTA kernels lose a part of their last wave.  Time of the CTA kernel
// over that of the blocked LU, at batches from 1 to 134e6 / n^2:
//   rows       FP32          split TF32
//   33-64      1.4-1.7       1.5-2.7
//   65-96      0.82-1.18     0.83-1.17
//   97-128     1.08-1.57     1.08-1.60
//   129-160    0.71-1.15     0.68-1.13
//   161-192    0.99-1.57     to 296 members 1.16-1.53, then 0.91-1.35
//   193-224    to 296 members 1.02-1.48, then 0.82-1.12;  to 222 1.04-1.40, then 0.73-1.05
//   225-256    1.08-1.91     to 296 members 1.14-1.83, then n < 250 0.90-1.24, 256 1.10-1.35
//   257-512    to 74 members 0.99-2.3 (TF32 below 284 rows 0.90-1.02), 75-148 0.73-1.16,
//              then 0.90-1.57 (TF32 0.77-1.33); at least 1.04 for 284 to 320 rows and, FP32,
//              above 480 rows and at multiples of 64
//   513-2048   1.2-57        0.96-23  (FP64 0.95-38)
// Panels with few columns (2 n <= m, more than 256 rows) have nothing to update beside the
// clusters: 300 x 64 0.42-0.84, 500 x 250 to 74 members 1.2, then 0.7; 1000 x 64 to 37 members
// 1.1 and 2.2, then 0.5; 2000 x 64 to 74 members 1.2 and 3.0, then 0.6 (FP64 0.83 at 74).
template <typename T>
static bool cta_lu_pays(int m, int n, int bc, bool tc)
{
    if(sizeof(T) == 8 && m <= 512)
        return true;
    if(m <= 64 || n >= 2 * m)
        return false;
    if(m > 256 && 2 * n <= m)
    {
        const int cluster = m <= 512 ? 2 : (m <= 1024 ? 4 : 8);
        return m <= 400 || (int64_t)bc * cluster * 700 > (int64_t)132 * std::max(m, 700);
    }
    if(m <= 96)
        return true;
    if(m <= 128)
        return false;
    if(m <= 160)
        return true;
    if(m <= 192)
        return tc && bc > 296;
    if(m <= 224)
        return bc > (tc ? 222 : 296);
    if(m <= 256)
        return tc && m < 250 && bc > 296;
    if(m <= 512)
    {
        if(bc <= 74)
            return tc && m < 284;
        if(bc <= 148)
            return true;
        const bool full = m >= 284 && m <= 320;
        return !(full || (!tc && (m > 480 || m % 64 == 0)));
    }
    return false;
}

// the CTA variant of a size (measured by rocsolver_b200/tune.py at the largest rows of each)
template <typename T>
static LuCfg cta_lu_builtin(int m, bool tc)
{
    if(sizeof(T) == 8)
        return m <= 64     ? LuCfg{128, 1, 32, 32, 1}
               : m <= 128  ? LuCfg{128, 1, 32, 64, 1}
               : m <= 256  ? LuCfg{256, 1, 32, 64, 1}
               : m <= 512  ? LuCfg{256, 2, 32, 128, 1}
               : m <= 1024 ? LuCfg{256, 4, 16, 128, 1}
                           : LuCfg{256, 8, 8, 96, 1};
    return m <= 128    ? LuCfg{128, 2, 32, 128, 1}
           : m <= 256  ? LuCfg{128, 2, 32, 64, 1}
           : m <= 512  ? LuCfg{256, 2, 32, 128, 1}
           : m <= 1024 ? LuCfg{256, 4, 16, 128, 1}
           : tc        ? LuCfg{256, 8, 8, 128, 3}
                       : LuCfg{256, 8, 8, 32, 1};
}

template <typename T, bool PIVOT, bool TC>
static rocblas_status getrf_dispatch(cudaStream_t s, int m, int n, Batch<T> A, int lda,
                                     int* ipiv, int64_t sP, int* info, int bc, Gate g)
{
    if(m <= 32 && n <= 32)
    {
        if(n <= 8)
            run_getrf_warp<T, 8, PIVOT>(s, m, n, A, lda, ipiv, sP, info, bc, g);
        else if(n <= 16)
            run_getrf_warp<T, 16, PIVOT>(s, m, n, A, lda, ipiv, sP, info, bc, g);
        else
            run_getrf_warp<T, 32, PIVOT>(s, m, n, A, lda, ipiv, sP, info, bc, g);
        return launch_status();
    }
    LuCfg c;
    const char prec = sizeof(T) == 8 ? 'd' : 's';
    if((TC && tuned_getrf('t', m, &c)) || tuned_getrf(prec, m, &c))
    {
        bool ran = false;
        const rocblas_status st =
            run_getrf_tuned<T, PIVOT, TC>(c, s, m, n, A, lda, ipiv, sP, info, bc, g, &ran);
        if(ran)
            return st;
    }
    if(cta_lu_pays<T>(m, n, bc, TC))
    {
        bool ran = false;
        const rocblas_status st = run_getrf_tuned<T, PIVOT, TC>(
            cta_lu_builtin<T>(m, TC), s, m, n, A, lda, ipiv, sP, info, bc, g, &ran);
        if(ran)
            return st;
    }
    LuBatch<T> L{};
    L.A = A;
    L.m = m;
    L.n = n;
    L.lda = lda;
    L.ipiv = ipiv;
    L.strideP = sP;
    L.info = info;
    L.gate = g;
    return launch_lu_blk<T>(s, L, m, n, bc, PIVOT, TC);
}

template <typename T>
rocblas_status launch_getrf(cudaStream_t s, int m, int n, Batch<T> A, int lda, int* ipiv,
                            int64_t sP, int* info, int bc, bool pivot, Gate g, bool tc)
{
    if constexpr(sizeof(T) == 4)
        if(tc && pivot)
            return getrf_dispatch<T, true, true>(s, m, n, A, lda, ipiv, sP, info, bc, g);
    return pivot ? getrf_dispatch<T, true, false>(s, m, n, A, lda, ipiv, sP, info, bc, g)
                 : getrf_dispatch<T, false, false>(s, m, n, A, lda, ipiv, sP, info, bc, g);
}

// ------------------------------------------------------------------------------ getrs
template <typename T, int NMAX, int NRC>
static void run_getrs_warp(cudaStream_t s, int trans, int n, int nrhs, Batch<T> A, int lda,
                           const int* ipiv, int64_t sP, Batch<T> B, int ldb, const int* skip,
                           int bc, Gate g)
{
    const int64_t tasks = (int64_t)bc * ((nrhs + NRC - 1) / NRC);
    dim3 grid((unsigned)((tasks + SMALL_WPB - 1) / SMALL_WPB));
    RSB_LOG_KERNEL("getrs_warp_kernel");
    getrs_warp_kernel<T, NMAX, NRC><<<grid, 32 * SMALL_WPB, 0, s>>>(trans, n, nrhs, A, lda, ipiv,
                                                                     sP, B, ldb, skip, bc, g);
}

template <typename T, int NMAX>
static void getrs_warp_nrc(cudaStream_t s, int trans, int n, int nrhs, Batch<T> A, int lda,
                           const int* ipiv, int64_t sP, Batch<T> B, int ldb, const int* skip,
                           int bc, Gate g)
{
    if(nrhs == 1)
        run_getrs_warp<T, NMAX, 1>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
    else
        run_getrs_warp<T, NMAX, 4>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
}

template <typename T, int NT, int NRC>
static rocblas_status run_getrs_cta_nt(cudaStream_t s, int trans, int n, int nrhs, Batch<T> A,
                                       int lda, const int* ipiv, int64_t sP, Batch<T> B,
                                       int ldb, const int* skip, int bc, Gate g)
{
    const size_t smem =
        sizeof(T) * ((size_t)n * NRC + sweep_scratch<NT>()) + sizeof(int) * (size_t)n;
    auto k = getrs_cta_kernel<T, NT, NRC>;
    if(!set_smem(k, smem))
        return rocblas_status_internal_error;
    const int64_t groups = (nrhs + NRC - 1) / NRC;
    RSB_LOG_KERNEL("getrs_cta_kernel");
    k<<<(unsigned)(bc * groups), NT, smem, s>>>(trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip,
                                                g);
    return launch_status();
}

// CTA size follows n: one thread per row for the off-diagonal updates
template <typename T, int NRC>
static rocblas_status run_getrs_cta(cudaStream_t s, int trans, int n, int nrhs, Batch<T> A,
                                    int lda, const int* ipiv, int64_t sP, Batch<T> B, int ldb,
                                    const int* skip, int bc, Gate g)
{
    if(n <= 64)
        return run_getrs_cta_nt<T, 64, NRC>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip,
                                            bc, g);
    if(n <= 128)
        return run_getrs_cta_nt<T, 128, NRC>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip,
                                             bc, g);
    return run_getrs_cta_nt<T, 256, NRC>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc,
                                         g);
}

template <typename T>
rocblas_status launch_getrs(cudaStream_t s, int trans, int n, int nrhs, Batch<T> A, int lda,
                            const int* ipiv, int64_t sP, Batch<T> B, int ldb, const int* skip,
                            int bc, Gate g)
{
    if(n <= 8)
        getrs_warp_nrc<T, 8>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
    else if(n <= 16)
        getrs_warp_nrc<T, 16>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
    else if(n <= 32)
        getrs_warp_nrc<T, 32>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
    else if(n <= 4096)
        return nrhs == 1
                   ? run_getrs_cta<T, 1>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g)
                   : run_getrs_cta<T, 4>(s, trans, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, g);
    else
        return rocblas_status_not_implemented;
    return launch_status();
}

// ------------------------------------------------------------------------------ gesv
template <typename T, int NMAX>
static void run_gesv_warp(cudaStream_t s, int n, int nrhs, Batch<T> A, int lda, int* ipiv,
                          int64_t sP, Batch<T> B, int ldb, int* info, int bc)
{
    dim3 grid((bc + SMALL_WPB - 1) / SMALL_WPB);
    RSB_LOG_KERNEL("gesv_warp_kernel");
    if(nrhs == 1)
        gesv_warp_kernel<T, NMAX, 1><<<grid, 32 * SMALL_WPB, 0, s>>>(n, nrhs, A, lda, ipiv, sP,
                                                                      B, ldb, info, bc);
    else
        gesv_warp_kernel<T, NMAX, 4><<<grid, 32 * SMALL_WPB, 0, s>>>(n, nrhs, A, lda, ipiv, sP,
                                                                      B, ldb, info, bc);
}

template <typename T>
rocblas_status launch_gesv(cudaStream_t s, int n, int nrhs, Batch<T> A, int lda, int* ipiv,
                           int64_t sP, Batch<T> B, int ldb, int* info, int bc)
{
    if(n <= 32)
    {
        if(n <= 8)
            run_gesv_warp<T, 8>(s, n, nrhs, A, lda, ipiv, sP, B, ldb, info, bc);
        else if(n <= 16)
            run_gesv_warp<T, 16>(s, n, nrhs, A, lda, ipiv, sP, B, ldb, info, bc);
        else
            run_gesv_warp<T, 32>(s, n, nrhs, A, lda, ipiv, sP, B, ldb, info, bc);
        return launch_status();
    }
    rocblas_status st = launch_getrf<T>(s, n, n, A, lda, ipiv, sP, info, bc, true);
    if(st != rocblas_status_success)
        return st;
    return launch_getrs<T>(s, 0, n, nrhs, A, lda, ipiv, sP, B, ldb, info, bc);
}

// ------------------------------------------------------------------------------ potrf
template <typename T, int N, bool BLOCK>
static rocblas_status run_potrf_reg(cudaStream_t s, int upper, int n, Batch<T> A, int lda,
                                    int* info, int bc, int j0 = 0)
{
    RSB_LOG_KERNEL("potrf_reg_kernel");
    if(upper)
        potrf_reg_kernel<T, N, true, BLOCK><<<bc, N, 0, s>>>(n, A, lda, info, j0);
    else
        potrf_reg_kernel<T, N, false, BLOCK><<<bc, N, 0, s>>>(n, A, lda, info, j0);
    return launch_status();
}

// n > 64: steps of 64 columns (chol_blk.cuh)
template <typename T, bool UPPER>
static rocblas_status run_potrf_blk(cudaStream_t s, int n, Batch<T> A, int lda, int* info, int bc)
{
    constexpr int NB = BLK_NB;
    if(!set_smem(potrf_trsm_kernel<T, UPPER>, sizeof(CholTrsmSmem<T>))
       || !set_smem(potrf_syrk_kernel<T, UPPER>, sizeof(GemmSmem<T>)))
        return rocblas_status_internal_error;
    for(int j0 = 0; j0 < n; j0 += NB)
    {
        const int jb = std::min(NB, n - j0), below = n - j0 - jb;
        const rocblas_status st =
            jb <= 32 ? run_potrf_reg<T, 32, true>(s, UPPER, jb, A, lda, info, bc, j0)
                     : run_potrf_reg<T, 64, true>(s, UPPER, jb, A, lda, info, bc, j0);
        if(st != rocblas_status_success || below <= 0)
            return st;
        const int chunks = (below + CHOL_CW - 1) / CHOL_CW, t = (below + 63) / 64;
        const int tiles = t * (t + 1) / 2;
        {
            RSB_LOG_KERNEL("potrf_trsm_kernel");
            potrf_trsm_kernel<T, UPPER><<<(unsigned)((int64_t)bc * chunks), CHOL_NT,
                                          sizeof(CholTrsmSmem<T>), s>>>(n, A, lda, info, j0,
                                                                        chunks);
        }
        if(launch_status() != rocblas_status_success)
            return rocblas_status_internal_error;
        {
            RSB_LOG_KERNEL("potrf_syrk_kernel");
            potrf_syrk_kernel<T, UPPER><<<(unsigned)((int64_t)bc * tiles), 128,
                                          sizeof(GemmSmem<T>), s>>>(n, A, lda, info, j0, tiles);
        }
        if(launch_status() != rocblas_status_success)
            return rocblas_status_internal_error;
    }
    return rocblas_status_success;
}

template <typename T>
rocblas_status launch_potrf(cudaStream_t s, int upper, int n, Batch<T> A, int lda, int* info,
                            int bc)
{
    if(n <= 32)
        return run_potrf_reg<T, 32, false>(s, upper, n, A, lda, info, bc);
    if(n <= 64)
        return run_potrf_reg<T, 64, false>(s, upper, n, A, lda, info, bc);
    if(n > MAX_CTA_ROWS)
        return rocblas_status_not_implemented;
    return upper ? run_potrf_blk<T, true>(s, n, A, lda, info, bc)
                 : run_potrf_blk<T, false>(s, n, A, lda, info, bc);
}

template <typename T, int NT, int NRC>
static rocblas_status run_potrs_nt(cudaStream_t s, int upper, int n, int nrhs, Batch<T> A,
                                   int lda, Batch<T> B, int ldb, const int* skip, int bc)
{
    const size_t smem = sizeof(T) * ((size_t)n * NRC + sweep_scratch<NT>());
    auto k = potrs_cta_kernel<T, NT, NRC>;
    if(!set_smem(k, smem))
        return rocblas_status_internal_error;
    const int64_t groups = (nrhs + NRC - 1) / NRC;
    RSB_LOG_KERNEL("potrs_cta_kernel");
    k<<<(unsigned)(bc * groups), NT, smem, s>>>(upper, n, nrhs, A, lda, B, ldb, skip);
    return launch_status();
}

template <typename T, int N, int NRC>
static rocblas_status run_potrs_small(cudaStream_t s, int upper, int n, int nrhs, Batch<T> A,
                                      int lda, Batch<T> B, int ldb, const int* skip, int bc)
{
    const int64_t groups = (nrhs + NRC - 1) / NRC;
    RSB_LOG_KERNEL("potrs_small_kernel");
    potrs_small_kernel<T, N, NRC>
        <<<(unsigned)(bc * groups), N, 0, s>>>(upper, n, nrhs, A, lda, B, ldb, skip);
    return launch_status();
}

template <typename T, int NRC>
static rocblas_status run_potrs(cudaStream_t s, int upper, int n, int nrhs, Batch<T> A,
                                int lda, Batch<T> B, int ldb, const int* skip, int bc)
{
    if(n <= 32)
        return run_potrs_small<T, 32, NRC>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc);
    if(n <= 64)
        return run_potrs_small<T, 64, NRC>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc);
    if(n <= 128)
        return run_potrs_nt<T, 128, NRC>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc);
    return run_potrs_nt<T, 256, NRC>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc);
}

template <typename T>
rocblas_status launch_potrs(cudaStream_t s, int upper, int n, int nrhs, Batch<T> A, int lda,
                            Batch<T> B, int ldb, const int* skip, int bc)
{
    if(n > 4096)
        return rocblas_status_not_implemented;
    return nrhs == 1 ? run_potrs<T, 1>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc)
                     : run_potrs<T, 4>(s, upper, n, nrhs, A, lda, B, ldb, skip, bc);
}

// Solve with many right-hand sides (getri's n columns of the identity): 32 columns per CTA
// through shared memory for 32 < n <= 512, so that each CTA's pass over the factors (and its
// diagonal-block inversions) serves 32 columns instead of 4; otherwise launch_getrs.
template <typename T>
rocblas_status launch_getrs_many(cudaStream_t s, int n, int nrhs, Batch<T> A, int lda,
                                 const int* ipiv, int64_t sP, Batch<T> B, int ldb,
                                 const int* skip, int bc)
{
    if(n <= 32 || n > 512 || nrhs < 32)
        return launch_getrs<T>(s, 0, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, no_gate());
    return run_getrs_cta<T, 32>(s, 0, n, nrhs, A, lda, ipiv, sP, B, ldb, skip, bc, no_gate());
}

// ------------------------------------------------------------------------------ instances
#define RSB_INST(T)                                                                          \
    template rocblas_status launch_getrf<T>(cudaStream_t, int, int, Batch<T>, int, int*,   \
                                            int64_t, int*, int, bool, Gate, bool);         \
    template rocblas_status launch_getrs<T>(cudaStream_t, int, int, int, Batch<T>, int,    \
                                            const int*, int64_t, Batch<T>, int, const int*, \
                                            int, Gate);                                    \
    template rocblas_status launch_gesv<T>(cudaStream_t, int, int, Batch<T>, int, int*,    \
                                           int64_t, Batch<T>, int, int*, int);             \
    template rocblas_status launch_potrf<T>(cudaStream_t, int, int, Batch<T>, int, int*,   \
                                            int);                                          \
    template rocblas_status launch_potrs<T>(cudaStream_t, int, int, int, Batch<T>, int,    \
                                            Batch<T>, int, const int*, int);               \
    template rocblas_status launch_getrs_many<T>(cudaStream_t, int, int, Batch<T>, int,    \
                                                 const int*, int64_t, Batch<T>, int,       \
                                                 const int*, int);
RSB_INST(float)
RSB_INST(double)

} // namespace rsb
