// lu_blk.cu -- launches of the blocked LU (lu_blk.cuh).
#include "lu_blk.h"

#include <algorithm>
#include <cstdlib>

#include "logger.h"

namespace rsb {
namespace {

template <typename K>
bool set_smem(K kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)
           == cudaSuccess;
}

rocblas_status launched()
{
    return cudaGetLastError() == cudaSuccess ? rocblas_status_success
                                             : rocblas_status_internal_error;
}

// polls after which a wait between the CTAs of a cluster gives up; the bounds-checked build
// takes another limit from the environment, so that a test can see the waits run out
int cluster_wait_limit()
{
#ifdef RSB_BOUNDS_CHECK
    if(const char* e = std::getenv("ROCSOLVER_B200_CLUSTER_WAIT"))
        return std::atoi(e);
#endif
    return CLUSTER_WAIT_LIMIT;
}

template <typename T, int S, bool PIVOT, bool CL>
rocblas_status panel(cudaStream_t s, const LuBatch<T>& L, int j0, int bc, int cluster, bool first)
{
    auto k = lu_panel_kernel<T, BLK_NB, S, PIVOT, CL>;
    const size_t smem = sizeof(PanelSmem<T, BLK_NB, S, CL>);
    if(first && !set_smem(k, smem))
        return rocblas_status_internal_error;
    RSB_LOG_KERNEL("getrf_panel_kernel");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((int64_t)bc * cluster));
    cfg.blockDim = dim3(PanelShape<T, S>::NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CL ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, L, j0, cluster_wait_limit()) == cudaSuccess
               ? launched()
               : rocblas_status_internal_error;
}

// CTAs of 64, 128 or 256 rows (1, 2, 3) or clusters of CTAs of 256 (4)
int panel_class(int rows)
{
    return rows <= 64 ? 1 : rows <= 128 ? 2 : rows <= 256 ? 3 : 4;
}

// the panel at j0: the smallest CTA that holds the rows, or a cluster of CTAs of 256 rows;
// first: this class's kernel has not been launched in this call
template <typename T, bool PIVOT>
rocblas_status panel_rows(cudaStream_t s, const LuBatch<T>& L, int j0, int rows, int bc,
                          bool first)
{
    switch(panel_class(rows))
    {
    case 1: return panel<T, 2, PIVOT, false>(s, L, j0, bc, 1, first);
    case 2: return panel<T, 4, PIVOT, false>(s, L, j0, bc, 1, first);
    case 3: return panel<T, 8, PIVOT, false>(s, L, j0, bc, 1, first);
    }
    return panel<T, 8, PIVOT, true>(s, L, j0, bc, rows <= 512 ? 2 : (rows <= 1024 ? 4 : 8), first);
}

template <typename T, bool PIVOT, bool TC>
rocblas_status lu_blk(cudaStream_t s, const LuBatch<T>& L, int m, int n, int bc)
{
    constexpr int NB = BLK_NB;
    const int mn = std::min(m, n);
    rocblas_status st = rocblas_status_success;
    int cls = 0;
    for(int j0 = 0; j0 < mn; j0 += NB)
    {
        const int rows = m - j0, jb = std::min(NB, mn - j0);
        const bool first = panel_class(rows) != cls;
        cls = panel_class(rows);
        st = panel_rows<T, PIVOT>(s, L, j0, rows, bc, first);
        if(st != rocblas_status_success)
            return st;
        const int right = n - j0 - jb, below = m - j0 - jb;
        if(right <= 0)
            break;
        {
            auto k = lu_swap_trsm_kernel<T, PIVOT>;
            if(j0 == 0 && !set_smem(k, sizeof(TrsmSmem<T>)))
                return rocblas_status_internal_error;
            const int chunks = (right + TRSM_CW - 1) / TRSM_CW;
            RSB_LOG_KERNEL("getrf_swap_trsm_kernel");
            k<<<(unsigned)((int64_t)bc * chunks), TRSM_NT, sizeof(TrsmSmem<T>), s>>>(L, j0, chunks);
            if((st = launched()) != rocblas_status_success)
                return st;
        }
        if(below > 0)
        {
            auto k = lu_gemm_kernel<T, TC>;
            if(j0 == 0 && !set_smem(k, sizeof(GemmSmem<T>)))
                return rocblas_status_internal_error;
            const int tm = (below + 63) / 64, tn = (right + 63) / 64;
            RSB_LOG_KERNEL("getrf_gemm_kernel");
            k<<<(unsigned)((int64_t)bc * tm * tn), 128, sizeof(GemmSmem<T>), s>>>(L, j0, tm * tn,
                                                                                 tm);
            if((st = launched()) != rocblas_status_success)
                return st;
        }
    }
    if(PIVOT && mn > NB)
    {
        const int blocks = (mn + NB - 1) / NB - 1, rows = m - NB;
        auto k = lu_left_kernel<T>;
        const size_t smem = LEFT_BUF + 2 * sizeof(int) * (size_t)rows;
        if(!set_smem(k, smem))
            return rocblas_status_internal_error;
        RSB_LOG_KERNEL("getrf_left_kernel");
        k<<<(unsigned)((int64_t)bc * blocks * (NB / LEFT_COLS)), LEFT_NT, smem, s>>>(L, blocks,
                                                                                     rows);
        st = launched();
    }
    return st;
}

} // namespace

template <typename T>
rocblas_status launch_lu_blk(cudaStream_t s, const LuBatch<T>& L, int m, int n, int bc,
                             bool pivot, bool tc)
{
    if(m > MAX_CTA_ROWS)
        return rocblas_status_not_implemented;
    if constexpr(sizeof(T) == 4)
        if(tc && pivot)
            return lu_blk<T, true, true>(s, L, m, n, bc);
    return pivot ? lu_blk<T, true, false>(s, L, m, n, bc) : lu_blk<T, false, false>(s, L, m, n, bc);
}

template rocblas_status launch_lu_blk<float>(cudaStream_t, const LuBatch<float>&, int, int, int,
                                             bool, bool);
template rocblas_status launch_lu_blk<double>(cudaStream_t, const LuBatch<double>&, int, int, int,
                                              bool, bool);

} // namespace rsb
