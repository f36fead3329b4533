// chol_blk.cuh -- right-looking blocked Cholesky for n > 64 in separate launches per step.
//
// Replaces the reference's blocked potrf (library/src/lapack/roclapack_potrf.hpp:90-228).  One
// step takes 64 columns of every member: potrf_reg_kernel (chol.cuh) factors the diagonal
// block, potrf_trsm_kernel forms the panel below it, L21 = A21 L11^{-T}, and
// potrf_syrk_kernel updates the trailing triangle, A22 -= L21 L21', on 64 x 64 tiles.  The
// upper case (A = U' U) is the same on the transposed view; both read and write along the
// stored columns.  Members whose info is set are left alone, except that a member that failed
// in this step still gets the finished columns of its panel (LAPACK potf2).
//
// potrf alone against one CTA per member with a barrier per column: FP32 n = 200 x 1500 0.56 ms
// (4.2), of it updates 0.25, panels 0.16 and diagonal blocks 0.15; FP64 n = 128 x 4882 0.62 (9.2),
// n = 65 x 1 0.040 (0.093), n = 2048 x 16 4.3 (358).  One launch of the diagonal block is a serial
// chain of 64 columns, which is what small batches wait for.
#pragma once

#include "lu_blk.cuh" // GemmTile, cp.async helpers

namespace rsb {

constexpr int CHOL_NT = 128, CHOL_CW = 64;

template <typename T>
struct CholTrsmSmem
{
    T L[BLK_NB][BLK_NB + 4];   // [k][i] = L11(i, k); only i >= k is used
    T X[CHOL_CW][BLK_NB + 1];  // [row of L21][k]
    T rd[BLK_NB];              // 1 / L11(k, k)
};

// rows of L21 in chunks of 64: X L11' = A21 by substitution over blocks of 16 columns (the
// finished columns' part on tensor tiles in FP64, as lu_swap_trsm_kernel), one thread per row
template <typename T, bool UPPER>
__global__ void __launch_bounds__(CHOL_NT, sizeof(T) == 8 ? 3 : 5)
    potrf_trsm_kernel(int n, Batch<T> A, int lda, const int* info, int j0, int chunks)
{
    constexpr int NB = BLK_NB, NT = CHOL_NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CholTrsmSmem<T>& sm = *reinterpret_cast<CholTrsmSmem<T>*>(smem_raw);
    const int64_t b = blockIdx.x / chunks;
    const int inf = info[b];
    const int jb = inf == 0 ? NB : inf - 1 - j0; // columns to form (a whole panel has NB)
    if(jb <= 0)
        return;
    T* a = A.at(b);
    const int r0 = j0 + NB + (blockIdx.x % chunks) * CHOL_CW;
    const int nr = min(CHOL_CW, n - r0);
    const int tid = threadIdx.x, warp = tid >> 5;
    auto at = [&](int r, int c) -> T& {
        return UPPER ? RSB_AT(a, c, r, lda, n, n) : RSB_AT(a, r, c, lda, n, n);
    };
    for(int e = tid; e < NB * NB; e += NT)
    {
        const int p = e & (NB - 1), q = e / NB; // p runs along the stored column
        const int i = UPPER ? q : p, k = UPPER ? p : q;
        if(i < jb && k <= i)
            cp_async(&sm.L[k][i], &at(j0 + i, j0 + k));
    }
    for(int e = tid; e < NB * CHOL_CW; e += NT)
    {
        const int p = e & (NB - 1), q = e / NB;
        const int r = UPPER ? q : p, k = UPPER ? p : q;
        if(r < nr && k < jb)
            cp_async(&sm.X[r][k], &at(r0 + r, j0 + k));
    }
    cp_async_wait();
    __syncthreads();
    if(tid < jb)
        sm.rd[tid] = T(1) / sm.L[tid][tid];
    __syncthreads();
#pragma unroll 1
    for(int ib = 0; ib < jb; ib += 16)
    {
        if constexpr(sizeof(T) == 8)
        {
            if(ib > 0 && warp * 16 < nr)
                trsm_tile(sm.L, &sm.X[warp * 16][0], ib);
            __syncthreads();
        }
        if(tid < nr)
        {
            T acc[16];
            T* x = sm.X[tid];
#pragma unroll
            for(int r = 0; r < 16; ++r)
                acc[r] = x[ib + r];
            if constexpr(sizeof(T) == 4)
            {
#pragma unroll 2
                for(int k = 0; k < ib; ++k)
                {
                    const T xk = x[k];
#pragma unroll
                    for(int r = 0; r < 16; ++r)
                        acc[r] = fma(-sm.L[k][ib + r], xk, acc[r]);
                }
            }
#pragma unroll
            for(int r = 0; r < 16; ++r)
            {
                acc[r] *= sm.rd[ib + r];
#pragma unroll
                for(int q = r + 1; q < 16; ++q)
                    acc[q] = fma(-sm.L[ib + r][ib + q], acc[r], acc[q]);
            }
#pragma unroll
            for(int r = 0; r < 16; ++r)
                x[ib + r] = acc[r];
        }
        if constexpr(sizeof(T) == 8)
            __syncthreads();
    }
    __syncthreads();
    for(int e = tid; e < NB * CHOL_CW; e += NT)
    {
        const int p = e & (NB - 1), q = e / NB;
        const int r = UPPER ? q : p, k = UPPER ? p : q;
        if(r < nr && k < jb)
            at(r0 + r, j0 + k) = sm.X[r][k];
    }
}

// W(i, j) -= sum_k X(i, k) X(j, k) on 64 x 64 tiles of the stored triangle of the trailing
// matrix, X the panel's 64 columns of L21 (upper: rows of U12): both operands are staged
// [k][row], the tile of W starts (negated) in the accumulators
template <typename T, bool UPPER>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 3 : 4)
    potrf_syrk_kernel(int n, Batch<T> A, int lda, const int* info, int j0, int tiles)
{
    using Tile = GemmTile<T, false>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GemmSmem<T>& sm = *reinterpret_cast<GemmSmem<T>*>(smem_raw);
    const int64_t b = blockIdx.x / tiles;
    if(info[b] != 0)
        return;
    T* a = A.at(b);
    // t-th pair (hi, lo) with hi >= lo
    const int t = blockIdx.x % tiles;
    int hi = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while((hi + 1) * (hi + 2) / 2 <= t)
        ++hi;
    while(hi * (hi + 1) / 2 > t)
        --hi;
    const int lo = t - hi * (hi + 1) / 2;
    const int base = j0 + BLK_NB;
    const int r0 = base + (UPPER ? lo : hi) * 64, c0 = base + (UPPER ? hi : lo) * 64;
    const int nr = min(64, n - r0), nc = min(64, n - c0);
    const bool diag = hi == lo;
    const int tid = threadIdx.x, warp = tid >> 5;
    auto stage = [&](T(*d)[GEMM_LD], int row0, int cnt) {
        for(int e = tid; e < 64 * 64; e += 128)
        {
            // lower: 64 consecutive rows; upper: 8 k x 4 rows (k is contiguous)
            const int i = UPPER ? (((e >> 3) & 15) | ((e >> 6) & 0x30)) : (e & 63);
            const int k = UPPER ? ((e & 7) | ((e >> 4) & 0x38)) : (e >> 6);
            if(i < cnt)
                cp_async(&d[k][i], UPPER ? &RSB_AT(a, j0 + k, row0 + i, lda, n, n)
                                         : &RSB_AT(a, row0 + i, j0 + k, lda, n, n));
            else
                d[k][i] = T(0);
        }
    };
    stage(sm.A, r0, nr);
    if(!diag)
        stage(sm.B, c0, nc);
    const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
    const bool live = wr < nr && wc < nc && !(diag && (UPPER ? wr > wc : wr < wc));
    auto in = [&](int r, int c) {
        return wr + r < nr && wc + c < nc
               && (!diag || (UPPER ? wr + r <= wc + c : wr + r >= wc + c));
    };
    Tile w;
    if(live)
        w.each([&](int r, int c, auto& v) {
            v = in(r, c) ? -RSB_AT(a, r0 + wr + r, c0 + wc + c, lda, n, n) : T(0);
        });
    cp_async_wait();
    __syncthreads();
    if(live)
    {
        w.template mma<false>(&sm.A[0][0], diag ? &sm.A[0][0] : &sm.B[0][0], wr, wc, BLK_NB);
        w.each([&](int r, int c, auto& v) {
            if(in(r, c))
                RSB_AT(a, r0 + wr + r, c0 + wc + c, lda, n, n) = -v;
        });
    }
}

} // namespace rsb
