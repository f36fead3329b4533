// chol.cuh -- register-resident Cholesky of up to 64 columns (lower or upper): whole members
// of n <= 64, and the diagonal blocks of the blocked factorisation (chol_blk.cuh).
//
// Replaces the reference's unblocked potf2 (library/src/lapack/roclapack_potf2.hpp:137-253),
// which at n = 64 issues ~256 launches per call (dot, sqrtDiagOnward with 1-thread blocks,
// gemv, scal per column).
//
// The upper case (A = U' U) is the lower algorithm on the transposed view
// M(r, c) = A[c + r*lda].  The first non-positive (or NaN) pivot is stored, info is set to
// its 1-based index and the factorisation stops, as LAPACK dpotf2 does; the reference
// (sqrtDiagOnward, :16-43) records the same info.
#pragma once

#include "common.cuh"

namespace rsb {

// ---------------------------------------------------------------------------------------
// Small orders (n <= N, N = 32 or 64): one thread per row, the row's lower-triangle
// entries in registers for the whole factorisation, one CTA barrier per column.
// Rolled column loop: at step c, v[i] holds A(r, c + i) of this thread's row r, so the
// active column is always v[0] and the rank-1 update writes column c+1+i into v[i].  At
// step c every row r >= c publishes A(r, c) (already updated by steps < c) at slot r-c of
// a double-buffered column vector, the diagonal row also publishes sqrt and 1/sqrt of its
// pivot (computed before the barrier), and after ONE barrier each row r > c forms
// l = A(r, c) / L(c, c), stores it, and updates
//   A(r, c+1+i) -= (l / L(c, c)) * A(c+1+i, c),   i = 0 .. N-2,
// reading the published column as aligned vectors.  Entries right of the diagonal are
// updated too (never stored) up to the warp's last row; beyond it they are skipped in
// groups of 8.  Each row stores its column-c entry as it is finalised.
// A non-positive or NaN pivot at step c: columns < c are final, A(c, c) keeps the updated
// value, the rest of the matrix is untouched and info = c + 1 (LAPACK dpotf2).
// UPPER: M(r, c) = A(c, r).  BLOCK: the n columns at (j0, j0) of a larger member (blocked
// potrf); members whose info is already set are left alone, and the upper triangle is staged in
// shared memory on the way in and out, along its stored columns.  Whole members of the upper
// case are not staged: the extra pass costs a small batch more than the strided accesses (FP64
// n = 32 x 16 14.2 against 10.1 us staged / direct, n = 48 x 148 21.2 / 17.0), and a large one
// at most orders (n = 24 x 20000 122 / 101 us, n = 48 x 20000 565 / 477, n = 64 x 20000 750 /
// 752; gains were FP32 n = 64 x 20000 449 / 508 and n = 32 x 20000 92 / 123).
template <typename T, int N, bool UPPER, bool BLOCK>
__global__ void __launch_bounds__(N, N <= 32 ? 16 : 6)
    potrf_reg_kernel(int n, Batch<T> A, int lda, int* info, int j0)
{
    constexpr bool STAGE = UPPER && BLOCK;
    __shared__ T tri[STAGE ? N : 1][N + 1]; // [row][column]
    // published column (slot r - c); rows of N + 4 elements keep both buffers 16-byte
    // aligned for the vector reads in FP32 and FP64
    __shared__ __align__(16) T scol[2][N + 4];
    __shared__ T sdiag[2][2];                  // sqrt(pivot), 1/sqrt(pivot)
    const int r = threadIdx.x;
    const int64_t b = blockIdx.x;
    if(BLOCK && j0 > 0 && info[b] != 0)
        return;
    T* a = A.at(b) + (BLOCK ? ix(j0, j0, lda) : 0);
    auto at = [&](int i, int j) -> T& {
        return STAGE ? tri[i][j] : (UPPER ? a[ix(j, i, lda)] : a[ix(i, j, lda)]);
    };
    if(STAGE)
    {
#pragma unroll 8
        for(int i = 0; i < n; ++i)
            if(r <= i)
                tri[i][r] = a[ix(r, i, lda)];
        __syncthreads();
    }
    T v[N];
#pragma unroll
    for(int i = 0; i < N; ++i)
        v[i] = (r < n && i <= r) ? at(r, i) : T(0);
    int inf = 0;
#pragma unroll 1
    for(int c = 0; c < n; ++c)
    {
        const int buf = c & 1;
        if(r == c)
        {
            const T d = v[0];
            const bool ok = d > T(0);
            const T sq = ok ? sqrt(d) : d;
            sdiag[buf][0] = sq;
            sdiag[buf][1] = ok ? T(1) / sq : T(0);
            at(c, c) = sq; // LAPACK also stores a failing pivot as it was computed
        }
        else if(r > c && r < n)
            scol[buf][r - c - 1] = v[0];
        __syncthreads();
        const T sq = sdiag[buf][0];
        if(!(sq > T(0)))
        {
            inf = c + 1;
            break;
        }
        const T rcp = sdiag[buf][1];
        if(r > c && r < n)
        {
            const T l = v[0] * rcp;
            at(r, c) = l;
            const T lr = l * rcp;
            const T* col = scol[buf];
            // only columns up to the warp's last row matter: groups of 8 registers above
            // that are skipped (the branch is uniform across the warp)
            const int lim = min(32 * (r >> 5) + 31, n - 1) - c - 1;
#pragma unroll
            for(int g = 0; g < N; g += 8)
            {
                if(g > lim)
                    break;
                if constexpr(sizeof(T) == 8)
                {
#pragma unroll
                    for(int i = g; i < g + 8; i += 2)
                    {
                        const double2 t = *reinterpret_cast<const double2*>(col + i);
                        if(i + 1 < N)
                            v[i] = fma(-lr, t.x, v[i + 1]);
                        if(i + 2 < N)
                            v[i + 1] = fma(-lr, t.y, v[i + 2]);
                    }
                }
                else
                {
#pragma unroll
                    for(int i = g; i < g + 8; i += 4)
                    {
                        const float4 t = *reinterpret_cast<const float4*>(col + i);
                        const float e[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                        for(int u = 0; u < 4; ++u)
                            if(i + u + 1 < N)
                                v[i + u] = fmaf(-lr, e[u], v[i + u + 1]);
                    }
                }
            }
        }
    }
    if(STAGE)
    {
        __syncthreads();
        for(int i = 0; i < n; ++i)
            if(r <= i)
                a[ix(r, i, lda)] = tri[i][r];
    }
    if(r == 0 && (!BLOCK || j0 == 0 || inf != 0))
        info[b] = inf != 0 && BLOCK ? j0 + inf : inf;
}

} // namespace rsb
