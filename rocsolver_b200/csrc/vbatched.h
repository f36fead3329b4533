// vbatched.h -- the description of a variable-size batch, shared by the kernels that walk it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace rsb {

constexpr int VB_SMALL = 32; // members with n <= VB_SMALL use the warp path

struct VbArgs
{
    int bc, max_n, max_nrhs, mode; // mode: 0 gesv, 1 getrf, 2 getrs
    const int* n;
    const int* nrhs;
    const int* lda;
    const int* ldb;
    int* const* ipiv;
    int* info;
    int* order;    // [bc]
    int* counters; // [0] big cursor, [1] small cursor, [2] number of big members
};

__device__ __forceinline__ bool vb_valid(const VbArgs& v, int b)
{
    const int n = v.n[b];
    if(n < 0 || n > v.max_n || v.lda[b] < max(1, n))
        return false;
    if(v.mode != 1)
    {
        const int r = v.nrhs[b];
        if(r < 0 || r > v.max_nrhs || v.ldb[b] < max(1, n))
            return false;
    }
    return true;
}

} // namespace rsb
