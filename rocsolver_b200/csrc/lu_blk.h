// lu_blk.h -- host interface of the blocked LU (lu_blk.cuh).
#pragma once

#include "launch.h"
#include "lu_blk.cuh"

namespace rsb {

// LU of the bc members of L (m x n, m <= 2048)
template <typename T>
rocblas_status launch_lu_blk(cudaStream_t s, const LuBatch<T>& L, int m, int n, int bc,
                             bool pivot, bool tc);

} // namespace rsb
