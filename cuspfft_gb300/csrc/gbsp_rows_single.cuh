// gbsp_rows_single.cuh -- launch helpers of the single-channel row kernels,
// shared by gbsp_rows.cu, gbsp_rows_384.cu and gbsp_rows_pad.cu (each compiles
// its own instances).
#pragma once
#include "gbsp_launch.h"

namespace gbsp {
namespace rows_single {

template <int NTMAX, int MODE, bool PAD>
int capacity(const RowsKernel& k, int sms, int* cap) {
    auto kern = k_bluestein_rows<NTMAX, MODE, PAD>;
    if (int rc = allow_full_smem((const void*)kern)) return rc;
    int nb = 0;
    GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, k.nt, k.smem));
    *cap = nb * sms;
    return GBSP_OK;
}

template <int NTMAX, int MODE, bool PAD>
int launch(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err) {
    GB_CUDA(launch_kernel(k_bluestein_rows<NTMAX, MODE, PAD>, grid, k.nt, k.smem, st, pdl, 1, a, fd, err));
    return GBSP_OK;
}

}  // namespace rows_single
}  // namespace gbsp
