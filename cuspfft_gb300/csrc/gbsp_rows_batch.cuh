// gbsp_rows_batch.cuh -- launch helpers of the batched row kernel, shared by
// gbsp_rows_batch.cu and gbsp_rows_batch_pad.cu (each compiles its own
// instances, at both block bounds).
#pragma once
#include "gbsp_launch.h"

namespace gbsp {
namespace rows_batch {

template <bool PAD, int NTMAX>
int blocks_per_sm(int nt, size_t smem, int* nb) {
    auto kern = k_bluestein_rows_batch<NTMAX, PAD>;
    if (int rc = allow_full_smem((const void*)kern)) return rc;
    GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(nb, kern, nt, smem));
    return GBSP_OK;
}
template <bool PAD>
int blocks_per_sm(const RowBlock& rb, size_t smem, int* nb) {
    return rb.ntmax == 512 ? blocks_per_sm<PAD, 512>(rb.nt, smem, nb) : blocks_per_sm<PAD, 1024>(rb.nt, smem, nb);
}

template <bool PAD>
int launch(const RowBlock& rb, int grid, size_t smem, cudaStream_t st, const RowsBatch* descs, const long* row_begin,
           int nmat, unsigned long long* queue, bool pdl, int* err) {
    GB_CUDA(launch_kernel(rb.ntmax == 512 ? k_bluestein_rows_batch<512, PAD> : k_bluestein_rows_batch<1024, PAD>, grid,
                          rb.nt, smem, st, pdl, 1, descs, row_begin, nmat, queue, err));
    return GBSP_OK;
}

}  // namespace rows_batch
}  // namespace gbsp
