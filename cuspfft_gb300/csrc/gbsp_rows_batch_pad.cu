// gbsp_rows_batch_pad.cu -- the batched row kernel with padded row buffers.
#include "gbsp_rows_batch.cuh"

namespace gbsp {

int rows_batch_blocks_per_sm_pad(const RowBlock& rb, size_t smem, int* nb) {
    return rows_batch::blocks_per_sm<true>(rb, smem, nb);
}

int rows_batch_launch_pad(const RowBlock& rb, int grid, size_t smem, cudaStream_t st, const RowsBatch* descs,
                          const long* row_begin, int nmat, unsigned long long* queue, bool pdl, int* err) {
    return rows_batch::launch<true>(rb, grid, smem, st, descs, row_begin, nmat, queue, pdl, err);
}

}  // namespace gbsp
