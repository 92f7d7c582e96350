// gbsp_rows_batch.cu -- the batched row kernel and its host launch functions.
#include "gbsp_rows_batch.cuh"

namespace gbsp {

int rows_batch_blocks_per_sm(const RowBlock& rb, bool pad, size_t smem, int* nb) {
    return pad ? rows_batch_blocks_per_sm_pad(rb, smem, nb) : rows_batch::blocks_per_sm<false>(rb, smem, nb);
}

int rows_batch_launch(const RowBlock& rb, bool pad, int grid, size_t smem, cudaStream_t st, const RowsBatch* descs,
                      const long* row_begin, int nmat, unsigned long long* queue, bool pdl, int* err) {
    return pad ? rows_batch_launch_pad(rb, grid, smem, st, descs, row_begin, nmat, queue, pdl, err)
               : rows_batch::launch<false>(rb, grid, smem, st, descs, row_begin, nmat, queue, pdl, err);
}

}  // namespace gbsp
