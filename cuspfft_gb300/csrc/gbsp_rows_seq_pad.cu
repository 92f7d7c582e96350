// gbsp_rows_seq_pad.cu -- sequential channels with a padded row buffer (last
// radix a power of two).
#include "gbsp_rows_impl.cuh"

namespace gbsp {

int rows_capacity_seq_pad(const RowsKernel& k, int sms, int* cap) {
    return k.mode == ROW_SEQ2 ? rows_impl::capacity<512, ROW_SEQ2, true>(k, sms, cap)
                              : rows_impl::capacity<512, ROW_SEQ, true>(k, sms, cap);
}

int rows_launch_seq_pad(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd,
                        int* err) {
    return k.mode == ROW_SEQ2 ? rows_impl::launch<512, ROW_SEQ2, true>(k, grid, st, pdl, a, fd, err)
                              : rows_impl::launch<512, ROW_SEQ, true>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
