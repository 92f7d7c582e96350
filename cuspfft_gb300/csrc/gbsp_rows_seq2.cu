// gbsp_rows_seq2.cu -- two sequential channels that hold the whole row.
#include "gbsp_rows_impl.cuh"

namespace gbsp {

int rows_capacity_seq2(const RowsKernel& k, int sms, int* cap) {
    return rows_impl::capacity<512, ROW_SEQ2>(k, sms, cap);
}

int rows_launch_seq2(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err) {
    return rows_impl::launch<512, ROW_SEQ2>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
