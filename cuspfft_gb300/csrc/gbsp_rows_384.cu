// gbsp_rows_384.cu -- the single-channel Bluestein row kernel for blocks of up
// to 384 threads (168 registers a thread).
#include "gbsp_rows_single.cuh"

namespace gbsp {

int rows_capacity_384(const RowsKernel& k, int sms, int* cap) {
    return rows_single::capacity<384, ROW_SINGLE, false>(k, sms, cap);
}

int rows_launch_384(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd,
                    int* err) {
    return rows_single::launch<384, ROW_SINGLE, false>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
