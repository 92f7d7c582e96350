// gbsp_rows_pad.cu -- the single-channel row kernels with a padded row buffer
// (plans whose last radix is a power of two).
#include "gbsp_rows_single.cuh"

namespace gbsp {

int rows_capacity_pad(const RowsKernel& k, int sms, int* cap) {
    using namespace rows_single;
    if (k.mode == ROW_DIRECT)
        return k.ntmax == 512 ? capacity<512, ROW_DIRECT, true>(k, sms, cap) : capacity<1024, ROW_DIRECT, true>(k, sms, cap);
    return k.ntmax == 512 ? capacity<512, ROW_SINGLE, true>(k, sms, cap) : capacity<1024, ROW_SINGLE, true>(k, sms, cap);
}

int rows_launch_pad(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err) {
    using namespace rows_single;
    if (k.mode == ROW_DIRECT)
        return k.ntmax == 512 ? launch<512, ROW_DIRECT, true>(k, grid, st, pdl, a, fd, err)
                              : launch<1024, ROW_DIRECT, true>(k, grid, st, pdl, a, fd, err);
    return k.ntmax == 512 ? launch<512, ROW_SINGLE, true>(k, grid, st, pdl, a, fd, err)
                          : launch<1024, ROW_SINGLE, true>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
