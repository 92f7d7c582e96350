// gbsp_rows.cu -- the single-channel row kernels, Bluestein and direct (both
// block-size bounds), and the host launch functions; padded row buffers
// compile in gbsp_rows_pad.cu, batches in gbsp_rows_batch.cu, the
// multi-channel modes in gbsp_rows_multi.cu.
#include "gbsp_rows_single.cuh"

namespace gbsp {
int rows_capacity(const RowsKernel& k, int sms, int* cap) {
    *cap = 0;
    if (k.ntmax == 384) return rows_capacity_384(k, sms, cap);
    if (k.pad && k.K == 1) return rows_capacity_pad(k, sms, cap);
    if (k.mode == ROW_DIRECT)
        return k.ntmax == 512 ? rows_single::capacity<512, ROW_DIRECT, false>(k, sms, cap)
                              : rows_single::capacity<1024, ROW_DIRECT, false>(k, sms, cap);
    if (k.mode != ROW_SINGLE) return rows_capacity_multi(k, sms, cap);
    return k.ntmax == 512 ? rows_single::capacity<512, ROW_SINGLE, false>(k, sms, cap)
                          : rows_single::capacity<1024, ROW_SINGLE, false>(k, sms, cap);
}

int rows_launch(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err) {
    if (k.ntmax == 384) return rows_launch_384(k, grid, st, pdl, a, fd, err);
    if (k.pad && k.K == 1) return rows_launch_pad(k, grid, st, pdl, a, fd, err);
    if (k.mode == ROW_DIRECT)
        return k.ntmax == 512 ? rows_single::launch<512, ROW_DIRECT, false>(k, grid, st, pdl, a, fd, err)
                              : rows_single::launch<1024, ROW_DIRECT, false>(k, grid, st, pdl, a, fd, err);
    if (k.mode != ROW_SINGLE) return rows_launch_multi(k, grid, st, pdl, a, fd, err);
    return k.ntmax == 512 ? rows_single::launch<512, ROW_SINGLE, false>(k, grid, st, pdl, a, fd, err)
                          : rows_single::launch<1024, ROW_SINGLE, false>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
