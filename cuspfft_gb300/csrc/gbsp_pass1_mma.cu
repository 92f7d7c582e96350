// gbsp_pass1_mma.cu -- tensor-core pass 1: host launch functions
// (gbsp_launch.h), single matrix and batch.
#include "gbsp_launch.h"

namespace gbsp {

int p1_mma_prepare(size_t smem, bool batch) {
    const void* kern = batch ? (const void*)k_twiddle_mma<true> : (const void*)k_twiddle_mma<false>;
    if (int rc = allow_full_smem(kern)) return rc;
    int nb = 0;
    GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, MM_THREADS, smem));
    if (nb < 1) return set_error(GBSP_ERR_UNSUPPORTED, "pass-1 kernel does not fit on an SM");
    return GBSP_OK;
}

int p1_mma_launch(int sms, size_t smem, cudaStream_t st, bool pdl, const P1MmaArgs& a) {
    const int grid = (int)std::min<long>(sms, p1_mma_items(a));
    GB_CUDA(launch_kernel(k_twiddle_mma<false>, grid, MM_THREADS, smem, st, pdl, 1, a, nullptr, nullptr, 1, a.queue));
    return GBSP_OK;
}

int p1_mma_batch_launch(int grid, size_t smem, cudaStream_t st, const P1MmaArgs* args, const long* item_begin,
                        int nmat, unsigned int* queue) {
    k_twiddle_mma<true><<<grid, MM_THREADS, smem, st>>>(P1MmaArgs{}, args, item_begin, nmat, queue);
    GB_CUDA(cudaGetLastError());
    return GBSP_OK;
}

}  // namespace gbsp
