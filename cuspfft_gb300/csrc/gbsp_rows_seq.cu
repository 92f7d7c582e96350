// gbsp_rows_seq.cu -- the Bluestein row kernel for convolutions split into
// K channels that one CTA runs in turn (512-thread bound; a separate instance
// above MAX_CHANNELS channels), and the dispatch to the two-channel and the
// padded ones (gbsp_rows_seq2.cu, gbsp_rows_seq_pad.cu).
#include "gbsp_rows_impl.cuh"

namespace gbsp {

int rows_capacity_seq(const RowsKernel& k, int sms, int* cap) {
    if (k.pad) return rows_capacity_seq_pad(k, sms, cap);
    if (k.mode == ROW_SEQ2) return rows_capacity_seq2(k, sms, cap);
    return k.mode == ROW_SEQW ? rows_impl::capacity<512, ROW_SEQW>(k, sms, cap)
                              : rows_impl::capacity<512, ROW_SEQ>(k, sms, cap);
}

int rows_launch_seq(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err) {
    if (k.pad) return rows_launch_seq_pad(k, grid, st, pdl, a, fd, err);
    if (k.mode == ROW_SEQ2) return rows_launch_seq2(k, grid, st, pdl, a, fd, err);
    return k.mode == ROW_SEQW ? rows_impl::launch<512, ROW_SEQW>(k, grid, st, pdl, a, fd, err)
                              : rows_impl::launch<512, ROW_SEQ>(k, grid, st, pdl, a, fd, err);
}

}  // namespace gbsp
