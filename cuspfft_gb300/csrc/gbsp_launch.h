// gbsp_launch.h -- host entry points of the kernel translation units.
//
// The kernels compile in separate translation units so the build runs them
// in parallel: pass 1 (gbsp_pass1*.cu), single-channel rows (gbsp_rows.cu,
// _384, _pad), batches of them (gbsp_rows_batch*.cu), multi-channel rows
// (gbsp_rows_multi.cu, gbsp_rows_seq*.cu).  The plan code (gbsp_plan.cu) reaches
// them through these functions.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <utility>

#include "gbspfft.h"
#include "gbsp_internal.h"
#include "gbsp_kernels.cuh"
#include "gbsp_pass1_mma.cuh"
#include "gbsp_planner.h"

// Returns a GBSP_ERR_* status (with the message recorded) from the calling
// function when a CUDA runtime call fails.
#define GB_CUDA(call)                                                                         \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return gbsp::set_error(e_ == cudaErrorMemoryAllocation ? GBSP_ERR_ALLOC : GBSP_ERR_CUDA, \
                                   std::string(#call) + ": " + cudaGetErrorString(e_));      \
    } while (0)

namespace gbsp {

// One kernel launch; pdl: it may start before the kernel ahead of it in the
// stream is complete (see pdl_wait in gbsp_kernels.cuh); cluster > 1: blocks
// per thread-block cluster.
template <typename... P, typename... A>
cudaError_t launch_kernel(void (*kern)(P...), int grid, int block, size_t smem, cudaStream_t st, bool pdl, int cluster,
                          A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    if (pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)cluster;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Per-device limits, queried once per device.
struct DeviceLimits {
    size_t smem_optin = 0;
    int sms = 0;
};
int device_limits(int dev, DeviceLimits* out);

// Lets `kern` take all the opt-in shared memory of a CTA on the current
// device.  The limit is a property of the kernel, shared by every plan in the
// process; one fixed value keeps a later, smaller plan from invalidating an
// earlier one.  Done once per (kernel, device).
int allow_full_smem(const void* kern);

// ---- pass 1 (gbsp_pass1.cu, gbsp_pass1_exact.cu): one compiled kernel per
// (index bytes, table layout, 64-bit phases, rows per lane, phase mode)
struct P1Kernel {
    int idx_bytes, tab;
    bool big;
    int ku;
    bool exact;  // every twiddle an exact table lookup (no recurrence)
};
// CTAs of k_twiddle_sum resident per SM with `smem` bytes (raises the limit)
int p1_blocks_per_sm(const P1Kernel& k, size_t smem, int* nb);
int p1_launch(const P1Kernel& k, int grid, size_t smem, cudaStream_t st, bool pdl, const P1Args& a);
int p1_batch_blocks_per_sm(const P1Kernel& k, size_t smem, int* nb);
int p1_batch_launch(const P1Kernel& k, int grid, size_t smem, cudaStream_t st, const P1Args* args,
                    const long* item_begin, int nmat, unsigned long long* queue);

// ---- pass 1 on the tensor cores (gbsp_pass1_mma.cu), one CTA per SM
int p1_mma_prepare(size_t smem, bool batch);  // raises the limit, checks that it fits
int p1_mma_launch(int sms, size_t smem, cudaStream_t st, bool pdl, const P1MmaArgs& a);
int p1_mma_batch_launch(int grid, size_t smem, cudaStream_t st, const P1MmaArgs* args, const long* item_begin,
                        int nmat, unsigned int* queue);

// ---- Bluestein rows: mode ROW_*, compiled block bound ntmax (512 or 1024;
// 384 for ROW_SINGLE without padding)
struct RowsKernel {
    int mode, ntmax, K, nt;
    size_t smem;
    bool pad;  // padded row buffer
};
// CTAs (single channel, sequential channels) or clusters resident at once
int rows_capacity(const RowsKernel& k, int sms, int* cap);
int rows_launch(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err);
// ... ROW_SINGLE at 168 registers a thread (gbsp_rows_384.cu)
int rows_capacity_384(const RowsKernel& k, int sms, int* cap);
int rows_launch_384(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd,
                    int* err);
// ... with a padded row buffer (gbsp_rows_pad.cu)
int rows_capacity_pad(const RowsKernel& k, int sms, int* cap);
int rows_launch_pad(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err);
// batches (gbsp_rows_batch.cu, gbsp_rows_batch_pad.cu)
int rows_batch_blocks_per_sm(const RowBlock& rb, bool pad, size_t smem, int* nb);
int rows_batch_blocks_per_sm_pad(const RowBlock& rb, size_t smem, int* nb);
int rows_batch_launch_pad(const RowBlock& rb, int grid, size_t smem, cudaStream_t st, const RowsBatch* descs,
                          const long* row_begin, int nmat, unsigned long long* queue, bool pdl, int* err);
int rows_batch_launch(const RowBlock& rb, bool pad, int grid, size_t smem, cudaStream_t st, const RowsBatch* descs,
                      const long* row_begin, int nmat, unsigned long long* queue, bool pdl, int* err);
// the multi-channel modes (clusters: gbsp_rows_multi.cu, sequential
// channels: gbsp_rows_seq.cu); rows_capacity / rows_launch forward to these
int rows_capacity_multi(const RowsKernel& k, int sms, int* cap);
int rows_launch_multi(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd,
                      int* err);
int rows_capacity_seq2(const RowsKernel& k, int sms, int* cap);
int rows_launch_seq2(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err);
int rows_capacity_seq_pad(const RowsKernel& k, int sms, int* cap);
int rows_launch_seq_pad(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd,
                        int* err);
int rows_capacity_seq(const RowsKernel& k, int sms, int* cap);
int rows_launch_seq(const RowsKernel& k, int grid, cudaStream_t st, bool pdl, const RowsArgs& a, const FFTDesc& fd, int* err);

}  // namespace gbsp
