// The prefill matmul with weights through tensor memory (okf_gemm_ts.cu), called by the planner in okf_gemm_tc.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace okf {

struct GemmTs {
    int ty, xdt, odt, sms;  // xdt: fp16 or bf16
    const uint8_t *w;
    const void *x;
    void *out;
    int *status;
    float *partial;
    uint32_t k, m, n, row_bytes;
    uint32_t tok;                        // tokens of an item, a multiple of 16, at most 256
    uint32_t waves, dealt, dealers, nt;  // how items are laid over the SMs
    uint32_t cluster, chains;            // CTAs that share an item along K (0, 1: none), accumulators each (1, 2, 4)
    uint32_t nout, out_ld, out_row0;     // row shards: fp32 into `nout` whole outputs
    void *outs[8];
    uint32_t *epoch;
    uint32_t epoch_inc;
};
cudaError_t launch_gemm_ts(const GemmTs &g, cudaStream_t s, int dev);
// How many clusters of 2 .. 8 of its CTAs the device has room for at once (index: size); null where that is not known.
const uint32_t *gemm_ts_clusters(int dev);

}  // namespace okf
