// FP8 (per-channel) and NVFP4 linears of more than 128 rows on CTA pairs (gemm_pair.cu): which calls, launch functions.
#pragma once
#include "common.cuh"

namespace eq {

// Both are launched as programmatic dependents and fetch the weight, and NVFP4's weight scales, before the grid ahead has ended: what
// writes the activations' codes and scales is the launch right before them in the stream, and no launch still under way writes the weight.
// qx [M][K] e4m3 codes, sx [M]; w [N][K], sw [N].  K % 128 == 0, N % 16 == 0, y 16-byte aligned.
int fp8_pair_launch(const uint8_t* qx, const float* sx, const uint8_t* w, const float* sw, void* y, int64_t M, int64_t N, int64_t K, int act_dtype,
                    int* status, cudaStream_t stream);
// codes [M][K/2], sfa: its scale atoms [ceil(M/128)][K/64][512 B]; w [N][K/2], sfw likewise; gx, gw: the global scales.
// K % 256 == 0, N % 8 == 0, y 16-byte aligned.
int nvfp4_pair_launch(const uint8_t* codes, const uint8_t* sfa, const float* gx, const uint8_t* w, const uint8_t* sfw, const float* gw, void* y, int64_t M,
                      int64_t N, int64_t K, int act_dtype, int* status, cudaStream_t stream);

}  // namespace eq
