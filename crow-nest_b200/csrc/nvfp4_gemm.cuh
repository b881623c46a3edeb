// Launch descriptor of the batched NVFP4 GEMM kernels on the container layout.
#pragma once
#include <cuda_runtime.h>

struct GemmCall {
    const void* w;
    const float* gs;
    const void* x;    // bf16 rows (bf16 results), or f16 x 2^k rows (x_f16, f32 results)
    const float* rs;  // per row 2^-k (x_f16)
    void* y;
    int rows, k, m, ldy;
    int x_f16;
};
// more than 128 rows: CTA pairs (nvfp4_gemm_pair.cu)
int cn_gemm_pair_launch(const GemmCall& c, cudaStream_t stream);
