// Launch descriptor of the batched NVFP4 GEMM on CTA pairs (nvfp4_gemm_pair.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct GemmCall {
    const void* w;       // container bytes
    const void* packed;  // or the re-laid form (cn_nvfp4_bs_repack)
    const float* gs;
    const void* x;    // bf16 rows, or f16 x 2^k rows (x_f16) that the kernel before this one in the stream wrote
    const float* rs;  // per row 2^-k (x_f16)
    void* y;
    int rows, k, m, ldy;
    int x_f16, out_bf16;
    float* part;     // room for the raw sums of max_splits parts of K, [max_splits][m][rows] (null: K is not split)
    int max_splits;  // m <= 65535 where above one
};
int cn_gemm_pair_launch(const GemmCall& c, cudaStream_t stream);
// the parts of K that the launch would take
int cn_gemm_pair_splits(int rows, int k, int m, bool x_f16, int max_splits);
// x -> f16 x 2^k rows [m][k] and rs[m] = 2^-k (nvfp4_gemm.cu); every later kernel of the stream may start early on what does not depend on it
int cn_gemm_prep_x(const void* x, int dtype, uint16_t* xh, float* rs, int k, int m, cudaStream_t stream);
