// Down projections and combine of a small routed-expert step in one launch (moe_step.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct MoeDownCall {
    // Combo (token, pick j) reads row token * topk + j of h (f32) and the matrix of expert ids[token * topk + j]. ids, wts and the table are
    // older than the kernel before this one in the stream, which waits for its own predecessor before it lets this one start.
    const int32_t* ids;
    const float* wts;
    const unsigned long long* table;
    int experts, topk;
    const float* h;
    const float* gs;
    int inter;
    const void* shared;  // the shared expert's down matrix, or null
    const float* hs;     // its activations [tokens][shared_inter]
    const float* shared_gs;
    const float* sgate;
    int shared_inter;
    void* y;  // [tokens][hidden]
    int tokens, hidden, out_bf16;
};
bool cn_moe_down_combine_fits(const MoeDownCall& c);
// 16 result rows of a token x eight 64-value blocks of one of its experts, over the whole call
long long cn_moe_down_combine_units(const MoeDownCall& c);
int cn_moe_down_combine_launch(const MoeDownCall& c, cudaStream_t stream);
