// MoE routing on the device: softmax top-k (Flash-Next) and sigmoid top-k (GLM), bit-exact
// indices against the host twins.
//
// Supersedes router_top10 (engine/src/kernels.rs:3109-3171; the residency bookkeeping of that
// kernel - cold mask, hit counters, pointer gather - is not part of this path: the MoE operator
// reads its pointer tables directly) and glm5_router_sig_topk (engine/src/kernels_glm5_moe.cu:44-96,
// host twin glm5_moe::route_from_logits, engine/src/glm5_moe.rs:196-236).
//
// One CTA per token row, one thread per expert slot (P = next power of two >= E, <= 1024).
// The softmax sum is the pairwise tree of the reference kernel (stride P/2, P/4, ..), so it rounds
// exactly as there; the maximum does not depend on the order and is taken with warp shuffles. exp() is
// taken in f64 and rounded once, which gives the correctly rounded f32 value the host twins' libm
// returns; selection is K rounds of "best value, lowest index on ties", as in both reference routers,
// by one warp with the keys in registers.
#include "common.cuh"

namespace {

__device__ __forceinline__ float exp_rn(float x) { return (float)exp((double)x); }

// max over the block's values (NaN operands are ignored, as fmaxf does in the reference's tree; the value does
// not depend on the order). buf: 32 floats; one barrier, the next use of `buf` must be a barrier later.
__device__ __forceinline__ float block_max(float v, float* buf, int e, int P) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((e & 31) == 0) buf[e >> 5] = v;
    __syncthreads();
    float r = (e & 31) < (P >> 5) ? buf[e & 31] : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    return r;
}
// K rounds of "best value, lowest index on ties" by one warp: lane l holds the keys of experts l, l + 32, .. in registers, and a round is a
// maximum and a minimum over the warp (redux) without a barrier; it was two barriers of the whole block. key: unsigned, in the order of the
// values; 0 = taken or never selectable. A round without a key left (a row of NaN) picks expert 0.
template <int NK>
__device__ __forceinline__ void select_rounds(const uint32_t* keys, const float* vals, float* s_w, int32_t* ids, int E, int K, int lane) {
    uint32_t key[NK];
#pragma unroll
    for (int i = 0; i < NK; i++) key[i] = keys[lane + 32 * i];
    for (int j = 0; j < K; j++) {
        uint32_t top = key[0];
#pragma unroll
        for (int i = 1; i < NK; i++) top = max(top, key[i]);
        top = __reduce_max_sync(0xffffffffu, top);
        int at = E;
#pragma unroll
        for (int i = NK - 1; i >= 0; i--)
            if (key[i] == top) at = lane + 32 * i;
        const int pick = top ? (int)__reduce_min_sync(0xffffffffu, (uint32_t)at) : 0;
#pragma unroll
        for (int i = 0; i < NK; i++)
            if (lane + 32 * i == pick) key[i] = 0u;
        if (lane == 0) s_w[j] = vals[pick], ids[j] = pick;
    }
    __syncwarp();
}
__device__ __forceinline__ void select_topk(const uint32_t* keys, const float* vals, float* s_w, int32_t* ids, int P, int E, int K, int lane) {
    switch (P >> 5) {
        case 1: return select_rounds<1>(keys, vals, s_w, ids, E, K, lane);
        case 2: return select_rounds<2>(keys, vals, s_w, ids, E, K, lane);
        case 4: return select_rounds<4>(keys, vals, s_w, ids, E, K, lane);
        case 8: return select_rounds<8>(keys, vals, s_w, ids, E, K, lane);
        case 16: return select_rounds<16>(keys, vals, s_w, ids, E, K, lane);
        default: return select_rounds<32>(keys, vals, s_w, ids, E, K, lane);
    }
}

// red[0..P) summed by the reference's stride-halving tree (red[e] += red[e + st], st = P/2, P/4, ..): strides of 32
// and more through shared memory, the last five inside warp 0 with the same pairs; every thread gets the sum
__device__ __forceinline__ float tree_sum(float* red, float* out, int e, int P) {
    for (int st = P >> 1; st >= 32; st >>= 1) {
        __syncthreads();
        if (e < st) red[e] = red[e] + red[e + st];
    }
    __syncthreads();
    if (e < 32) {
        float v = red[e];
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const float o = __shfl_down_sync(0xffffffffu, v, st);
            if (e < st) v = v + o;
        }
        if (e == 0) *out = v;
    }
    __syncthreads();
    return *out;
}

__global__ void route_softmax_kernel(const float* __restrict__ logits, int32_t* __restrict__ ids, float* __restrict__ wts, int E, int K) {
    extern __shared__ float sm[];
    float* red = sm;                        // [P]
    float* s_w = sm + blockDim.x;           // [K]
    uint32_t* keys = (uint32_t*)(s_w + K);  // [P]
    __shared__ float bmax[32];
    __shared__ float s_den;
    // In this order: kernels behind this one read what is older than it (tensor scales) before they wait. The launch itself goes on under the kernel in front: a MUL1 step of
    // one token 44.2 -> 42.0 us, 64 tokens of the NVFP4 step 198 -> 193.
    pdl_wait();
    pdl_launch_dependents();
    const int P = blockDim.x, e = threadIdx.x, t = blockIdx.x;
    const bool in = e < E;
    const float l = in ? logits[(size_t)t * E + e] : -INFINITY;
    // missing leaves of a non-power-of-two E are absent from the trees: -inf for max, 0 for sum
    const float mx = block_max(l, bmax, e, P);
    const float ex = in ? exp_rn(l - mx) : 0.0f;
    red[e] = ex;
    const float den = tree_sum(red, &s_den, e, P);
    const float p = ex / den;  // >= 0, or NaN in a whole row
    red[e] = p;
    keys[e] = in && p == p ? __float_as_uint(p) + 1u : 0u;
    __syncthreads();
    if (e >= 32) return;
    select_topk(keys, red, s_w, ids + (size_t)t * K, P, E, K, e);
    float sum = 0.0f;  // in pick order
    for (int j = 0; j < K; j++) sum += s_w[j];
    for (int j = e; j < K; j += 32) wts[(size_t)t * K + j] = s_w[j] / sum;
}

__global__ void route_sigmoid_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int32_t* __restrict__ ids,
                                     float* __restrict__ wts, int E, int K, float scale) {
    extern __shared__ float sm[];
    float* vals = sm;
    float* s_w = sm + blockDim.x;
    uint32_t* keys = (uint32_t*)(s_w + K);
    pdl_wait();  // (as above)
    pdl_launch_dependents();
    const int P = blockDim.x, e = threadIdx.x, t = blockIdx.x;
    float s = 0.0f;
    uint32_t key = 0u;
    if (e < E) {
        s = 1.0f / (1.0f + exp_rn(-logits[(size_t)t * E + e]));
        const float v = s + (bias ? bias[e] : 0.0f);
        const float c = (v != v) ? -INFINITY : v + 0.0f;  // NaN never wins; one zero
        const uint32_t b = __float_as_uint(c);
        key = (b & 0x80000000u) ? ~b : b | 0x80000000u;  // ordered; above 0 for every c
    }
    vals[e] = s;
    keys[e] = key;
    __syncthreads();
    if (e >= 32) return;
    select_topk(keys, vals, s_w, ids + (size_t)t * K, P, E, K, e);
    float sum = 0.0f;
    for (int j = 0; j < K; j++) sum += s_w[j];
    const float den = sum + 1e-20f;
    for (int j = e; j < K; j += 32) wts[(size_t)t * K + j] = (s_w[j] / den) * scale;
}

int pow2_at_least(int n) {
    int p = 32;
    while (p < n) p <<= 1;
    return p;
}

int check(int tokens, int experts, int k, const char* who) {
    if (tokens < 1 || experts < 1 || experts > 1024 || k < 1 || k > experts || k > 64)
        CN_FAIL(CN_ERR_SHAPE, "%s: %d experts top-%d: the router takes 1 <= K <= 64, K <= E <= 1024", who, experts, k);
    return CN_OK;
}

}  // namespace

extern "C" int cn_route_softmax_topk(const float* logits, int32_t* ids, float* wts, int tokens, int experts, int k, cn_stream_t stream) {
    if (int rc = check(tokens, experts, k, "cn_route_softmax_topk")) return rc;
    const int P = pow2_at_least(experts);
    CN_CUDA(cn_launch_pdl(route_softmax_kernel, dim3(tokens), dim3(P), (2 * P + k) * sizeof(float), (cudaStream_t)stream, logits, ids, wts, experts, k));
    return CN_OK;
}

extern "C" int cn_route_sigmoid_topk(const float* logits, const float* bias, int32_t* ids, float* wts, int tokens, int experts, int k,
                                     float scale, cn_stream_t stream) {
    if (int rc = check(tokens, experts, k, "cn_route_sigmoid_topk")) return rc;
    const int P = pow2_at_least(experts);
    CN_CUDA(cn_launch_pdl(route_sigmoid_kernel, dim3(tokens), dim3(P), (2 * P + k) * sizeof(float), (cudaStream_t)stream, logits, bias, ids, wts, experts, k, scale));
    return CN_OK;
}
