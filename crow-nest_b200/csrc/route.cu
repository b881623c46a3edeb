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
// returns; selection is "best value, lowest index on ties" K times, as in both reference routers: by rank among the few
// keys that can be picked, or by one warp in K rounds with the keys in registers.
#include "common.cuh"

#include <type_traits>

namespace {

__device__ __forceinline__ float exp_rn(float x) { return (float)exp((double)x); }

// max over the block's values (NaN operands are ignored, as fmaxf does in the reference's tree; the value does
// not depend on the order). buf: 32 floats; one barrier, the next use of `buf` must be a barrier later.
template <int NK>
__device__ __forceinline__ float block_max(float v, float* buf, int e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((e & 31) == 0) buf[e >> 5] = v;
    __syncthreads();
    float r = (e & 31) < NK ? buf[e & 31] : -INFINITY;
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

// What the warps leave each other while the best K are found.
struct Found {
    uint32_t best[32];  // a warp's largest key, 0 for warps that are not there
    uint32_t key[32];
    int at[32], n;
};
// The same picks with two barriers and no rounds, by all threads of the block, where there are as many warps as picks: the K-th largest of the warps' largest keys is a bound that K keys
// reach, and not many more do (15 of 512 for ten picks, as many as it takes to come from ten warps); these find their ranks at once, a lane each. Rows with more than 32 such keys (ties) or
// with fewer selectable warps than picks take the rounds. vals and keys are those of all threads. 512 experts, ten picks: 3.97 -> 2.9 us a launch in a stream of them; the rounds are 250 cycles each.
template <int NK>
__device__ __forceinline__ void select_block(uint32_t key, const uint32_t* keys, const float* vals, float* s_w, int32_t* ids, int E, int K, int e) {
    __shared__ Found f;
    const int lane = e & 31;
    uint32_t least = 0u;
    if (NK >= 8 && NK >= K) {  // (NK warps; fewer than eight have rounds short enough)
        const uint32_t best = __reduce_max_sync(0xffffffffu, key);
        if (lane == 0) f.best[e >> 5] = best;
        if (e == 0) f.n = 0;
        __syncthreads();
        const uint32_t mine = lane < NK ? f.best[lane] : 0u;
        int rank = 0;  // among the warps, the first on ties
#pragma unroll 8
        for (int j = 0; j < NK; j++) {
            const uint32_t o = f.best[j];
            rank += o > mine || (o == mine && j < lane);
        }
        least = __reduce_max_sync(0xffffffffu, lane < NK && rank == K - 1 ? mine : 0u);
        const bool take = least != 0u && key >= least;
        const uint32_t some = __ballot_sync(0xffffffffu, take);
        if (some) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&f.n, __popc(some));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(some & ((1u << lane) - 1u));
            if (take && at < 32) f.key[at] = key, f.at[at] = e;
        }
    }
    __syncthreads();
    if (e >= 32) return;
    if (NK < 8 || least == 0u || f.n > 32) {
        select_rounds<NK>(keys, vals, s_w, ids, E, K, lane);
        return;
    }
    const int n = f.n;
    const uint32_t mine = lane < n ? f.key[lane] : 0u;
    const int at = lane < n ? f.at[lane] : 0;
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; j++) {
        const uint32_t o = f.key[j];
        rank += o > mine || (o == mine && f.at[j] < at);
    }
    if (lane < n && rank < K) s_w[rank] = vals[at], ids[rank] = at;
    __syncwarp();
}

// red[0..P) summed by the reference's stride-halving tree (red[e] += red[e + st], st = P/2, P/4, ..): warp 0 takes the strides of 32 and more from shared memory, a lane its column of
// them, and the last five inside the warp, the same pairs at every step; every thread gets the sum
template <int NK>
__device__ __forceinline__ float tree_column(const float* red, int lane) {
    float v[NK];
#pragma unroll
    for (int i = 0; i < NK; i++) v[i] = red[lane + 32 * i];
#pragma unroll
    for (int st = NK / 2; st > 0; st >>= 1)
#pragma unroll
        for (int i = 0; i < st; i++) v[i] = v[i] + v[i + st];
    return v[0];
}
template <int NK>
__device__ __forceinline__ float tree_sum(const float* red, float* out, int e) {
    __syncthreads();
    if (e < 32) {
        float v = tree_column<NK>(red, e);
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

// NK: warps, a thread for every expert
template <int NK>
__global__ void __launch_bounds__(32 * NK) route_softmax_kernel(const float* __restrict__ logits, int32_t* __restrict__ ids, float* __restrict__ wts, int E, int K) {
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
    const int e = threadIdx.x, t = blockIdx.x;
    const bool in = e < E;
    const float l = in ? logits[(size_t)t * E + e] : -INFINITY;
    // missing leaves of a non-power-of-two E are absent from the trees: -inf for max, 0 for sum
    const float mx = block_max<NK>(l, bmax, e);
    const float ex = in ? exp_rn(l - mx) : 0.0f;
    red[e] = ex;
    const float den = tree_sum<NK>(red, &s_den, e);
    const float p = ex / den;  // >= 0, or NaN in a whole row
    red[e] = p;
    const uint32_t key = in && p == p ? __float_as_uint(p) + 1u : 0u;
    keys[e] = key;
    select_block<NK>(key, keys, red, s_w, ids + (size_t)t * K, E, K, e);
    if (e >= 32) return;
    float sum = 0.0f;  // in pick order
    for (int j = 0; j < K; j++) sum += s_w[j];
    for (int j = e; j < K; j += 32) wts[(size_t)t * K + j] = s_w[j] / sum;
}

template <int NK>
__global__ void __launch_bounds__(32 * NK) route_sigmoid_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int32_t* __restrict__ ids,
                                     float* __restrict__ wts, int E, int K, float scale) {
    extern __shared__ float sm[];
    float* vals = sm;
    float* s_w = sm + blockDim.x;
    uint32_t* keys = (uint32_t*)(s_w + K);
    pdl_wait();  // (as above)
    pdl_launch_dependents();
    const int e = threadIdx.x, t = blockIdx.x;
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
    select_block<NK>(key, keys, vals, s_w, ids + (size_t)t * K, E, K, e);
    if (e >= 32) return;
    float sum = 0.0f;
    for (int j = 0; j < K; j++) sum += s_w[j];
    const float den = sum + 1e-20f;
    for (int j = e; j < K; j += 32) wts[(size_t)t * K + j] = (s_w[j] / den) * scale;
}

// f(the kernels' number of warps: a power of two)
template <typename F>
int with_warps(int experts, F f) {
    if (experts <= 32) return f(std::integral_constant<int, 1>());
    if (experts <= 64) return f(std::integral_constant<int, 2>());
    if (experts <= 128) return f(std::integral_constant<int, 4>());
    if (experts <= 256) return f(std::integral_constant<int, 8>());
    if (experts <= 512) return f(std::integral_constant<int, 16>());
    return f(std::integral_constant<int, 32>());
}

int check(int tokens, int experts, int k, const char* who) {
    if (tokens < 1 || experts < 1 || experts > 1024 || k < 1 || k > experts || k > 64)
        CN_FAIL(CN_ERR_SHAPE, "%s: %d experts top-%d: the router takes 1 <= K <= 64, K <= E <= 1024", who, experts, k);
    return CN_OK;
}

}  // namespace

extern "C" int cn_route_softmax_topk(const float* logits, int32_t* ids, float* wts, int tokens, int experts, int k, cn_stream_t stream) {
    if (int rc = check(tokens, experts, k, "cn_route_softmax_topk")) return rc;
    return with_warps(experts, [&](auto warps) -> int {
        constexpr int NK = decltype(warps)::value;
        CN_CUDA(cn_launch_pdl(route_softmax_kernel<NK>, dim3(tokens), dim3(32 * NK), (64 * NK + k) * sizeof(float), (cudaStream_t)stream, logits, ids, wts, experts, k));
        return CN_OK;
    });
}

extern "C" int cn_route_sigmoid_topk(const float* logits, const float* bias, int32_t* ids, float* wts, int tokens, int experts, int k,
                                     float scale, cn_stream_t stream) {
    if (int rc = check(tokens, experts, k, "cn_route_sigmoid_topk")) return rc;
    return with_warps(experts, [&](auto warps) -> int {
        constexpr int NK = decltype(warps)::value;
        CN_CUDA(cn_launch_pdl(route_sigmoid_kernel<NK>, dim3(tokens), dim3(32 * NK), (64 * NK + k) * sizeof(float), (cudaStream_t)stream, logits, bias, ids, wts, experts, k, scale));
        return CN_OK;
    });
}
