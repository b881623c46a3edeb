// NVFP4 GEMM over any number of activation rows (batched verify, prompts): Y[t][n] = gs * sum_k X[t][k] * W[n][k]. The entry point and the
// pass that brings rows into f16; the product itself runs on CTA pairs (nvfp4_gemm_pair.cu).
//
// Arithmetic. A = w * s: an E2M1 code times a UE4M3 scale has at most 5 significant bits, so the product is exact in f16 and in bf16.
// B: bf16 rows as they are beyond 128 of them; else x * 2^k as f16 with one power of two per activation row (row amax brought to
// [2^13, 2^14) where f32 has that power of two, k <= 127): exact for bf16 input down to 2^-27 of the row maximum. Products are exact in the
// tensor core, accumulation is f32 in tensor memory, the epilogue multiplies by gs, then by 2^-k (which may be a subnormal f32: the two
// are not multiplied with one another first).
#include "common.cuh"
#include "nvfp4_gemm.cuh"

namespace {

constexpr int PREP_THREADS = 256, PREP_KEEP = 4;
// activation rows -> f16 * 2^k (k per row), and the rows' 2^-k. grid (M). What bounds it: one trip to memory and its launch; a thread's first
// PREP_KEEP chunks of eight values are asked for at once and kept between the two passes over the row (whole rows up to 8192 values).
// Small blocks, so that they fit beside the CTAs of the GEMM, which start at once and decode weights meanwhile.
template <int XT>
__global__ void __launch_bounds__(PREP_THREADS) gemm_prep_x_kernel(const void* __restrict__ x, uint16_t* __restrict__ xh, float* __restrict__ rs, int k) {
    __shared__ float amax_w[PREP_THREADS / 32];
    pdl_wait();  // the activations may come from the kernel before this one, and one before it may still read what this one overwrites
    // Only now: the GEMM reads weights and the tensor scale without waiting for this kernel, so whatever wrote them must be complete by the time
    // it starts.
    pdl_launch_dependents();
    const size_t row = blockIdx.x;
    const int n = k >> 3;
    constexpr int NV = XT == 1 ? 1 : 2;
    auto load = [&](int i, uint4 r[NV]) {
#pragma unroll
        for (int v = 0; v < NV; v++) r[v] = __ldcg((const uint4*)x + (row * n + i) * NV + v);
    };
    auto widen = [&](const uint4 r[NV], float v[8]) {
        const uint32_t a[4] = {r[0].x, r[0].y, r[0].z, r[0].w}, b[4] = {r[NV - 1].x, r[NV - 1].y, r[NV - 1].z, r[NV - 1].w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (XT == 1)
                v[2 * q] = __uint_as_float(a[q] << 16), v[2 * q + 1] = __uint_as_float(a[q] & 0xffff0000u);
            else
                v[q] = __uint_as_float(a[q]), v[4 + q] = __uint_as_float(b[q]);
        }
    };
    float amax = 0.0f;
    auto top = [&](const uint4 r[NV]) {
        float v[8];
        widen(r, v);
#pragma unroll
        for (int j = 0; j < 8; j++) amax = fmaxf(amax, fabsf(v[j]) < INFINITY ? fabsf(v[j]) : 0.0f);
    };
    uint4 kept[PREP_KEEP][NV];
#pragma unroll
    for (int q = 0; q < PREP_KEEP; q++)
        if ((int)threadIdx.x + q * PREP_THREADS < n) load((int)threadIdx.x + q * PREP_THREADS, kept[q]);
#pragma unroll
    for (int q = 0; q < PREP_KEEP; q++)
        if ((int)threadIdx.x + q * PREP_THREADS < n) top(kept[q]);
#pragma unroll 4
    for (int i = threadIdx.x + PREP_KEEP * PREP_THREADS; i < n; i += PREP_THREADS) {
        uint4 r[NV];
        load(i, r);
        top(r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) amax_w[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = 0.0f;
#pragma unroll
    for (int w = 0; w < PREP_THREADS / 32; w++) amax = fmaxf(amax, amax_w[w]);
    // The largest finite value * mul in [2^13, 2^14), two binades under the largest f16; rows below 2^-114 get the largest power of two there is,
    // 2^127, which leaves bf16 values of any size exact (2^-133 * 2^127 = 2^-6). Infinities and NaN stay what they are.
    const uint32_t e = max((__float_as_uint(amax) >> 23) & 0xFFu, 13u);
    const float mul = __uint_as_float((127u + 13u + 127u - e) << 23);
    const float inv = e == 13u ? 0x1p-127f : __uint_as_float((e - 13u) << 23);
    auto store = [&](int i, const uint4 r[NV]) {
        float v[8];
        widen(r, v);
        uint32_t h[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const __half2 p = __floats2half2_rn(v[2 * q] * mul, v[2 * q + 1] * mul);
            h[q] = *(const uint32_t*)&p;
        }
        ((uint4*)xh)[row * n + i] = make_uint4(h[0], h[1], h[2], h[3]);
    };
#pragma unroll
    for (int q = 0; q < PREP_KEEP; q++)
        if ((int)threadIdx.x + q * PREP_THREADS < n) store((int)threadIdx.x + q * PREP_THREADS, kept[q]);
#pragma unroll 4
    for (int i = threadIdx.x + PREP_KEEP * PREP_THREADS; i < n; i += PREP_THREADS) {
        uint4 r[NV];
        load(i, r);
        store(i, r);
    }
    if (threadIdx.x == 0) rs[row] = inv;
}

constexpr int MAX_KSPLITS = 8;
constexpr size_t PART_ROWS = 32768;  // output rows x parts of K that the workspace holds sums of (m <= 128: that many for each of 8 parts)
// Activation rows up to which K is split: what the sums of more would take from every caller's workspace. Few output rows do not fill the machine beyond
// it either: 1024 x 10240 takes 22.5 us at 512 rows and 41.0 at 513 (2048 x 9984: 32.6 at 512, 41.2 at 600).
constexpr int MAX_SPLIT_M = 512;
// f16 activations and row factors, which every call may need
size_t front_bytes(int k, int m) { return (size_t)m * k * 2 + (((size_t)m * 4 + 255) & ~(size_t)255) + 256; }
// the raw sums that cn_nvfp4_gemm_workspace_bytes makes room for, whatever the output rows
size_t sum_bytes(int m) { return m <= 128 ? (size_t)MAX_KSPLITS * m * PART_ROWS * 4 : (m <= MAX_SPLIT_M ? (size_t)m * PART_ROWS * 4 : 0); }
// More than 128 rows of bf16 go to the tensor cores as they are: their MMAs hide the decode to bf16, which takes twice the instructions
// of that to f16. Everything else goes as f16 x 2^k per row.
bool rows_as_f16(int dtype, int m) { return dtype != CN_BF16 || m <= 128; }
// Parts of K that `bytes` of raw sums allow. Never more than what sum_bytes gives: a larger workspace does not change the order of a sum.
int splits_allowed(int rows, int m, size_t bytes) {
    if (m > MAX_SPLIT_M || (size_t)rows > PART_ROWS) return 1;
    const size_t have = bytes < sum_bytes(m) ? bytes : sum_bytes(m), most = have / ((size_t)m * rows * 4);
    return most > (size_t)MAX_KSPLITS ? MAX_KSPLITS : (most < 1 ? 1 : (int)most);
}
int splits_of(int rows, int k, int m, int dtype, size_t bytes) { return cn_gemm_pair_splits(rows, k, m, rows_as_f16(dtype, m), splits_allowed(rows, m, bytes)); }

}  // namespace

int cn_gemm_prep_x(const void* x, int dtype, uint16_t* xh, float* rs, int k, int m, cudaStream_t stream) {
    if (dtype == CN_BF16)
        CN_CUDA(cn_launch_pdl(gemm_prep_x_kernel<1>, dim3((unsigned)m), dim3(PREP_THREADS), 0, stream, x, xh, rs, k));
    else
        CN_CUDA(cn_launch_pdl(gemm_prep_x_kernel<0>, dim3((unsigned)m), dim3(PREP_THREADS), 0, stream, x, xh, rs, k));
    return CN_OK;
}

extern "C" size_t cn_nvfp4_gemm_workspace_bytes(int k, int m) {
    if (k <= 0 || m <= 0) return 0;
    return front_bytes(k, m) + sum_bytes(m);
}

extern "C" size_t cn_nvfp4_gemm_workspace_bytes_of(int rows, int k, int m) {
    if (rows <= 0 || k <= 0 || k % 256 || m <= 0) return 0;
    const int a = splits_of(rows, k, m, CN_F32, sum_bytes(m)), b = splits_of(rows, k, m, CN_BF16, sum_bytes(m)), s = a > b ? a : b;
    return front_bytes(k, m) + (s > 1 ? (size_t)s * m * rows * 4 : 0);
}

extern "C" int cn_nvfp4_gemm_launches(int rows, int k, int m, int dtype) {
    if (rows <= 0 || k <= 0 || k % 256 || m <= 0) return 0;
    return (rows_as_f16(dtype, m) ? 1 : 0) + 1 + (splits_of(rows, k, m, dtype, sum_bytes(m)) > 1 ? 1 : 0);
}

extern "C" int cn_nvfp4_gemm(const void* w, const float* gs, const void* x, void* y, int rows, int k, int m, int ldy, int dtype, void* workspace,
                             size_t workspace_bytes, cn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (rows <= 0 || k <= 0 || k % 256 != 0) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemm: k = %d must be a positive multiple of 256", k);
    if (m < 1) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemm: m = %d", m);
    if (ldy < rows) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemm: ldy %d < rows %d", ldy, rows);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemm: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    if (((uintptr_t)w & 15) || ((uintptr_t)x & 15) || ((uintptr_t)workspace & 255))
        CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemm: weights and activations must be 16-byte aligned, the workspace 256-byte aligned");
    if (!workspace || workspace_bytes < front_bytes(k, m))
        CN_FAIL(CN_ERR_LIMIT, "cn_nvfp4_gemm: workspace of %zu B, %zu B needed", workspace_bytes, front_bytes(k, m));
    uint16_t* xh = (uint16_t*)workspace;
    float* rs = (float*)((char*)workspace + (((size_t)m * k * 2 + 255) & ~(size_t)255));
    GemmCall c = {};
    c.w = w, c.gs = gs, c.rs = rs, c.y = y, c.rows = rows, c.k = k, c.m = m, c.ldy = ldy, c.out_bf16 = dtype == CN_BF16;
    c.x_f16 = rows_as_f16(dtype, m);
    c.x = c.x_f16 ? (const void*)xh : x;
    c.max_splits = splits_allowed(rows, m, workspace_bytes - front_bytes(k, m));
    if (c.max_splits > 1) c.part = (float*)((char*)rs + (((size_t)m * 4 + 255) & ~(size_t)255));
    if (c.x_f16) {
        if (int rc = cn_gemm_prep_x(x, dtype, xh, rs, k, m, stream)) return rc;
    } else {
        // results may take the place of the activations: bf16 rows are then read from a copy (every row tile reads them again)
        const size_t xbytes = (size_t)m * k * 2, ybytes = ((size_t)(m - 1) * ldy + rows) * 2;
        if ((uintptr_t)x < (uintptr_t)y + ybytes && (uintptr_t)y < (uintptr_t)x + xbytes) {
            CN_CUDA(cudaMemcpyAsync(xh, x, xbytes, cudaMemcpyDeviceToDevice, stream));
            c.x = xh;
        }
    }
    return cn_gemm_pair_launch(c, stream);
}
