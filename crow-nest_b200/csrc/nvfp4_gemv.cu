// NVFP4 GEMV for M = 1..8 f32 activation rows of smaller matrices and for the f32 rows of single routed experts (bf16 rows: nvfp4_gemv_m1.cu; larger matrices of either type:
// nvfp4_gemv_tc.cu; the rules are in cn_gemv_launch and cn_gemv_m1_launch), plain or with the fused gate/up activation.
//
// Supersedes gemv_nvfp4_w / _gu / _wm / _gum (engine/src/kernels_p2.rs:355-530) and the record
// kernels gemv_fp4(_b) (engine/src/kernels.rs:118-189), glm5_gemv_fp4 (engine/src/kernels_glm5_moe.cu:284).
//
// Shape of the kernel (HBM-bound; the container layout is consumed as it lies, no repack):
//   - a CTA owns ROWS output rows over the whole K. A producer warp streams the rows' bytes
//     through a ring of shared-memory stages with 1-D bulk copies (TMA, completion counted on an
//     mbarrier), one piece of TX 36-byte blocks per row and stage; it never waits for anything
//     but a free stage, so the weight stream runs ahead of the arithmetic;
//   - the activation rows are staged once per CTA, as they are;
//   - consumer warps: lane (ry, tx) owns k-block tx of the stage for RT rows; the nine words of a
//     block are read with conflict-free 4-byte loads (36-byte stride), codes are decoded in
//     registers (cvt.rn.f16x2.e2m1x2: every E2M1 value is exact in f16) and multiplied in f32, each 16-value sub-block's partial sum is multiplied by its UE4M3 scale * tensor
//     scale (a 256-entry table, the reference's scale_lut) and accumulated in f32; the K split
//     over the TX lanes is reduced with xor shuffles in a fixed order.
// Each (row, m) pair runs the same instruction sequence whatever M is, so row m of an M-row call
// is bit-identical to a one-row call (the batch invariance of engine/src/kernels_p2.rs:391-396).
#include <cstdarg>
#include <cstdio>

#include "common.cuh"
#include "nvfp4_gemv.cuh"

namespace {

constexpr int NW = 4;  // consumer warps
constexpr int NTHREADS = (NW + 1) * 32;
constexpr int MAX_STAGES = 8;
constexpr int XB = 272;  // bytes of one k-block's 64 activations, padded: conflict-free 16-byte loads
constexpr int HDR_BYTES = 256 + 2048;  // barriers, two scale tables

// MP: activation rows compiled in (1, 2, 4, 8). RT: rows per consumer thread.
template <int MP, int RT>
__global__ void __launch_bounds__(NTHREADS, (MP <= 2 ? 4 : 1)) nvfp4_gemv_kernel(const GemvParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int TX = p.tx;
    const int G = NW * (32 / TX);  // row groups per CTA
    const int ROWS = G * RT;       // row slots per stage
    const int piece = TX * 36;     // bytes of one row's share of a stage
    const int bpr = p.k >> 6;
    const size_t row_bytes = (size_t)bpr * 36;
    const int nchunks = bpr / TX;
    const int S = p.stages;
    const uint8_t* w0 = p.w0;
    const uint8_t* w1 = p.w1;
    const char* xbase = (const char*)p.x;
    char* ybase = (char*)p.y;
    int rows = p.rows;
    const float *gs0 = p.gs0, *gs1 = p.gs1;
    if (p.ids) {
        // ids, order and tables may come from the kernels just before this one, and a CTA whose expert is not resident
        // returns at once: wait for the predecessor grid first, so that even a grid whose CTAs all return early
        // completes only after its predecessor has
        pdl_wait();
        if ((int)blockIdx.y >= p.combos) {  // a row of the side pair
            const int row = (int)blockIdx.y - p.combos;
            w0 = p.side_w0, w1 = p.side_w1, rows = p.side_rows, gs0 = p.side_gs, gs1 = p.side_gs + 1;
            xbase += (size_t)row * p.k * 4;
            ybase = (char*)(p.side_y + (size_t)row * rows);
        } else {
            const int c = p.order ? p.order[blockIdx.y] : (int)blockIdx.y;
            const int e = p.ids[c];
            if (e < 0 || (p.experts > 0 && e >= p.experts)) return;  // uniform over the CTA, before any barrier
            w0 = (const uint8_t*)p.tab0[e];
            if (!w0) return;  // the expert is not resident here: nothing to read or write
            w1 = p.tab1 ? (const uint8_t*)p.tab1[e] : (p.fused_up_rows > 0 ? w0 + (size_t)p.fused_up_rows * row_bytes : nullptr);
            xbase += (size_t)(c / p.x_div) * p.k * 4;
            ybase = p.yptrs ? (char*)p.yptrs[c] : ybase + (size_t)c * p.ldy * 4;
        }
    }
    const bool gu = w1 != nullptr;

    uint64_t* full = (uint64_t*)smem;
    uint64_t* empty = full + MAX_STAGES;
    float* lut = (float*)(smem + 256);    // [2][256]
    uint8_t* xs0 = smem + HDR_BYTES;                              // [MP][bpr][XB] staged activations
    uint8_t* stage0 = xs0 + (size_t)MP * bpr * XB;                // the weight ring
    const int stage_bytes = ROWS * piece;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // output rows of this CTA: plain ROWS consecutive rows; gate/up ROWS/2 consecutive indices
    const int per_cta = gu ? ROWS / 2 : ROWS;
    const int row0 = blockIdx.x * per_cta;
    if (row0 >= rows) return;  // routed and side matrices of one launch may differ in rows

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);  // the producer's expect_tx arrive; the copies count bytes
            mbar_init(&empty[s], NW);
        }
        mbar_fence_init();
    }
    // scale tables: ue4m3(rule(byte)) * gs, the product the reference tabulates (cpu_nvfp4.rs:98)
    {
        const float g0 = gs0[0], g1 = gu ? gs1[0] : g0;
        for (int b = tid; b < 256; b += NTHREADS) {
            const float u = ue4m3_f32((uint32_t)b, true);
            lut[b] = u * g0;
            lut[256 + b] = u * g1;
        }
    }
    __syncthreads();
    // let the next kernel of the stream begin its own weight prefetch while this one drains
    pdl_launch_dependents();

    if (warp == NW) {
        // ------------------------------------------------------------ weight producer warp
        // source row of slot sl = j*G + g: plain row0 + sl; gate/up: matrix j & 1, index row0 + (j>>1)*G + g
        const uint64_t pol = l2_policy_evict_first();
        const uint8_t* src[4];
        uint32_t total = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int sl = lane + 32 * i;
            src[i] = nullptr;
            if (sl < ROWS) {
                const int j = sl / G, g = sl % G;
                const int r = gu ? row0 + (j >> 1) * G + g : row0 + sl;
                const uint8_t* base = (gu && (j & 1)) ? w1 : w0;
                if (r < rows) src[i] = base + (size_t)r * row_bytes;
            }
            total += src[i] ? piece : 0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        for (int c = 0; c < nchunks; c++) {
            const int s = c % S;
            if (c >= S && !mbar_wait(&empty[s], ((c / S) - 1) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                return;
            }
            uint8_t* st = stage0 + (size_t)s * stage_bytes;
            if (lane == 0) {
                mbar_expect_tx(&full[s], total);
                mbar_arrive(&full[s]);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (src[i]) bulk_g2s_stream(st + (size_t)(lane + 32 * i) * piece, src[i] + (size_t)c * piece, piece, &full[s], pol);
        }
        return;
    }

    // ---------------------------------------------------------------- consumer warps
    // First the activations: every row, the whole K, staged once per CTA while the producer fills
    // the weight ring. Groups of 8 values; lane & 7 = position in the 64-value block, so the 8
    // lanes of a block sit side by side. All loads of a batch are in flight before the first
    // conversion (one L2 round trip per batch, not per group).
    pdl_wait();  // activations may come from the previous kernel of the stream
    constexpr int BATCH = 4;
    const int groups = MP * bpr * 8;
    for (int g0 = 0; g0 < groups; g0 += BATCH * NW * 32) {
        uint4 raw[BATCH][2];
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            const int gq = g0 + b * NW * 32 + tid;
            const int m = gq / (bpr * 8), gi = gq % (bpr * 8);
            raw[b][0] = raw[b][1] = make_uint4(0, 0, 0, 0);
            if (gq < groups && m < p.m) {
                const uint4* x = (const uint4*)((const float*)xbase + (size_t)m * p.k + (size_t)gi * 8);
                raw[b][0] = x[0], raw[b][1] = x[1];
            }
        }
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            const int gq = g0 + b * NW * 32 + tid;
            const int m = gq / (bpr * 8), gi = gq % (bpr * 8), kb = gi >> 3, wi = gi & 7;
            if (gq < groups) {
                uint4* dst = (uint4*)(xs0 + (size_t)(m * bpr + kb) * XB + wi * 32);
                dst[0] = raw[b][0], dst[1] = raw[b][1];
            }
        }
    }
    // the consumer warps only (the producer warp is streaming): named barrier 1
    asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
    const int txi = lane % TX, ry = lane / TX;
    const int g = warp * (32 / TX) + ry;
    float acc[RT][MP];
#pragma unroll
    for (int r = 0; r < RT; r++)
#pragma unroll
        for (int m = 0; m < MP; m++) acc[r][m] = 0.0f;

    for (int c = 0; c < nchunks; c++) {
        const int s = c % S;
        if (!mbar_wait(&full[s], (c / S) & 1)) {
            cn_dev_fail(CN_DEV_WAIT_FULL);
            return;
        }
        const uint8_t* st = stage0 + (size_t)s * stage_bytes;
        uint32_t wv[RT][9];
#pragma unroll
        for (int r = 0; r < RT; r++) {
            const uint32_t* wp = (const uint32_t*)(st + (size_t)(r * G + g) * piece + txi * 36);
#pragma unroll
            for (int i = 0; i < 9; i++) wv[r][i] = wp[i];
        }
        const uint8_t* xs = xs0 + (size_t)(c * TX + txi) * XB;
        float blk[RT][MP];
#pragma unroll
        for (int r = 0; r < RT; r++)
#pragma unroll
            for (int m = 0; m < MP; m++) blk[r][m] = 0.0f;
#pragma unroll
        for (int sb = 0; sb < 4; sb++) {
            float xv[MP][16];
#pragma unroll
            for (int m = 0; m < MP; m++) {
                const float4* xp = (const float4*)(xs + (size_t)m * bpr * XB + sb * 64);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float4 t = xp[i];
                    xv[m][4 * i] = t.x, xv[m][4 * i + 1] = t.y, xv[m][4 * i + 2] = t.z, xv[m][4 * i + 3] = t.w;
                }
            }
#pragma unroll
            for (int r = 0; r < RT; r++) {
                const float sc = lut[((gu && (r & 1)) ? 256 : 0) + ((wv[r][0] >> (8 * sb)) & 0xFF)];
                const uint32_t c0 = wv[r][1 + 2 * sb], c1 = wv[r][2 + 2 * sb];
                float wf[16];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t h0 = e2m1x2_to_f16x2((c0 >> (8 * i)) & 0xFF), h1 = e2m1x2_to_f16x2((c1 >> (8 * i)) & 0xFF);
                    wf[2 * i] = f16lo_to_f32(h0), wf[2 * i + 1] = f16hi_to_f32(h0);
                    wf[8 + 2 * i] = f16lo_to_f32(h1), wf[8 + 2 * i + 1] = f16hi_to_f32(h1);
                }
#pragma unroll
                for (int m = 0; m < MP; m++) {
                    float p0 = 0.0f, p1 = 0.0f;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        p0 = fmaf(wf[2 * i], xv[m][2 * i], p0);
                        p1 = fmaf(wf[2 * i + 1], xv[m][2 * i + 1], p1);
                    }
                    blk[r][m] = fmaf(p0 + p1, sc, blk[r][m]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < RT; r++)
#pragma unroll
            for (int m = 0; m < MP; m++) acc[r][m] += blk[r][m];
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }

    // K split over the TX lanes: xor-shuffle tree, fixed order
#pragma unroll
    for (int r = 0; r < RT; r++)
#pragma unroll
        for (int m = 0; m < MP; m++) {
            float v = acc[r][m];
            for (int o = TX >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            acc[r][m] = v;
        }
    if (txi == 0) {
        if (!gu) {
#pragma unroll
            for (int r = 0; r < RT; r++) {
                const int row = row0 + r * G + g;
                if (row < rows) {
#pragma unroll
                    for (int m = 0; m < MP; m++)
                        if (m < p.m) ((float*)ybase)[(size_t)m * p.ldy + row] = acc[r][m];
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r + 1 < RT; r += 2) {
                const int row = row0 + (r >> 1) * G + g;
                if (row < rows) {
#pragma unroll
                    for (int m = 0; m < MP; m++)
                        if (m < p.m) ((float*)ybase)[(size_t)m * p.ldy + row] = act_gu(acc[r][m], acc[r + 1][m], p.limit);
                }
            }
        }
    }
}

// out[r][c] = e2m1(code) * (ue4m3(byte) * gs): one thread per 8 values (one code word)
__global__ void nvfp4_dequant_kernel(const uint8_t* __restrict__ w, const float* __restrict__ gs, float* __restrict__ out,
                                     long long nwords, int rule) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nwords) return;
    const long long blk = i >> 3;
    const int wi = (int)(i & 7);
    const uint8_t* b = w + blk * 36;
    const float s = ue4m3_f32(b[wi >> 1], rule != 0) * gs[0];
    const uint32_t cw = *(const uint32_t*)(b + 4 + 4 * wi);
    float* o = out + blk * 64 + wi * 8;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t h = e2m1x2_to_f16x2((cw >> (8 * j)) & 0xFF);
        o[2 * j] = f16lo_to_f32(h) * s;
        o[2 * j + 1] = f16hi_to_f32(h) * s;
    }
}

template <int MP, int RT>
int launch_one(const GemvParams& p, int grid, int gy, size_t smem, cudaStream_t stream) {
    auto kern = nvfp4_gemv_kernel<MP, RT>;
    CN_ALLOW_SMEM(kern, 200 * 1024);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, (unsigned)gy);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CN_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return CN_OK;
}

// Four rows per thread only for the many tiles of a routed call, which has one row: a plain call that large (9472 rows of 1024 values) is the tcgen05 kernel's.
int launch_m(const GemvParams& p, int mp, int rt, int grid, int gy, size_t smem, cudaStream_t stream) {
    if (mp == 1 && rt == 4) return launch_one<1, 4>(p, grid, gy, smem, stream);
    if (rt == 2) {
        if (mp == 1) return launch_one<1, 2>(p, grid, gy, smem, stream);
        if (mp == 2) return launch_one<2, 2>(p, grid, gy, smem, stream);
        if (mp == 4) return launch_one<4, 2>(p, grid, gy, smem, stream);
        if (mp == 8) return launch_one<8, 2>(p, grid, gy, smem, stream);
    }
    CN_FAIL(CN_ERR_SHAPE, "nvfp4 gemv: no kernel for m %d, rows per thread %d", mp, rt);
}

}  // namespace

// f32 activations on the fifth-generation tensor cores where a row is long, a matrix large, or a row no whole number of this kernel's steps of 512 values. us a call in a stream of
// dependent ones, there / here for one and eight rows: 12288 x 512 3.0 / 3.4 and 5.7 / 12.6, 8192 x 512 2.9 / 3.1 and 5.4 / 6.4, 4096 x 512 2.8 / 2.3 and 5.0 / 6.0, 2048 x 1024 3.4 / 2.4 and 5.3 / 6.8,
// 256 x 1792 3.2 / 5.3 and 5.4 / 14.7, 256 x 1280 3.2 / 4.1 and 5.5 / 11.4, 256 x 768 3.0 / 3.0 and 5.6 / 8.1; gate / up of 256 x 1280 3.5 / 4.2 and 5.6 / 12.2, of 256 x 768 3.5 / 3.1 and
// 7.4 / 8.8. Against 64 bits a row is 2.7e-8 off there, 1.0e-7 here (normally distributed rows, SiLU rows, cubes, a few channels of a hundred times the rest); where
// three and more of a block's sixteen values are 1e4 times the others and meet zero weights, 3e-6 there, 9e-8 here. The routed form stays here at any k (its rows are as short); from 16 combos on nvfp4_rows_tc.cu takes what it can of it (moe.cu).
// A rule of the matrix alone: a row's result does not depend on how many rows the call has.
static bool f32_digits(int rows, int k, bool gu) {
    const bool odd_steps = k % 512 != 0 && (k >= 1280 || (k >= 768 && rows >= 64 && !gu));
    return k >= 2048 || odd_steps || (k >= 512 && rows >= 8192 && !gu) || (long long)rows * k * (gu ? 2 : 1) >= 6000000;
}
extern "C" int cn_nvfp4_gemv_fixed_bits(int rows, int k, int gate_up, int dtype) {
    if (rows < 1 || k < 256 || k % 256 != 0) return 0;
    return dtype == CN_F32 ? (f32_digits(rows, k, gate_up != 0) ? 31 : 0) : dtype == CN_BF16 && cn_gemv_bf16_digits(rows, k, gate_up != 0) ? 22 : 0;
}

// One launch of the GEMV family (declared in nvfp4_gemv.cuh for the MoE operator).
int cn_gemv_launch(const GemvCall& a, cudaStream_t stream, const char* who) {
    const int rows = a.rows, k = a.k, m = a.m;
    if (rows <= 0 || k <= 0 || k % 256 != 0) CN_FAIL(CN_ERR_SHAPE, "%s: k = %d must be a positive multiple of 256 (rows of 16-byte multiples)", who, k);
    if (m < 1 || m > CN_MAX_M) CN_FAIL(CN_ERR_LIMIT, "%s: m = %d, the kernel takes 1..%d activation rows", who, m, CN_MAX_M);
    if (a.ldy < rows) CN_FAIL(CN_ERR_SHAPE, "%s: ldy %d < rows %d", who, a.ldy, rows);
    if (a.dtype != CN_F32 && a.dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "%s: dtype %d is neither CN_F32 nor CN_BF16", who, a.dtype);
    if (((uintptr_t)a.w0 & 15) || ((uintptr_t)a.w1 & 15) || ((uintptr_t)a.x & 15) || (((uintptr_t)a.side_w0 | (uintptr_t)a.side_w1) & 15))
        CN_FAIL(CN_ERR_SHAPE, "%s: weight and activation pointers must be 16-byte aligned", who);
    const bool routed = a.ids != nullptr;
    if (routed && (m != 1 || a.combos < 1 || a.x_div < 1)) CN_FAIL(CN_ERR_SHAPE, "%s: the routed form takes one row per combo", who);
    // bf16 activations: the tensor-core kernel
    if (a.dtype == CN_BF16) return cn_gemv_m1_launch(a, stream, who);
    if (a.line_bases) CN_FAIL(CN_ERR_SHAPE, "%s: line output takes bf16 activations", who);
    if (!routed && f32_digits(rows, k, a.w1 != nullptr)) {
        if (k > 108544) CN_FAIL(CN_ERR_LIMIT,  // (the library's limit for f32 rows, as it was; this kernel has none)
                                 "%s: k = %d, f32 rows have up to 108544 values", who, k);
        return cn_gemv_tc_launch(a, stream, who);
    }
    const bool gu = a.w1 != nullptr || a.tab1 != nullptr || a.fused_up_rows > 0;
    const int bpr = k / 64;
    const int tx = bpr % 16 == 0 ? 16 : (bpr % 8 == 0 ? 8 : 4);
    const int mp = m == 1 ? 1 : (m == 2 ? 2 : (m <= 4 ? 4 : 8));
    const int G = NW * (32 / tx);
    int rt = 4;
    const long long slots = (long long)rows * (gu ? 2 : 1) * (routed ? a.combos : 1);
    if (slots / (G * 4) < 2 * 148) rt = 2;
    const int ROWS = G * rt;
    const int per_cta = gu ? ROWS / 2 : ROWS;
    const int grid = ((routed && a.side_tokens > 0 && a.side_rows > rows ? a.side_rows : rows) + per_cta - 1) / per_cta;
    const size_t stage_bytes = (size_t)ROWS * tx * 36;
    const size_t xbytes = (size_t)mp * bpr * XB;
    const int nchunks = bpr / tx;
    // ring depth: enough bytes in flight per SM to cover the HBM latency (about 96 KB), shared between
    // the CTAs that will be resident together (at most four, fewer when the grid is small)
    const long long total_ctas = (long long)grid * (routed ? a.combos + a.side_tokens : 1);
    int resident = (int)((total_ctas + 147) / 148);
    resident = resident < 1 ? 1 : (resident > 4 ? 4 : resident);
    long long want = (96 * 1024) / resident;                                         // in-flight bytes per CTA
    long long cap = (208 * 1024) / resident - (long long)HDR_BYTES - (long long)xbytes;  // what fits beside the activations
    if (want > cap) want = cap;
    int stages = (int)((want + (long long)stage_bytes - 1) / (long long)stage_bytes);
    stages = stages < 2 ? 2 : (stages > MAX_STAGES ? MAX_STAGES : stages);
    if (stages > nchunks) stages = nchunks < 1 ? 1 : nchunks;
    const size_t smem = HDR_BYTES + xbytes + stages * stage_bytes;
    if (smem + (size_t)mp * bpr * 4 > 200 * 1024) {  // (four bytes a block to spare: the limits are those of a layout that had a scale beside each)
        // the staged activations of all m rows do not fit one CTA: two calls over half the rows each
        // (each row's arithmetic is the same whatever the split, so results do not change)
        if (m == 1) CN_FAIL(CN_ERR_LIMIT, "%s: k = %d needs %zu B of shared memory per block", who, k, smem);
        const int m0 = m / 2;
        GemvCall lo = a, hi = a;
        lo.m = m0;
        hi.m = m - m0;
        hi.x = (const float*)a.x + (size_t)m0 * k;
        hi.y = (float*)a.y + (size_t)m0 * a.ldy;
        int rc = cn_gemv_launch(lo, stream, who);
        return rc ? rc : cn_gemv_launch(hi, stream, who);
    }
    GemvParams p;
    p.w0 = (const uint8_t*)a.w0, p.w1 = (const uint8_t*)a.w1, p.gs0 = a.gs0, p.gs1 = a.gs1 ? a.gs1 : a.gs0, p.x = a.x, p.y = a.y;
    p.rows = rows, p.k = k, p.m = m, p.ldy = a.ldy, p.limit = a.limit, p.tx = tx, p.stages = stages, p.out_f32 = a.out_f32;
    p.ids = a.ids, p.order = a.order, p.tab0 = a.tab0, p.tab1 = a.tab1, p.fused_up_rows = a.fused_up_rows, p.x_div = a.x_div;
    p.experts = a.experts, p.yptrs = a.yptrs;
    p.combos = a.combos, p.side_w0 = (const uint8_t*)a.side_w0, p.side_w1 = (const uint8_t*)a.side_w1, p.side_gs = a.side_gs, p.side_y = a.side_y;
    p.side_rows = a.side_rows;
    const int gy = routed ? a.combos + a.side_tokens : 1;
    return launch_m(p, mp, rt, grid, gy, smem, stream);
}

extern "C" int cn_nvfp4_gemv(const void* w, const float* gs, const void* x, void* y, int rows, int k, int m, int ldy, int dtype,
                             cn_stream_t stream) {
    GemvCall a = {};
    a.w0 = w, a.gs0 = gs, a.x = x, a.y = y, a.rows = rows, a.k = k, a.m = m, a.ldy = ldy, a.dtype = dtype;
    return cn_gemv_launch(a, (cudaStream_t)stream, "cn_nvfp4_gemv");
}

extern "C" int cn_nvfp4_gemv_gu(const void* wg, const void* wu, const float* gs_g, const float* gs_u, const void* x, void* h, int inter,
                                int k, int m, int ldh, float limit, int dtype, cn_stream_t stream) {
    if (!wu) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemv_gu: the up matrix is null");
    GemvCall a = {};
    a.w0 = wg, a.w1 = wu, a.gs0 = gs_g, a.gs1 = gs_u, a.x = x, a.y = h, a.rows = inter, a.k = k, a.m = m, a.ldy = ldh, a.limit = limit,
    a.dtype = dtype;
    return cn_gemv_launch(a, (cudaStream_t)stream, "cn_nvfp4_gemv_gu");
}

extern "C" int cn_nvfp4_gemv_lines(const void* w, const float* gs, const void* x, void* y, int rows, int k, const unsigned long long* line_bases,
                                   int world, int row0, size_t line_stride, const unsigned int* epoch, int tag, int buf, int flip, cn_stream_t stream) {
    if (!line_bases || !epoch) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemv_lines: null line buffers or step counter");
    GemvCall a = {};
    a.w0 = w, a.gs0 = gs, a.x = x, a.y = y, a.rows = rows, a.k = k, a.m = 1, a.ldy = rows, a.dtype = CN_BF16;
    a.line_bases = line_bases, a.line_world = world, a.line_row0 = row0, a.line_stride = line_stride, a.line_epoch = epoch;
    a.line_tag = tag, a.line_buf = buf, a.line_flip = flip;
    return cn_gemv_launch(a, (cudaStream_t)stream, "cn_nvfp4_gemv_lines");
}

extern "C" int cn_nvfp4_gemv_gu_lines(const void* wg, const void* wu, const float* gs_g, const float* gs_u, const void* x, void* h, int inter, int k,
                                      float limit, const unsigned long long* line_bases, int world, int row0, size_t line_stride,
                                      const unsigned int* epoch, int tag, int buf, int flip, cn_stream_t stream) {
    if (!wu) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemv_gu_lines: the up matrix is null");
    if (!line_bases || !epoch) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_gemv_gu_lines: null line buffers or step counter");
    GemvCall a = {};
    a.w0 = wg, a.w1 = wu, a.gs0 = gs_g, a.gs1 = gs_u, a.x = x, a.y = h, a.rows = inter, a.k = k, a.m = 1, a.ldy = inter, a.limit = limit,
    a.dtype = CN_BF16;
    a.line_bases = line_bases, a.line_world = world, a.line_row0 = row0, a.line_stride = line_stride, a.line_epoch = epoch;
    a.line_tag = tag, a.line_buf = buf, a.line_flip = flip;
    return cn_gemv_launch(a, (cudaStream_t)stream, "cn_nvfp4_gemv_gu_lines");
}

extern "C" int cn_nvfp4_dequant(const void* w, const float* gs, float* out, int rows, int k, int rule, cn_stream_t stream) {
    if (rows <= 0 || k <= 0 || k % 64 != 0) CN_FAIL(CN_ERR_SHAPE, "cn_nvfp4_dequant: %d columns are not whole 64-value NVFP4 blocks", k);
    const long long nwords = (long long)rows * (k / 64) * 8;
    const int threads = 256;
    const long long blocks = (nwords + threads - 1) / threads;
    nvfp4_dequant_kernel<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>((const uint8_t*)w, gs, out, nwords, rule);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}
