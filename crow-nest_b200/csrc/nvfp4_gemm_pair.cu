// NVFP4 GEMM for more than 128 activation rows (prompt chunks): Y[t][n] = gs * sum_k X[t][k] * W[n][k] on CTA pairs.
//
// Supersedes the reference's prompt GEMMs gemm_fp4_dense (engine/src/kernels.rs:533) and glm5_gemm_fp4_tc
// (engine/src/kernels_glm5_moe.cu:349: weights decoded losslessly, f32 accumulate). Same arithmetic here: an E2M1 code
// times its UE4M3 scale is exact in bf16 and in f16, so bf16 activations go to the tensor cores as they are (no pass
// over them at all), f32 activations as f16 x 2^k per row (gemm_prep_x_kernel), and accumulation is f32.
//
// What bounds it: the tensor pipe. A 128-row x 256-token tile of one CTA would move 32 KB of activations into shared
// memory and read them (and 16 KB of widened weights) back per 64 values of K, 96 KB against the 64 KB that the port
// moves in the 512 cycles of the MMAs. Hence
//   - the widened weights never touch shared memory: they are the A operand in TENSOR MEMORY. A decode thread owns one
//     weight row (= one lane), reads its 36-byte block from a 144-byte row piece (TMA box of four blocks, 128-bit loads
//     at an odd multiple of 16 bytes: no bank conflicts) and stores the 32 registers of the 64 values with one tcgen05.st;
//   - two CTAs share a 256-row tile (cta_group::2): each holds half of the tile's activation rows, 16 KB per step.
//
// Roles of a CTA (640 threads): warp 0 brings in the weights (its own 128 rows) and the activations (its half of the
// tile's rows), warp 1 of the even CTA issues the MMAs of the pair, two sets of four warps (4-11) decode alternate 64-value blocks,
// warps 12-19 write results. Tiles are walked persistently, one pair per two SMs; with up to 192 tokens per tile there
// are two accumulators and the epilogue of a tile runs under the MMAs of the next.
// Rings: weights 3 x 18 KB (256 values of K each), activations up to 8 x 16 KB and A slots 4..8 x 32 columns (64 values).
// Every wait is bounded. The weights are read with L2's ordinary policy: kept as evict-last, for the token tiles that read them again, they
// gained nothing (512 rows 76.6 and 76.9 us) and stayed behind: a 50 MB matrix read twice after the call took 83 us the second time, 75 now.
// Measured over the public call with inputs that change from pass to pass: 17408 x 5120 at 512 rows 155 -> 76 us (1.2 PFLOP/s; one CTA
// per tile with both operands in shared memory before), 5120 x 17408 at 4096 rows 1190 -> 560 us (1.3 PFLOP/s, at the power cap). What
// got it there beside the layout: MMA issue from a converged warp (elect_lane) and no cluster-scope fences on the rings' barriers (tc5.cuh).
#include "nvfp4_gemm.cuh"
#include "tc5.cuh"

namespace {

constexpr int W_STAGE = 128 * 144, NW_STAGES = 3;
constexpr int PAIR_THREADS = 640;
constexpr int HDR = 1024;
constexpr int SMEM_MAX = 227 * 1024;
constexpr int TMEM_COLS = 512;

struct PairParams {
    const float* gs;
    const float* rs;  // per activation row (f16 rows)
    void* y;
    int rows, m, ldy, pair_store;
    int nk;                      // 64-value blocks of K
    int tn, acc_stride, nacc, na, nb;  // tokens per tile; accumulator columns and count; A and activation ring depths
    int row_tiles, tiles;
};

// Blocks SET and SET + 2 of every weight stage, one row per thread: block b is nine words from word 9 b of the row's 144
// bytes, inside three 16-byte chunks. (Four sets of one block each measured 5 % slower at 200 - 1000 rows.)
template <bool BF16, int SET>
__device__ __forceinline__ void decode_set(uint32_t src, uint32_t dst, uint64_t* wfull, uint64_t* wempty, uint64_t* aempty, uint32_t afull_base, int stages,
                                           int na, int lane) {
    int ws = 0, as = SET;
    uint32_t wp = 0, ap = 1;
    for (int w = 0; w < stages; w++) {
        if (!mbar_wait(&wfull[ws], wp)) {
            cn_dev_fail(CN_DEV_WAIT_FULL);
            return;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int b = SET + 2 * h;
            uint32_t c[12], v[32];
            const uint32_t at = src + (uint32_t)ws * W_STAGE + (uint32_t)((9 * b) >> 2) * 16u;
#pragma unroll
            for (int i = 0; i < 3; i++)
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(c[4 * i]), "=r"(c[4 * i + 1]), "=r"(c[4 * i + 2]), "=r"(c[4 * i + 3])
                             : "r"(at + 16u * i));
            if (BF16)
                decode64_bf16(c + b, v);
            else
                decode64_f16(c + b, v);
            if (h == 1) {  // the stage has been read
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[ws]);
            }
            if (!mbar_wait(&aempty[as], ap)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                return;
            }
            tc_after();
            tc_st32(dst + (uint32_t)as * 32u, v);
            tc_wait_st();
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(afull_base + 8u * (uint32_t)as);
            as += 2;
            if (as >= na) as -= na, ap ^= 1u;
        }
        if (++ws == NW_STAGES) ws = 0, wp ^= 1u;
    }
}

template <bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
    nvfp4_gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const PairParams p) {
    extern __shared__ uint8_t smem_raw[];
    // barriers: wfull 3, wempty 3, bfull 8, bempty 8, afull 8, aempty 8, accfull 2, accempty 2
    uint64_t* wfull = (uint64_t*)smem_raw;
    uint64_t* wempty = wfull + NW_STAGES;
    uint64_t* bfull = wempty + NW_STAGES;
    uint64_t* bempty = bfull + 8;
    uint64_t* afull = bempty + 8;
    uint64_t* aempty = afull + 8;
    uint64_t* accfull = aempty + 8;
    uint64_t* accempty = accfull + 2;
    uint32_t* tmem_slot = (uint32_t*)(accempty + 2);
    const uint32_t ring = (smem_u32(smem_raw) + HDR + 1023u) & ~1023u;
    const uint32_t bbox = (uint32_t)p.tn * 64u, bslot = 2u * bbox;  // tn / 2 rows of 128 bytes, twice
    const uint32_t wring = ring + (uint32_t)p.nb * bslot;

    const int tid = threadIdx.x, warp = (int)warp_uniform((uint32_t)tid >> 5), lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int nw = p.nk >> 2;  // weight stages per tile (k is a multiple of 256)

    if (tid == 0) {
        for (int i = 0; i < NW_STAGES; i++) mbar_init(&wfull[i], 1), mbar_init(&wempty[i], 8);
        for (int i = 0; i < 8; i++) mbar_init(&bfull[i], 1), mbar_init(&bempty[i], 1), mbar_init(&afull[i], 8), mbar_init(&aempty[i], 1);
        for (int i = 0; i < 2; i++) mbar_init(&accfull[i], 1), mbar_init(&accempty[i], 16);
        mbar_fence_init();
    }
    if (warp == 2) tc_alloc<2>(tmem_slot, TMEM_COLS);
    tc_before();
    __syncthreads();
    cluster_sync_ctas();  // both CTAs' barriers exist before anything arrives on them
    tc_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    const uint32_t acol = tmem + (uint32_t)(p.nacc * p.acc_stride);

    if (warp == 0) {
        // ------------------------------------------------------------ weights and activations in
        if (lane == 0) {
            tma_prefetch_map(&wmap), tma_prefetch_map(&xmap);
            int ws = 0, bs = 0;
            uint32_t wp = 1, bp = 1;  // parity of "empty": the first round passes at once
            bool ok = true;
            const uint32_t bfull0 = smem_u32(bfull) & 0xFEFFFFFFu;  // the even CTA's barriers
            for (int tile = pair; tile < p.tiles && ok; tile += npairs) {
                const int row0 = (tile % p.row_tiles) * 256 + (int)rank * 128, tok0 = (tile / p.row_tiles) * p.tn + (int)rank * (p.tn >> 1);
                for (int w = 0; w < nw && ok; w++) {
                    if (!mbar_wait(&wempty[ws], wp)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&wfull[ws], W_STAGE);
                    mbar_arrive(&wfull[ws]);
                    tma_load_2d(wring + (uint32_t)ws * W_STAGE, &wmap, w * 36, row0, smem_u32(&wfull[ws]));
                    if (++ws == NW_STAGES) ws = 0, wp ^= 1u;
                    for (int q = 0; q < 2; q++) {
                        if (!mbar_wait(&bempty[bs], bp)) {
                            cn_dev_fail(CN_DEV_WAIT_EMPTY);
                            ok = false;
                            break;
                        }
                        if (rank == 0) {  // the even CTA's barrier counts both halves
                            mbar_expect_tx(&bfull[bs], 2u * bslot);
                            mbar_arrive(&bfull[bs]);
                        }
                        tma_load_2d_pair(ring + (uint32_t)bs * bslot, &xmap, (w * 4 + 2 * q) * 64, tok0, bfull0 + 8u * (uint32_t)bs);
                        tma_load_2d_pair(ring + (uint32_t)bs * bslot + bbox, &xmap, (w * 4 + 2 * q + 1) * 64, tok0, bfull0 + 8u * (uint32_t)bs);
                        if (++bs == p.nb) bs = 0, bp ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issue, even CTA only
        if (rank == 0) {
            const uint32_t idesc = tc_idesc_f16(256, p.tn, BF16);
            const uint64_t bdesc0 = tc_desc_sw128(warp_uniform(ring));
            int as = 0, bs = 0, ab = 0;
            uint32_t ap = 0, bp = 0, cp = 1;
            bool ok = true;
            for (int tile = pair; tile < p.tiles && ok; tile += npairs) {
                if (!mbar_wait(&accempty[ab], cp)) {
                    cn_dev_fail(CN_DEV_WAIT_EMPTY);
                    break;
                }
                tc_after();
                const uint32_t d = tmem + (uint32_t)(ab * p.acc_stride);
                for (int kb = 0; kb < p.nk; kb += 2) {
                    if (!mbar_wait(&bfull[bs], bp)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        if (!mbar_wait(&afull[as], ap)) ok = false;
                        tc_after();
                        const uint32_t a = acol + (uint32_t)as * 32u;
                        const uint64_t b = bdesc0 + (((uint32_t)bs * bslot + (uint32_t)h * bbox) >> 4);
                        if (elect_lane()) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)  // 16 values: 8 columns of A, 32 bytes of B inside the swizzled row
                                tc_mma_ts<2>(d, a + 8u * kk, b + 2u * kk, idesc, (kb > 0 || h > 0 || kk > 0) ? 1u : 0u);
                            tc_commit<2>(&aempty[as]);
                            if (h == 1) tc_commit<2>(&bempty[bs]);
                        }
                        __syncwarp();
                        if (++as == p.na) as = 0, ap ^= 1u;
                    }
                    if (!ok) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        break;
                    }
                    if (++bs == p.nb) bs = 0, bp ^= 1u;
                }
                if (!ok) break;
                if (elect_lane()) tc_commit<2>(&accfull[ab]);
                __syncwarp();
                if (++ab == p.nacc) ab = 0, cp ^= 1u;
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------------------------------------ decode
        const uint32_t src = wring + (uint32_t)(32 * (warp & 3) + lane) * 144u;
        const uint32_t dst = acol + ((uint32_t)(32 * (warp & 3)) << 16);
        const uint32_t afull_base = cluster_addr(smem_u32(afull), 0);
        const int stages = pair < p.tiles ? nw * ((p.tiles - pair + npairs - 1) / npairs) : 0;
        if (warp < 8)
            decode_set<BF16, 0>(src, dst, wfull, wempty, aempty, afull_base, stages, p.na, lane);
        else
            decode_set<BF16, 1>(src, dst, wfull, wempty, aempty, afull_base, stages, p.na, lane);
    } else if (warp >= 12) {
        // ------------------------------------------------------------ results: lane = weight row, 32 tokens per load, two warps per
        // quarter of the rows take alternate loads
        const int quarter = warp & 3;
        const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
        const uint32_t accempty_base = cluster_addr(smem_u32(accempty), 0);
        const float gs = p.gs[0] * (BF16 ? BF16_UNSCALE : F16_UNSCALE);
        const int odd = lane & 1;
        int ab = 0;
        uint32_t cp = 0;
        for (int tile = pair; tile < p.tiles; tile += npairs) {
            if (!mbar_wait(&accfull[ab], cp)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            tc_after();
            const int rbase = (tile % p.row_tiles) * 256 + (int)rank * 128 + 32 * quarter, row = rbase + lane, tok0 = (tile / p.row_tiles) * p.tn;
            const int live = min(p.tn, p.m - tok0);
            for (int c0 = 32 * ((warp - 12) >> 2); c0 < live; c0 += 64) {
                uint32_t v[32];
                tc_ld32(tmem + lanes + (uint32_t)(ab * p.acc_stride + c0), v);
                tc_wait_ld();
                if (BF16 && p.pair_store) {
                    // bf16 rows two at a time: lanes l, l + 1 trade so that the even one holds both rows of token c0 + i, the odd one
                    // both of token c0 + i + 1, and a warp's store is 64 contiguous bytes of each
                    __nv_bfloat16* yp = (__nv_bfloat16*)p.y + (size_t)(tok0 + c0 + odd) * p.ldy + (row & ~1);
                    const size_t step = 2 * (size_t)p.ldy;
                    const bool whole = live - c0 >= 32 && rbase + 32 <= p.rows;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float a = __uint_as_float(v[i]) * gs, b = __uint_as_float(v[i + 1]) * gs;
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
                        const __nv_bfloat162 o = __floats2bfloat162_rn(odd ? other : a, odd ? b : other);
                        if (whole || (c0 + i + odd < live && row < p.rows)) *(__nv_bfloat162*)yp = o;
                        yp += step;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const int tok = tok0 + c0 + i;
                        if (c0 + i < live && row < p.rows) {
                            const float r = __uint_as_float(v[i]) * (BF16 ? gs : gs * p.rs[tok]);
                            if (BF16)
                                ((__nv_bfloat16*)p.y)[(size_t)tok * p.ldy + row] = __float2bfloat16_rn(r);
                            else
                                ((float*)p.y)[(size_t)tok * p.ldy + row] = r;
                        }
                    }
                }
            }
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(accempty_base + 8u * (uint32_t)ab);
            if (++ab == p.nacc) ab = 0, cp ^= 1u;
        }
    }
    tc_before();
    __syncthreads();
    cluster_sync_ctas();  // nobody leaves while the other CTA may still arrive on its barriers or the pair's MMAs read its memory
    if (warp == 2) tc_dealloc<2>(tmem, TMEM_COLS);
}

// Tokens per tile: the multiple of 32 up to 256 whose tiles fill the pairs' rounds best. A round costs the longer of the
// MMAs (2 cycles per token and 64-value block) and the decode (about 300 cycles per block bf16, 170 f16), plus the
// epilogue where a single accumulator leaves it exposed.
int pair_tokens(int rows, int nk, int m, int pairs, bool bf16) {
    const int rt = (rows + 255) / 256, most = (m + 31) / 32 * 32 < 256 ? (m + 31) / 32 * 32 : 256;
    double best = 1e30;
    int tn = most;
    for (int n = (m + most - 1) / most; n <= (m + 31) / 32; n++) {  // token tiles
        const int t = ((m + n - 1) / n + 31) / 32 * 32;
        const long long tiles = (long long)rt * ((m + t - 1) / t);
        const long long rounds = (tiles + pairs - 1) / pairs;
        const double step = 2.0 * t > (bf16 ? 300.0 : 170.0) ? 2.0 * t : (bf16 ? 300.0 : 170.0);
        const double tail = 2500.0 + 16.0 * t;
        const double cost = rounds * (nk * step + (t > 192 ? tail : 400.0)) + (t > 192 ? 0.0 : tail);
        if (cost < best) best = cost, tn = t;
        if (t <= 64) break;
    }
    return tn;
}

}  // namespace

int cn_gemm_pair_launch(const GemmCall& c, cudaStream_t stream) {
    CUtensorMap wmap, xmap;
    const int nk = c.k / 64;
    PairParams p = {};
    p.gs = c.gs, p.rs = c.x_f16 ? c.rs : nullptr, p.y = c.y, p.rows = c.rows, p.m = c.m, p.ldy = c.ldy, p.nk = nk;
    p.pair_store = !((c.rows | c.ldy) & 1) && !((uintptr_t)c.y & 3);
    const int pairs = 74;
    p.tn = pair_tokens(c.rows, nk, c.m, pairs, !c.x_f16);
    p.acc_stride = p.tn;
    p.nacc = p.tn <= 192 ? 2 : 1;
    p.na = (TMEM_COLS - p.nacc * p.acc_stride) / 32;
    p.na = p.na > 8 ? 8 : p.na & ~1;
    p.nb = (SMEM_MAX - HDR - 1024 - NW_STAGES * W_STAGE) / (p.tn * 128);
    if (p.nb > 8) p.nb = 8;
    p.row_tiles = (c.rows + 255) / 256;
    p.tiles = p.row_tiles * ((c.m + p.tn - 1) / p.tn);
    if (int rc = cn_tmap_2d(&wmap, c.w, 4, (unsigned long long)nk * 9, c.rows, (unsigned long long)nk * 36, 36, 128)) return rc;
    if (int rc = cn_tmap_2d(&xmap, c.x, c.x_f16 ? 2 : 3, c.k, c.m, (unsigned long long)c.k * 2, 64, p.tn / 2)) return rc;
    const size_t smem = HDR + 1024 + (size_t)NW_STAGES * W_STAGE + (size_t)p.nb * p.tn * 128;
    auto kern = c.x_f16 ? nvfp4_gemm_pair_kernel<false> : nvfp4_gemm_pair_kernel<true>;
    CN_ALLOW_SMEM(kern, SMEM_MAX);
    const int grid = 2 * (p.tiles < pairs ? p.tiles : pairs);
    kern<<<grid, PAIR_THREADS, smem, stream>>>(wmap, xmap, p);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}
