// NVFP4 GEMM on CTA pairs (batched verify, prompts): Y[t][n] = gs * sum_k X[t][k] * W[n][k], weights in the container layout or re-laid
// (the stage images of nvfp4_gemm_bs.cu).
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
// Rings: weights 3 to 6 x 18 KB (256 values of K each); beyond 128 rows activations in slots of 128 values (up to 8) and A slots of 64 (4 to 8, 32 columns each), up to 128 rows both in slots
// of 256 (four and three): every slot costs the thread that asks for it some 300 cycles and the one that issues its MMAs 100, whatever it holds.
//
// Up to 128 rows the way of a block through a decode warp bounds it (650 cycles of 1000 a stage), up to some 90 rows, then the MMAs, and the start and end of a launch (8 us of a call: the
// kernel that prepares the rows, this one, and the one that adds the parts wait for one another); hence f16 (half the instructions of the decode to bf16), with the rows brought into f16 by a
// kernel before this one that runs under this one's prologue, all sixteen warps decoding, and K split where row tiles do not fill the pairs. 17408 x 5120 at 64 rows, us in a graph of
// calls: 80 (one CTA per tile, widened weights through shared memory), 20.6 (rings of 64 and 128 values, two boxes for each activation slot: 303 cycles a block, the rate
// of the thread that asked for the boxes, at 16 rows as at 64), 17.1; container bytes 20.9 -> 18.2; 5120 x 17408 26.1 -> 21.5, 8192 x 5120 at 128 rows 20.2 -> 16.7.
// Every wait is bounded. The weights are read with L2's ordinary policy: kept as evict-last, for the token tiles that read them again, they
// gained nothing (512 rows 76.6 and 76.9 us) and stayed behind: a 50 MB matrix read twice after the call took 83 us the second time, 75 now.
// Measured over the public call with inputs that change from pass to pass: 17408 x 5120 at 512 rows 155 -> 76 us (1.2 PFLOP/s; one CTA
// per tile with both operands in shared memory before), 5120 x 17408 at 4096 rows 1190 -> 560 us (1.3 PFLOP/s, at the power cap). What
// got it there beside the layout: MMA issue from a converged warp (elect_lane) and no cluster-scope fences on the rings' barriers (tc5.cuh).
#include "nvfp4_gemm.cuh"
#include "tc5.cuh"

namespace {

constexpr int W_STAGE = 128 * 144;  // 256 values of K of 128 rows: container bytes, or the stage image of the re-laid weights
constexpr int MAX_W_STAGES = 6;
__host__ __device__ constexpr int slot_blocks(int sets) { return sets == 4 ? 4 : 1; }  // 64-value blocks of an A slot
__host__ __device__ constexpr int box_blocks(int sets) { return sets == 4 ? 4 : 2; }   // and of an activation slot
constexpr int PAIR_THREADS = 640;
constexpr int HDR = 1024;
constexpr int SMEM_MAX = 227 * 1024;
constexpr int TMEM_COLS = 512;

struct PairParams {
    const float* gs;
    const float* rs;  // per activation row (f16 rows)
    void* y;
    int rows, m, ldy, out_bf16, pair_store;  // pair_store: bf16 results two rows at a time
    int nk;                      // 64-value blocks of K
    int tn, acc_stride, nacc, na, nb, nws;  // tokens per tile; accumulator columns and count; A, activation and weight ring depths (slots)
    int row_tiles, tiles, ksplits;
    int split_stages, split_more;  // weight stages of a part of K; the first split_more parts have one more
    const uint8_t* packed;  // re-laid weights (cn_nvfp4_bs_repack), or null: container bytes through wmap
    int packed_tiles;       // 128-row tiles of them
    float* part;            // ksplits > 1: raw sums [ksplits][m][rows]
};
// A pair's work comes in units, a tile and a part of K (all of it with one split), in the order of the splits. Counted up instead of
// divided out, so that the compiler sees what the whole warp shares: with a quotient in the MMA warp's loop bounds its operands left the
// uniform registers (17408 x 5120, 64 rows: 25 -> 29 us; 4096 rows of 5120 x 17408: 585 -> 616).
template <bool SPLIT>
struct Unit {
    int tile, split;
    __device__ __forceinline__ explicit Unit(int pair, const PairParams& p) : tile(pair), split(0) { wrap(p); }
    __device__ __forceinline__ void wrap(const PairParams& p) {
        while (SPLIT && tile >= p.tiles && split < p.ksplits) tile -= p.tiles, split++;
    }
    __device__ __forceinline__ bool live(const PairParams& p) const { return SPLIT ? split < p.ksplits : tile < p.tiles; }
    __device__ __forceinline__ void next(int npairs, const PairParams& p) { tile += npairs, wrap(p); }
    __device__ __forceinline__ int first(const PairParams& p) const { return SPLIT ? split * p.split_stages + min(split, p.split_more) : 0; }
    __device__ __forceinline__ int count(const PairParams& p) const { return SPLIT ? p.split_stages + (split < p.split_more ? 1 : 0) : p.nk >> 2; }
};

// Where a decode warp stands in the rings of weight stages and A slots.
struct DecodeAt {
    int ws, as;
    uint32_t wp, ap;
};
// Block b of the stage's row at `at` (its scale word at `scale` where the weights are re-laid): scale word and eight code words. Container: nine words from word 9 b of the row's 144 bytes,
// inside three 16-byte chunks. Re-laid: codes are chunks 2 b and 2 b + 1 of the row's 128 swizzled bytes, the scale word lies in the image's scale part.
__device__ __forceinline__ void lds128(uint32_t* v, uint32_t at) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at));
}
template <int B>
__device__ __forceinline__ void load_container(uint32_t (&c)[9], uint32_t at) {
    uint32_t t[12];
#pragma unroll
    for (int i = 0; i < 3; i++) lds128(t + 4 * i, at + (uint32_t)(((9 * B) >> 2) + i) * 16u);
#pragma unroll
    for (int i = 0; i < 9; i++) c[i] = t[B + i];
}
template <bool PACKED>
__device__ __forceinline__ void load_block(uint32_t (&c)[9], uint32_t at, uint32_t scale, int b, int lane) {
    if (PACKED) {
        lds128(c + 1, at + (uint32_t)(((2 * b) ^ (lane & 7)) << 4));
        lds128(c + 5, at + (uint32_t)(((2 * b + 1) ^ (lane & 7)) << 4));
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(c[0]) : "r"(scale + 512u * b));
    } else if (b == 0) {
        load_container<0>(c, at);
    } else if (b == 1) {
        load_container<1>(c, at);
    } else if (b == 2) {
        load_container<2>(c, at);
    } else {
        load_container<3>(c, at);
    }
}
// Every SETS-th block of `stages` weight stages from block `set` on, one row per thread. Two sets of warps where the MMAs or the ALUs bound the loop (four of one block each measured 5 %
// slower at 200 - 1000 rows of bf16), four where it is the way of a block - load, decode, store to tensor memory, arrival - that does. Four sets run one copy of the code (SET = -1): with
// one for each, instructions come late (17408 x 5120, 64 rows: 18.0 us a call on re-laid weights, 17.1 so). Two have one each, SET = 0 and 1, whose blocks the compiler knows
// (5120 x 17408 at 512 rows: 72 us, 77 with one copy).
template <bool BF16, bool PACKED, int SETS, int SET>
__device__ __forceinline__ void decode_set(uint32_t src, uint32_t scales, uint32_t dst, uint64_t* wfull, uint64_t* wempty, uint64_t* aempty, uint32_t afull_base,
                                           int stages, int nws, int na, int lane, int which, DecodeAt& at_) {
    constexpr int G = slot_blocks(SETS);
    const int set = SET < 0 ? which : SET;
    int ws = at_.ws, as = at_.as;
    uint32_t wp = at_.wp, ap = at_.ap;
    const uint32_t col = dst + 32u * (uint32_t)(set % G);
    for (int w = 0; w < stages; w++) {
        if (!mbar_wait(&wfull[ws], wp)) {
            cn_dev_fail(CN_DEV_WAIT_FULL);
            return;
        }
#pragma unroll
        for (int j = 0; j < 4 / SETS; j++) {
            uint32_t c[9], v[32];
            load_block<PACKED>(c, src + (uint32_t)ws * W_STAGE, scales + (uint32_t)ws * W_STAGE, set + SETS * j, lane);
            if (BF16)
                decode64_bf16(c, v);
            else
                decode64_f16(c, v);
            if (j == 4 / SETS - 1) {  // the stage has been read
                __syncwarp();
                if (lane == 0) mbar_arrive(&wempty[ws]);
            }
            if (!mbar_wait(&aempty[as], ap)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                return;
            }
            tc_after();
            tc_st32(col + (uint32_t)as * (32u * G), v);
            tc_wait_st();
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(afull_base + 8u * (uint32_t)as);
            as += SETS / G;
            if (as >= na) as -= na, ap ^= 1u;
        }
        if (++ws == nws) ws = 0, wp ^= 1u;
    }
    at_ = {ws, as, wp, ap};
}

// SETS = 4 (f16 rows, at most 128 tokens per tile): all sixteen warps decode and write a unit's results when they have decoded it.
// SPLIT: K may be split; without it the exposed epilogue of a single accumulator carries none of that code (512 rows 77.6 us with, 77.0 without).
template <bool BF16, bool PACKED, int SETS, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
    nvfp4_gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const PairParams p) {
    constexpr int G = slot_blocks(SETS), KB = box_blocks(SETS);
    extern __shared__ uint8_t smem_raw[];
    // barriers: wfull 6, wempty 6, bfull 8, bempty 8, afull 8, aempty 8, accfull 2, accempty 2
    uint64_t* wfull = (uint64_t*)smem_raw;
    uint64_t* wempty = wfull + MAX_W_STAGES;
    uint64_t* bfull = wempty + MAX_W_STAGES;
    uint64_t* bempty = bfull + 8;
    uint64_t* afull = bempty + 8;
    uint64_t* aempty = afull + 8;
    uint64_t* accfull = aempty + 8;
    uint64_t* accempty = accfull + 2;
    uint32_t* tmem_slot = (uint32_t*)(accempty + 2);
    const uint32_t ring = (smem_u32(smem_raw) + HDR + 1023u) & ~1023u;
    const uint32_t bbox = (uint32_t)p.tn * 64u, bslot = KB * bbox;  // tn / 2 rows of 128 bytes, for every block of a slot
    const uint32_t wring = ring + (uint32_t)p.nb * bslot;

    const int tid = threadIdx.x, warp = (int)warp_uniform((uint32_t)tid >> 5), lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int nw = p.nk >> 2;  // weight stages per tile (k is a multiple of 256)

    if (tid == 0) {
        for (int i = 0; i < MAX_W_STAGES; i++) mbar_init(&wfull[i], 1), mbar_init(&wempty[i], 4 * SETS);
        for (int i = 0; i < 8; i++) mbar_init(&bfull[i], 1), mbar_init(&bempty[i], 1), mbar_init(&afull[i], 8 * G), mbar_init(&aempty[i], 1);
        for (int i = 0; i < 2; i++) mbar_init(&accfull[i], 1), mbar_init(&accempty[i], SETS == 4 ? 32 : 16);
        mbar_fence_init();
    }
    if (warp == 2) tc_alloc<2>(tmem_slot, TMEM_COLS);
    tc_before();
    __syncthreads();
    cluster_sync_ctas();  // both CTAs' barriers exist before anything arrives on them
    tc_after();
    pdl_launch_dependents();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    const uint32_t acol = tmem + (uint32_t)(p.nacc * p.acc_stride);

    DecodeAt at = {0, ((warp - 4) >> 2) / G, 0u, 1u};
    auto decode = [&](int stages) {
        const uint32_t src = wring + (uint32_t)(32 * (warp & 3) + lane) * (PACKED ? 128u : 144u);
        const uint32_t scales = wring + 128u * 128u + (uint32_t)lane * 16u + 4u * (uint32_t)(warp & 3);
        const uint32_t dst = acol + ((uint32_t)(32 * (warp & 3)) << 16);
        const uint32_t afull_base = cluster_addr(smem_u32(afull), 0);
        const int set = (warp - 4) >> 2;
        if (SETS == 4) decode_set<BF16, PACKED, SETS, -1>(src, scales, dst, wfull, wempty, aempty, afull_base, stages, p.nws, p.na, lane, set, at);
        if (SETS == 2 && set == 0) decode_set<BF16, PACKED, SETS, 0>(src, scales, dst, wfull, wempty, aempty, afull_base, stages, p.nws, p.na, lane, set, at);
        if (SETS == 2 && set == 1) decode_set<BF16, PACKED, SETS, 1>(src, scales, dst, wfull, wempty, aempty, afull_base, stages, p.nws, p.na, lane, set, at);
    };
    auto load_w = [&](int ws, int rt, int w) {
        if (PACKED)  // (the upper half of the last 256-row tile may lie beyond the matrix: it reads the last one, and its results are not stored)
            bulk_g2s(smem_raw + (wring - smem_u32(smem_raw)) + (uint32_t)ws * W_STAGE, p.packed + ((size_t)min(rt, p.packed_tiles - 1) * nw + w) * W_STAGE,
                     W_STAGE, &wfull[ws]);
        else
            tma_load_2d(wring + (uint32_t)ws * W_STAGE, &wmap, w * 36, rt * 128, smem_u32(&wfull[ws]));
    };
    if (BF16 && warp == 0) {
        // ------------------------------------------------------------ weights and activations in, by one thread: two of them, each as far
        // ahead as its ring allows, cost 4 - 20 % beyond 128 rows
        if (lane == 0) {
            if (!PACKED) tma_prefetch_map(&wmap);
            tma_prefetch_map(&xmap);
            int ws = 0, bs = 0;
            uint32_t wp = 1, bp = 1;  // parity of "empty": the first round passes at once
            bool ok = true;
            const uint32_t bfull0 = smem_u32(bfull) & 0xFEFFFFFFu;  // the even CTA's barriers
            for (Unit<SPLIT> u(pair, p); u.live(p) && ok; u.next(npairs, p)) {
                const int rt = (u.tile % p.row_tiles) * 2 + (int)rank, tok0 = (u.tile / p.row_tiles) * p.tn + (int)rank * (p.tn >> 1);
                const int w0 = u.first(p), w1 = w0 + u.count(p);
                for (int w = w0; w < w1 && ok; w++) {
                    if (!mbar_wait(&wempty[ws], wp)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&wfull[ws], W_STAGE);
                    mbar_arrive(&wfull[ws]);
                    load_w(ws, rt, w);
                    if (++ws == p.nws) ws = 0, wp ^= 1u;
                    for (int q = 0; q < 4 / KB; q++) {
                        if (!mbar_wait(&bempty[bs], bp)) {
                            cn_dev_fail(CN_DEV_WAIT_EMPTY);
                            ok = false;
                            break;
                        }
                        if (rank == 0) {  // the even CTA's barrier counts both halves
                            mbar_expect_tx(&bfull[bs], 2u * bslot);
                            mbar_arrive(&bfull[bs]);
                        }
                        tma_load_3d_pair(ring + (uint32_t)bs * bslot, &xmap, 0, tok0, w * 4 + KB * q, bfull0 + 8u * (uint32_t)bs);
                        if (++bs == p.nb) bs = 0, bp ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 0) {
        // ------------------------------------------------------------ f16 rows: weights in, while the kernel that prepares the activations still
        // runs. That one has waited for everything before it when it lets this one start, so weights and tensor scale are complete, also where the
        // kernel in front of the call wrote them.
        if (lane == 0) {
            if (!PACKED) tma_prefetch_map(&wmap);
            int ws = 0;
            uint32_t wp = 1;  // parity of "empty": the first round passes at once
            bool ok = true;
            for (Unit<SPLIT> u(pair, p); u.live(p) && ok; u.next(npairs, p)) {
                const int rt = (u.tile % p.row_tiles) * 2 + (int)rank, w0 = u.first(p), w1 = w0 + u.count(p);
                for (int w = w0; w < w1; w++) {
                    if (!mbar_wait(&wempty[ws], wp)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&wfull[ws], W_STAGE);
                    mbar_arrive(&wfull[ws]);
                    load_w(ws, rt, w);
                    if (++ws == p.nws) ws = 0, wp ^= 1u;
                }
            }
        }
    } else if (!BF16 && warp == 3) {
        // ------------------------------------------------------------ f16 rows: activations in
        if (lane == 0) {
            tma_prefetch_map(&xmap);
            int bs = 0;
            uint32_t bp = 1;
            bool ok = true;
            const uint32_t bfull0 = smem_u32(bfull) & 0xFEFFFFFFu;  // the even CTA's barriers
            pdl_wait();  // f16 rows come from the kernel before this one
            for (Unit<SPLIT> u(pair, p); u.live(p) && ok; u.next(npairs, p)) {
                const int tok0 = (u.tile / p.row_tiles) * p.tn + (int)rank * (p.tn >> 1), w0 = u.first(p), w1 = w0 + u.count(p);
                for (int q = w0 * (4 / KB); q < w1 * (4 / KB); q++) {
                    if (!mbar_wait(&bempty[bs], bp)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    if (rank == 0) {  // the even CTA's barrier counts both halves
                        mbar_expect_tx(&bfull[bs], 2u * bslot);
                        mbar_arrive(&bfull[bs]);
                    }
                    tma_load_3d_pair(ring + (uint32_t)bs * bslot, &xmap, 0, tok0, KB * q, bfull0 + 8u * (uint32_t)bs);
                    if (++bs == p.nb) bs = 0, bp ^= 1u;
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
            for (Unit<SPLIT> u(pair, p); u.live(p) && ok; u.next(npairs, p)) {
                if (!mbar_wait(&accempty[ab], cp)) {
                    cn_dev_fail(CN_DEV_WAIT_EMPTY);
                    break;
                }
                tc_after();
                const uint32_t d = tmem + (uint32_t)(ab * p.acc_stride);
                const int nk = 4 * u.count(p);
                for (int kb = 0; kb < nk; kb += KB) {
                    if (!mbar_wait(&bfull[bs], bp)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int h = 0; h < KB; h++) {
                        if (h % G == 0) {
                            if (!mbar_wait(&afull[as], ap)) ok = false;
                            tc_after();
                        }
                        const uint32_t a = acol + (uint32_t)as * (32u * G) + 32u * (h % G);
                        const uint64_t b = bdesc0 + (((uint32_t)bs * bslot + (uint32_t)h * bbox) >> 4);
                        if (elect_lane()) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)  // 16 values: 8 columns of A, 32 bytes of B inside the swizzled row
                                tc_mma_ts<2>(d, a + 8u * kk, b + 2u * kk, idesc, (kb > 0 || h > 0 || kk > 0) ? 1u : 0u);
                            if (h % G == G - 1) tc_commit<2>(&aempty[as]);
                            if (h == KB - 1) tc_commit<2>(&bempty[bs]);
                        }
                        __syncwarp();
                        if (h % G == G - 1 && ++as == p.na) as = 0, ap ^= 1u;
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
    } else if (SETS == 2 && warp >= 4 && warp < 12) {
        // ------------------------------------------------------------ decode
        int stages = 0;
        for (Unit<SPLIT> u(pair, p); u.live(p); u.next(npairs, p)) stages += u.count(p);
        decode(stages);
    } else if (warp >= 4) {
        // ------------------------------------------------------------ results: lane = weight row, 32 tokens per load, the two (four) warps of a
        // quarter of the rows take alternate loads
        constexpr int FIRST = SETS == 4 ? 4 : 12, STEP = SETS == 4 ? 128 : 64;
        const int quarter = warp & 3;
        const uint32_t lanes = (uint32_t)(32 * quarter) << 16;
        const uint32_t accempty_base = cluster_addr(smem_u32(accempty), 0);
        const float gs = p.gs[0] * (BF16 ? BF16_UNSCALE : F16_UNSCALE);
        const int odd = lane & 1;
        int ab = 0;
        uint32_t cp = 0;
        if (SETS == 2) pdl_wait();  // the row factors come from the kernel before this one
        for (Unit<SPLIT> u(pair, p); u.live(p); u.next(npairs, p)) {
            const int tile = u.tile;
            float* part = SPLIT && p.ksplits > 1 ? p.part + (size_t)u.split * p.m * p.rows : nullptr;
            if (SETS == 4) {
                decode(u.count(p));
                pdl_wait();
            }
            if (!mbar_wait(&accfull[ab], cp)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            tc_after();
            const int rbase = (tile % p.row_tiles) * 256 + (int)rank * 128 + 32 * quarter, row = rbase + lane, tok0 = (tile / p.row_tiles) * p.tn;
            const int live = min(p.tn, p.m - tok0);
            for (int c0 = 32 * ((warp - FIRST) >> 2); c0 < live; c0 += STEP) {
                uint32_t v[32];
                tc_ld32(tmem + lanes + (uint32_t)(ab * p.acc_stride + c0), v);
                tc_wait_ld();
                if (SPLIT && part) {
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (c0 + i < live && row < p.rows) part[(size_t)(tok0 + c0 + i) * p.rows + row] = __uint_as_float(v[i]);
                } else if (p.pair_store) {
                    // bf16 rows two at a time: lanes l, l + 1 trade so that the even one holds both rows of token c0 + i, the odd one
                    // both of token c0 + i + 1, and a warp's store is 64 contiguous bytes of each
                    __nv_bfloat16* yp = (__nv_bfloat16*)p.y + (size_t)(tok0 + c0 + odd) * p.ldy + (row & ~1);
                    const size_t step = 2 * (size_t)p.ldy;
                    const bool whole = live - c0 >= 32 && rbase + 32 <= p.rows;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float a = __uint_as_float(v[i]), b = __uint_as_float(v[i + 1]);
                        if (BF16)
                            a *= gs, b *= gs;
                        else
                            a = a * gs * p.rs[min(tok0 + c0 + i, p.m - 1)], b = b * gs * p.rs[min(tok0 + c0 + i + 1, p.m - 1)];
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
                            const float r = BF16 ? __uint_as_float(v[i]) * gs : __uint_as_float(v[i]) * gs * p.rs[tok];
                            if (p.out_bf16)
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

// Tokens per tile, and parts of K: the multiple of 32 up to 256 and the split whose units fill the pairs' rounds best. A round costs the
// longer of the MMAs (2 cycles per token and 64-value block) and the decode (about 300 cycles per block bf16, 170 f16), plus the
// epilogue where a single accumulator leaves it exposed. A split adds the partial sums' way through L2 and a kernel that adds them.
struct PairShape {
    int tn, ksplits;
};
PairShape pair_shape(int rows, int nk, int m, int pairs, bool bf16, int max_splits) {
    const int rt = (rows + 255) / 256, most = (m + 31) / 32 * 32 < 256 ? (m + 31) / 32 * 32 : 256, nw = nk / 4;
    double best = 1e30;
    PairShape r = {most, 1};
    for (int n = (m + most - 1) / most; n <= (m + 31) / 32; n++) {  // token tiles
        const int t = ((m + n - 1) / n + 31) / 32 * 32;
        const long long tiles = (long long)rt * ((m + t - 1) / t);
        const double step = 2.0 * t > (bf16 ? 300.0 : 170.0) ? 2.0 * t : (bf16 ? 300.0 : 170.0);
        const double tail = 2500.0 + 16.0 * t;
        for (int ks = 1; ks <= max_splits && (ks == 1 || ks <= nw / 2); ks++) {
            const long long rounds = (tiles * ks + pairs - 1) / pairs;
            const int blocks = 4 * ((nw + ks - 1) / ks);
            const double add = ks > 1 ? 5000.0 + (double)ks * m * rows / 300.0 : 0.0;
            const double cost = rounds * (blocks * step + (t > 192 ? tail : 400.0)) + (t > 192 ? 0.0 : tail) + add;
            if (cost < best) best = cost, r = {t, ks};
        }
        if (t <= 64) break;
    }
    return r;
}

// y[t][n] = (sum over splits, in order, of part[s][t][n]) * f * gs * rs[t], four outputs per thread where rows and results allow it
template <int V>
__global__ void gemm_splitk_reduce_kernel(const float* __restrict__ part, const float* __restrict__ gs, const float* __restrict__ rs, float f, void* __restrict__ y,
                                          int rows, int m, int ldy, int ksplits, int out_bf16) {
    const int n = (blockIdx.x * blockDim.x + threadIdx.x) * V, t = blockIdx.y;
    pdl_launch_dependents();
    pdl_wait();
    if (n >= rows) return;
    float v[V];
    auto load = [&](int s, float* o) {
        const float* q = part + ((size_t)s * m + t) * rows + n;
        if constexpr (V == 4)
            *(float4*)o = __ldcg((const float4*)q);
        else
            o[0] = __ldcg(q);
    };
    load(0, v);
    for (int s = 1; s < ksplits; s++) {
        float a[V];
        load(s, a);
#pragma unroll
        for (int i = 0; i < V; i++) v[i] += a[i];
    }
    const float c = gs[0] * f, r = rs ? rs[t] : 1.0f;
#pragma unroll
    for (int i = 0; i < V; i++) v[i] = v[i] * c * r;
    if (out_bf16) {
        __nv_bfloat16* o = (__nv_bfloat16*)y + (size_t)t * ldy + n;
        if constexpr (V == 4) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
            *(uint2*)o = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
        } else {
            *o = __float2bfloat16_rn(v[0]);
        }
    } else {
        float* o = (float*)y + (size_t)t * ldy + n;
        if constexpr (V == 4)
            *(float4*)o = *(float4*)v;
        else
            *o = v[0];
    }
}

template <bool BF16, bool PACKED, int SETS, bool SPLIT>
int launch_pair(const CUtensorMap& wmap, const CUtensorMap& xmap, const PairParams& p, int grid, size_t smem, bool after, cudaStream_t stream) {
    auto kern = nvfp4_gemm_pair_kernel<BF16, PACKED, SETS, SPLIT>;
    CN_ALLOW_SMEM(kern, SMEM_MAX);
    if (after)
        CN_CUDA(cn_launch_pdl(kern, dim3((unsigned)grid), dim3(PAIR_THREADS), smem, stream, wmap, xmap, p));
    else
        kern<<<grid, PAIR_THREADS, smem, stream>>>(wmap, xmap, p);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

constexpr int PAIRS = 74;

}  // namespace

int cn_gemm_pair_splits(int rows, int k, int m, bool x_f16, int max_splits) { return pair_shape(rows, k / 64, m, PAIRS, !x_f16, max_splits).ksplits; }

int cn_gemm_pair_launch(const GemmCall& c, cudaStream_t stream) {
    CUtensorMap wmap = {}, xmap;
    const int nk = c.k / 64;
    PairParams p = {};
    p.gs = c.gs, p.rs = c.x_f16 ? c.rs : nullptr, p.y = c.y, p.rows = c.rows, p.m = c.m, p.ldy = c.ldy, p.nk = nk, p.out_bf16 = c.out_bf16;
    p.pair_store = c.out_bf16 && !((c.rows | c.ldy) & 1) && !((uintptr_t)c.y & 3);
    p.packed = (const uint8_t*)c.packed, p.packed_tiles = (c.rows + 127) / 128, p.part = c.part;
    const PairShape shape = pair_shape(c.rows, nk, c.m, PAIRS, !c.x_f16, c.part ? c.max_splits : 1);
    p.tn = shape.tn, p.ksplits = shape.ksplits, p.split_stages = nk / 4 / shape.ksplits, p.split_more = nk / 4 % shape.ksplits;
    const bool four = c.x_f16 && p.tn <= 128;
    const int slot = slot_blocks(four ? 4 : 2), box = box_blocks(four ? 4 : 2);
    p.acc_stride = p.tn;
    p.nacc = p.tn <= 192 && !four ? 2 : 1;  // (the warps that decode write the results too: a second accumulator would have no one to fill its A slots meanwhile)
    p.na = (TMEM_COLS - p.nacc * p.acc_stride) / (32 * slot);
    p.na = p.na > 8 ? 8 : four ? p.na : p.na & ~1;
    const int bslot = p.tn * 64 * box;
    p.nb = (SMEM_MAX - HDR - 1024 - 3 * W_STAGE) / bslot;
    if (p.nb > 16 / box) p.nb = 16 / box;
    p.nws = (SMEM_MAX - HDR - 1024 - p.nb * bslot) / W_STAGE;
    if (p.nws > MAX_W_STAGES) p.nws = MAX_W_STAGES;
    p.row_tiles = (c.rows + 255) / 256;
    p.tiles = p.row_tiles * ((c.m + p.tn - 1) / p.tn);
    if (!c.packed)
        if (int rc = cn_tmap_words(&wmap, c.w, (unsigned long long)nk * 9, c.rows, 36, 128)) return rc;
    if (int rc = cn_tmap_blocks(&xmap, c.x, !c.x_f16, nk, c.m, (unsigned long long)c.k * 2, p.tn / 2, box)) return rc;
    const size_t smem = HDR + 1024 + (size_t)p.nws * W_STAGE + (size_t)p.nb * bslot;
    const int units = p.tiles * p.ksplits, grid = 2 * (units < PAIRS ? units : PAIRS);
    int rc = CN_ERR_SHAPE;
#define CN_PAIR_CASE(BF16V, PACKEDV, SETSV, SPLITV)                                                                                       \
    if (!c.x_f16 == BF16V && (c.packed != nullptr) == PACKEDV && four == (SETSV == 4) && (c.x_f16 || p.ksplits > 1) == SPLITV)             \
        rc = launch_pair<BF16V, PACKEDV, SETSV, SPLITV>(wmap, xmap, p, grid, smem, c.x_f16, stream);
    CN_PAIR_CASE(true, false, 2, false) CN_PAIR_CASE(true, false, 2, true) CN_PAIR_CASE(false, false, 2, true) CN_PAIR_CASE(false, false, 4, true)
    CN_PAIR_CASE(true, true, 2, false) CN_PAIR_CASE(true, true, 2, true) CN_PAIR_CASE(false, true, 4, true)
#undef CN_PAIR_CASE
    if (rc || p.ksplits == 1) return rc;
    const float f = c.x_f16 ? F16_UNSCALE : BF16_UNSCALE;
    const bool wide = !((c.rows | c.ldy) & 3) && !((uintptr_t)c.y & 15);
    if (wide)
        CN_CUDA(cn_launch_pdl(gemm_splitk_reduce_kernel<4>, dim3((unsigned)((c.rows / 4 + 127) / 128), (unsigned)c.m), dim3(128), 0, stream, p.part, c.gs, p.rs, f, c.y,
                              c.rows, c.m, c.ldy, p.ksplits, c.out_bf16));
    else
        CN_CUDA(cn_launch_pdl(gemm_splitk_reduce_kernel<1>, dim3((unsigned)((c.rows + 127) / 128), (unsigned)c.m), dim3(128), 0, stream, p.part, c.gs, p.rs, f, c.y,
                              c.rows, c.m, c.ldy, p.ksplits, c.out_bf16));
    return CN_OK;
}
