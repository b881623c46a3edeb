// NVFP4 GEMV for 1..8 bf16 or f32 activation rows on the fifth-generation tensor cores (tcgen05.mma kind::mxf4nvf4, block scale): plain and gate / up form, with or without
// the tensor-parallel line output (bf16). Supersedes gemv_nvfp4_w / _gu / _wm / _gum (engine/src/kernels_p2.rs:355-530).
//
// The weights are the A operand as they are: E2M1 codes with one UE4M3 scale per 16 values is what this MMA multiplies, so nothing is decoded. A bf16
// row is the B operand as eight columns of signed octal digits, an f32 row as eleven: per 16 values a power of two and a number of 23 (32) bits, digit j of a value being one
// of -4..3, all of them E2M1 values (what they hold of a value, and the blocks that are multiplied out instead: nvfp4_digits.cuh).
// Products, scales and digits are exact; a column's sum over 256 values is the tensor core's, which is the f32 nearest to it or the one beside (k = 256:
// 2.5e-8 of a row against 64 bits, as much as the last rounding alone). The columns are added from the smallest up and the chunks of 256 in order; bf16 rows in f32
// (k = 4096: 6.2e-8, 17408: 8.6e-8), f32 rows with what the last two additions round off kept, chunks in 64 bits (2.5e-8: the result's own rounding). The columns of one row do not
// depend on those of another: a row of an m-row call has the bits of a one-row call, and eight rows (64 or 96 columns) take the tensor core little longer than one, which is bound by
// reading A.
//
// A CTA owns 128 rows (64 of gate and 64 of up) over a part of k; a cluster of C CTAs shares the tile, part by part, and every CTA adds and stores
// 128 / C of its rows, the parts in order. Warps: 0-3 add up and store (a thread is a row), 4-7 move container blocks (36 bytes): codes into
// tensor memory, scales into the chunks that are copied there; 8-11 turn activations into digits, 12 loads (TMA, boxes of 128 rows x 144 bytes of container), 13 issues the MMAs. Loads and the move do
// not wait for the kernel in front: when the activations come, six chunks of weights a CTA lie ready or nearly so.
//
// What bounds it, one row: HBM for large matrices (gate / up of 17408 x 5120: 100 MB in 17.4 us, of which 2.6 until the first product);
// for small ones the chain from one call to the next, some 3 us: end of the grid in front 0.8, activations 0.4, digits 0.35, first sum 0.4, adding up in
// the cluster 0.4, output and end of the grid 0.6. From four rows on also the digits (one warp and row: 0.35 us a chunk). In a stream of dependent calls, us
// here / mma.sync kernel (nvfp4_gemv_m1.cu): gate / up of 17408 x 5120 17.4 / 20.7, two rows 17.7 / 27.3, four 21.5 / 30.1, eight 30.7 / 46.5; 5120 x 17408
// 10.7 / 15.5, 11.4 / 18.5, 14.0 / 21.1, 19.2 / 34.7; 25000 x 8192 19.5 / 28.2, four rows 25.0 / 32.0. f32 rows, here / mma.sync with three f16 planes a row: gate / up of
// 17408 x 5120 17.7 / 26.7, 19.0 / 39.8, 29.0 / 41.2, 49.3 / 85; 5120 x 17408 11.1 / 22.1, 12.7 / 38, 18.2 / 62, 29.2 / 122.
// Measured and not kept: a fifth container stage (the same); weight and activation warps on schedulers of their own (4096 x 4096 4.7 -> 4.9); and, while the operand lay in shared memory: tiles of fewer rows so that every SM has the same bytes (the CTAs more hold up the next kernel: 5120 x 5120 5.9 -> 6.9); two teams of
// warps for the move (18.6 -> 20.0, gate / up); L2 prefetches beyond the stages (18.6 -> 19.3 and more); a third operand stage in a container stage's place (20.6).
#include "nvfp4_digits.cuh"
#include "nvfp4_gemv.cuh"

#include <atomic>
#include <type_traits>

namespace {

constexpr int CH = 256;                                       // values of k in a chunk: four MMAs
constexpr int RAW_STAGE = 128 * 144;                          // container bytes of a chunk
constexpr int NX = 16;      // chunk factors in flight (a warp is at most a few chunks ahead of another)
constexpr int NDONE = 4;    // barriers of finished chunks
constexpr int MAX_RAW = 4;  // container stages
constexpr int NA = 2;       // chunks laid out for the tensor core
constexpr int NSLOT = 3;    // tiles whose sums are on their way in a cluster
constexpr int NBAR = 2 * MAX_RAW + NA + NX + NDONE + NSLOT + 2;
constexpr int EPI_WARPS = 4, LOADER = 12, ISSUER = 13;  // warps 0-3 sums and output, 4-7 weights, 8-11 activations
constexpr int THREADS = 448;
constexpr int FS_OFF = 512, WF_OFF = 1536, HEADER = 2048;  // barriers; chunk factors [NX][8] {factor, blocks without digits}; [NX][4] scale bytes of 0xFF seen
__host__ __device__ constexpr int ncol(int mt, bool f32) { return (mt * digits_of(f32) + 15) / 16 * 16; }  // columns of the MMA
__host__ __device__ constexpr int b_codes(int mt, bool f32) { return ncol(mt, f32) * 128; }
__host__ __device__ constexpr int b_stage(int mt, bool f32) { return b_codes(mt, f32) + 4 * 512; }
// chunks of digits (us with two / four: four rows of gate / up 17408 x 5120 22.0 / 21.6, eight 31.6 / 30.7). They leave room for three container stages or four, but for two where eight rows of either type
// have the sums of three tiles on their way
__host__ __device__ constexpr int nb_of(int mt, bool f32) { return mt == 8 && f32 ? 2 : 4; }
// accumulators, in half of an SM's tensor memory beside the codes of two chunks and the scales: those of two chunks where they fit (all but eight f32 rows)
constexpr int TMEM = 256, TM_FIXED = NA * A_COLS + 64;
__host__ __device__ constexpr int nacc(int mt, bool f32) { return 2 * ncol(mt, f32) + TM_FIXED <= TMEM ? 2 : 1; }
__host__ __device__ constexpr int fixed_smem(int mt, bool f32) { return HEADER + 1024 + NA * A_SCALES + nb_of(mt, f32) * b_stage(mt, f32); }

struct TcParams {
    const uint8_t* w0;
    const uint8_t* w1;  // gate / up: up
    const float* gs0;
    const float* gs1;
    const void* x;
    void* y;
    int rows, k, m, ldy, out_f32;
    float limit;
    uint32_t qinv;                 // 2^20 / share, rounded up: idx / share for idx < 1024
    int ex_bytes;                  // a slot of sums handed over
    int csize, tiles, raw, share;  // CTAs per cluster, row tiles, container stages, rows (or pairs) of a tile that a CTA stores
    unsigned long long yl[8];
    int yl_world, yl_row0;
    unsigned long long yl_stride;
    const unsigned int* yl_epoch;
    int yl_tag, yl_buf, yl_flip;
#ifdef CN_M1_TRACE
    unsigned long long* trace;  // [8] globaltimer stamps per CTA of this launch, or null
#endif
};

// Diagnostic build (-DCN_M1_TRACE): the stamps of nvfp4_gemv_m1.cu, by a lane each: entry (0), wait on the predecessor over (1), first digits (2), first chunk laid
// out (3), sums stored (4), first (5) and last (6) load asked for.
#ifdef CN_M1_TRACE
__device__ __forceinline__ unsigned long long gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define CN_STAMP(i) \
    if (p.trace && lane == 0) p.trace[(size_t)blockIdx.x * 8 + (i)] = gtime()
#else
#define CN_STAMP(i)
#endif

__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst), "l"(m),
        "r"(x), "r"(y), "r"(bar), "l"(policy)
        : "memory");
}
// a value into another CTA's shared memory, counted there on a barrier of the same CTA
__device__ __forceinline__ void st_async_f32(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) { st_async_f32(addr, v, bar); }
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity) {  // bounded, with cluster-scope acquire
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > 2000000000LL) return false;
    }
}

template <int MT, bool F32>
__global__ void __launch_bounds__(THREADS, 2) nvfp4_gemv_tc_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                                                                   const TcParams p) {
    constexpr int LV = digits_of(F32), ES = F32 ? 4 : 2;
    constexpr int N = ncol(MT, F32), NB = nb_of(MT, F32), B_STAGE = b_stage(MT, F32), B_CODES = b_codes(MT, F32);
    using Acc = typename std::conditional<F32, double, float>::type;
    constexpr int NACC = nacc(MT, F32);
    constexpr uint32_t IDESC = idesc_bs(N), SFA_COL = NACC * N, SFB_COL = NACC * N + 32, A_COL = NACC * N + 64;
    static_assert(NACC * N + TM_FIXED <= TMEM, "tensor memory columns");
    extern __shared__ uint8_t smem[];
    uint64_t* raw_full = (uint64_t*)smem;
    uint64_t* raw_empty = raw_full + MAX_RAW;
    uint64_t* a_full = raw_empty + MAX_RAW;   // [NA]
    uint64_t* xbar = a_full + NA;            // [NX] digits of a chunk, and its accumulators (those of two chunks before) have been read
    uint64_t* done = xbar + NX;               // [NDONE] MMAs of a chunk; the issuer arrives too, and hands on what weight and activation warps wrote beside the operands
    uint64_t* exbar = done + NDONE;           // [NSLOT] sums handed over
    uint64_t* meet = exbar + NSLOT;           // [2] the four adding warps, tile by tile: its sums are in the slot (one CTA), have been read from it (cluster)
    uint32_t* tmem_slot = (uint32_t*)(meet + 2);
    float2* fs = (float2*)(smem + FS_OFF);    // [NX][8]
    uint32_t* wf = (uint32_t*)(smem + WF_OFF);  // [NX][4]
    const uint32_t base = (smem_u32(smem) + HEADER + 1023u) & ~1023u;
    uint8_t* a0 = smem + (base - smem_u32(smem));
    uint8_t* b0 = a0 + NA * A_SCALES;
    uint8_t* r0 = b0 + NB * B_STAGE;
    const int R = p.raw;
    uint8_t* ex = r0 + (size_t)R * RAW_STAGE;
    const int tid = threadIdx.x, warp = (int)warp_uniform((uint32_t)tid >> 5), lane = tid & 31;
    const int C = p.csize, rank = C > 1 ? (int)cluster_rank() : 0;
    const int cid = (int)blockIdx.x / C, ncl = (int)gridDim.x / C;
    const int nk = p.k / CH, ck0 = rank * nk / C, nc = (rank + 1) * nk / C - ck0;
    const int ntl = (p.tiles - cid + ncl - 1) / ncl, total = ntl * nc;
    const bool gu = p.w1 != nullptr;
    const int per_tile = gu ? 64 : 128;

    auto load = [&](int s, int tile, int chunk, uint64_t pol) {
        mbar_expect_tx(&raw_full[s], RAW_STAGE);
        mbar_arrive(&raw_full[s]);
        const uint32_t dst = smem_u32(r0) + (uint32_t)(s * RAW_STAGE), bar = smem_u32(&raw_full[s]);
        tma_load_2d_hint(dst, &map0, chunk * 36, tile * per_tile, bar, pol);
        if (gu) tma_load_2d_hint(dst + RAW_STAGE / 2, &map1, chunk * 36, tile * per_tile, bar, pol);
    };
    if (warp == 0) { CN_STAMP(0); }
    if (warp == LOADER) {
        // a barrier a lane: container stages, operand stages, digits and accumulators, finished chunks, sums handed over
        for (int i = lane; i < NBAR; i += 32)
            mbar_init(raw_full + i, i < MAX_RAW                         ? 1
                                    : i < 2 * MAX_RAW + NA              ? 4
                                    : i < 2 * MAX_RAW + NA + NX         ? (MT < 4 ? MT : 4) + EPI_WARPS
                                    : i < 2 * MAX_RAW + NA + NX + NDONE ? 2
                                    : i < NBAR - 2                      ? 1
                                                                        : EPI_WARPS);
        mbar_fence_init();
        __syncwarp();
        if (lane == 0) {
            // the weights do not depend on the kernel in front: the first stages are asked for at once
            const uint64_t pol = l2_policy_evict_first();
            CN_STAMP(5);
            for (int i = 0, tile = cid, c = 0; i < R && i < total; i++) {
                load(i, tile, ck0 + c, pol);
                if (++c == nc) c = 0, tile += ncl;
            }
        }
        __syncwarp();
    } else if (warp == ISSUER) {
        tc_alloc<1>(tmem_slot, TMEM);
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    if (C > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");

    if (warp == LOADER) {
        // ------------------------------------------------------------ loads
        if (lane == 0) {
            const uint64_t pol = l2_policy_evict_first();
            int s = 0, tile = cid, c = 0;
            uint32_t par = 1;
            for (int i = 0; i < total; i++) {
                if (i >= R) {
                    if (!mbar_wait(&raw_empty[s], par)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        for (int j = 0; j < R; j++) mbar_wait(&raw_full[j], ((uint32_t)((i - 1 - j) / R)) & 1u);  // copies in flight
                        break;
                    }
                    load(s, tile, ck0 + c, pol);
                }
                // The next kernel may start when only three loads of this one are left: its weights then stream while this one drains. Earlier, its first
                // loads would hold up the last ones here (16384 x 2048: 6.9 us a call, 5.6 so; 4096 x 8192 7.5 and 6.3; behind the last load 6.1 and 6.4).
                // (Behind the allocation in any case: a kernel that starts early finds this one's tensor memory taken.)
                if (i == max(total - 3, 0)) pdl_launch_dependents();
                if (++c == nc) c = 0, tile += ncl;
                if (++s == R) s = 0, par ^= 1u;
            }
            CN_STAMP(6);
        }
        __syncwarp();
    } else if (warp == ISSUER) {
        // ------------------------------------------------------------ scale copies and MMAs
        const uint32_t a_u = warp_uniform(smem_u32(a0)), b_u = warp_uniform(smem_u32(b0));
        for (int i = 0; i < total; i++) {
            const int a = i & 1, b = i % NB;
            if (!mbar_wait(&a_full[a], (i >> 1) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            tc_after();
            const uint64_t db = tc_desc_sw128(b_u + (uint32_t)(b * B_STAGE));
            const uint64_t sa = desc_sf(a_u + (uint32_t)(a * A_SCALES)), sb = desc_sf(b_u + (uint32_t)(b * B_STAGE + B_CODES));
            const uint32_t ta = tmem + SFA_COL + 16 * a, tb = tmem + SFB_COL + 16 * a, td = tmem + N * (i % NACC);
            if (elect_lane()) {
#pragma unroll
                for (int j = 0; j < 4; j++) cp_sf(ta + 4 * j, sa + 32 * j);
            }
            __syncwarp();
            if (!mbar_wait(&xbar[i % NX], (i / NX) & 1)) {  // (one wait for both: each costs the issuer some 75 cycles, passed or not)
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            tc_after();
            if (elect_lane()) {
#pragma unroll
                for (int j = 0; j < 4; j++) cp_sf(tb + 4 * j, sb + 32 * j);
#pragma unroll
                for (int j = 0; j < 4; j++) umma_bs(td, tmem + A_COL + A_COLS * a + 8 * j, db + 2 * j, IDESC, ta + 4 * j, tb + 4 * j, j > 0 ? 1u : 0u);
                tc_commit<1>(&done[i % NDONE]);
                mbar_arrive(&done[i % NDONE]);
            }
            __syncwarp();
        }
    } else if (warp >= 8) {
        // ------------------------------------------------------------ activations -> digits: a warp takes whole rows of a chunk
        constexpr int CPR = MT < 4 ? 4 / MT : 1;  // chunks side by side in the four warps
        constexpr int TPW = MT > 4 ? MT / 4 : 1;  // rows of a warp
        const int w = warp - 8, myrow = MT < 4 ? w % MT : w, mychunk = MT < 4 ? w / MT : 0;
        pdl_wait();  // the activations may come from the kernel before this one
        if (w == 0) { CN_STAMP(1); }
        constexpr int XR = F32 ? 2 : 1;           // 16-byte pieces of a lane's eight values
        uint4 nx[TPW][XR];
        int c = mychunk % nc;
        auto fetch = [&]() {
#pragma unroll
            for (int t = 0; t < TPW; t++) {
                const int row = myrow + 4 * t;
#pragma unroll
                for (int q = 0; q < XR; q++) {
                    nx[t][q] = make_uint4(0u, 0u, 0u, 0u);
                    if (row < p.m) nx[t][q] = __ldcg((const uint4*)((const char*)p.x + ((size_t)row * p.k + (size_t)(ck0 + c) * CH) * ES) + lane * XR + q);
                }
            }
            c += CPR;
            while (c >= nc) c -= nc;
        };
        fetch();
        for (int i = mychunk; i < total; i += CPR) {
            uint4 now[TPW][XR];
#pragma unroll
            for (int t = 0; t < TPW; t++)
#pragma unroll
                for (int q = 0; q < XR; q++) now[t][q] = nx[t][q];
            fetch();
            if (i >= NB && !mbar_wait(&done[(i - NB) % NDONE], ((i - NB) / NDONE) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                break;
            }
            uint8_t* bs = b0 + (i % NB) * B_STAGE;
#pragma unroll
            for (int t = 0; t < TPW; t++) {
                const int row = myrow + 4 * t;  // (beyond p.m: zeros, in columns that nothing reads)
                to_digits<F32>(now[t], lane, bs, bs + B_CODES, row, &fs[(i % NX) * 8 + row]);
            }
            fence_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&xbar[i % NX]);
            if (i == 0) { CN_STAMP(2); }
        }
    } else if (warp >= EPI_WARPS) {
        // ------------------------------------------------------------ container blocks -> operand layout: a warp takes 32 rows, a lane the four
        // blocks of a row (144 bytes: no bank twice among eight lanes)
        const int w = warp - 4;
        int s = 0;
        uint32_t par = 0;
        for (int i = 0; i < total; i++) {
            if (!mbar_wait(&raw_full[s], par)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            const uint4* src = (const uint4*)(r0 + (size_t)s * RAW_STAGE) + (w * 32 + lane) * 9;
            uint32_t v[36];
            const uint32_t odd = load_row(src, v);
            if (i >= NA && !mbar_wait(&done[(i - NA) % NDONE], ((i - NA) / NDONE) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                break;
            }
            store_row(tmem + A_COL + A_COLS * (i & 1), a0 + (i & 1) * A_SCALES, w, lane, v);
            if (lane == 0) wf[(i % NX) * 4 + w] = odd;
            fence_async();
            __syncwarp();
            // (the stage is given back here and not behind the loads: an arrival can overtake loads whose values nothing has used yet)
            if (lane < 2) mbar_arrive(lane == 0 ? &a_full[i & 1] : &raw_empty[s]);
            if (w == 0 && i == 0) { CN_STAMP(3); }
            if (++s == R) s = 0, par ^= 1u;
        }
    } else {
        // ------------------------------------------------------------ sums and output
        if (lane < NACC) mbar_arrive(&xbar[lane]);  // the accumulators of the first two chunks
        pdl_wait();
        const float gs0 = *p.gs0, gs1 = gu ? *p.gs1 : 0.0f, gs = gu && warp >= 2 ? gs1 : gs0;
        const unsigned int epoch = p.yl_world > 0 ? *(volatile const unsigned int*)p.yl_epoch : 0u;
        const int r = warp * 32 + lane;  // this thread's row of the tile
        Acc acc[MT];  // f32 rows: without the tensor scale
#pragma unroll
        for (int m = 0; m < MT; m++) acc[m] = 0;
        bool met = C == 1;
        int c = 0, tile = cid, nt = 0;
        for (int i = 0; i < total; i++) {
            if (!mbar_wait(&done[i % NDONE], (i / NDONE) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            tc_after();
            const uint32_t td = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(N * (i % NACC));
            const uint32_t odd = wf[(i % NX) * 4 + warp];
            uint32_t slow = odd;
            constexpr int G = MT < 4 ? MT : F32 && MT == 4 ? 2 : 1;  // rows at a time (eight bf16 rows of gate / up 17408 x 5120: four 32.7 us, two 32.4, one 31.6; four rows: four 21.6, one 21.5)
#pragma unroll
            for (int m0 = 0; m0 < MT; m0 += G) {
                uint32_t d[G * LV];
#pragma unroll
                for (int m = 0; m < G; m++) tc_ld_digits<F32>(td + LV * (m0 + m), d + LV * m);
                tc_wait_ld();
                if (m0 + G == MT) {
                    tc_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&xbar[(i + NACC) % NX]);
                }
#pragma unroll
                for (int m = 0; m < G; m++) {
                    const float2 f = fs[(i % NX) * 8 + m0 + m];
                    float rest;
                    const float s = sum_digits<F32>(d + LV * m, rest);
                    if constexpr (F32)
                        acc[m0 + m] += ((double)s + (double)rest) * power_of_two(f.x);  // the chunks are added in 64 bits
                    else
                        acc[m0 + m] = fmaf(s * gs, f.x, acc[m0 + m]);
                    slow |= __float_as_uint(f.y);
                }
            }
            if (slow) {
                const int row = tile * per_tile + (gu ? r & 63 : r);
                if (row < p.rows) {
                    const uint8_t* wr = (gu && r >= 64 ? p.w1 : p.w0) + ((size_t)row * nk + ck0 + c) * 144;
#pragma unroll 1
                    for (int m = 0; m < p.m; m++) {
                        const uint32_t blocks = __float_as_uint(fs[(i % NX) * 8 + m].y);
                        if (!(blocks | odd)) continue;
                        Acc v = whole_blocks<F32>(wr, blocks, odd != 0u, (const char*)p.x + ((size_t)m * p.k + (size_t)(ck0 + c) * CH) * ES);
                        if (!F32) v *= gs;
#pragma unroll
                        for (int j = 0; j < MT; j++)
                            if (j == m) acc[j] += v;
                    }
                }
            }
            if (++c < nc) continue;
            // the tile's last chunk of this part
            if (C == 1 && !gu && p.yl_world == 0) {
                const int row = tile * 128 + r;
#pragma unroll
                for (int m = 0; m < MT; m++)
                    if (row < p.rows && m < p.m) {
                        if (F32)
                            ((float*)p.y)[(size_t)m * p.ldy + row] = (float)(acc[m] * gs);
                        else if (p.out_f32)
                            ((float*)p.y)[(size_t)m * p.ldy + row] = acc[m];
                        else
                            ((__nv_bfloat16*)p.y)[(size_t)m * p.ldy + row] = __float2bfloat16_rn(acc[m]);
                    }
            } else {
                // CTA o of the cluster adds and stores the rows (pairs) [o, o + 1) x share of the tile. Three slots in turn. Whoever sends tile n has all of tile n - 1; every CTA owns
                // rows, so a part of that came from every CTA, and from a warp that sent it only when all four adding warps of its CTA had read tile n - 3 (`meet`),
                // which had the slot before.
                const int q = p.share, half = gu ? r >> 6 : 0, at = gu ? r & 63 : r, o = at / q, halves = gu ? 2 : 1;
                const int turn = nt % NSLOT;
                Acc* slot = (Acc*)(ex + turn * p.ex_bytes);
                Acc* mine = slot + (size_t)((rank * halves + half) * MT) * q + (at - o * q);
                if (C == 1) {
#pragma unroll
                    for (int m = 0; m < MT; m++) mine[m * q] = acc[m];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&meet[nt & 1]);
                    if (!mbar_wait(&meet[nt & 1], (nt >> 1) & 1)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        break;
                    }
                } else {
                    if (!met) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // every CTA of the cluster has its barriers
                    met = true;
                    if (nt > 1 && ntl > NSLOT && !mbar_wait(&meet[nt & 1], ((nt - 2) >> 1) & 1)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        break;
                    }
                    const uint32_t there = cluster_addr(smem_u32(mine), (uint32_t)o), bar = cluster_addr(smem_u32(&exbar[turn]), (uint32_t)o);
#pragma unroll
                    for (int m = 0; m < MT; m++)
                        if (m < p.m) st_async(there + (uint32_t)(m * q * (int)sizeof(Acc)), acc[m], bar);
                    if (r == 0) {
                        mbar_expect_tx(&exbar[turn], (uint32_t)(C * halves * p.m * (int)sizeof(Acc) * max(0, min(q, per_tile - rank * q))));
                        mbar_arrive(&exbar[turn]);
                    }
                    if (!wait_cluster(&exbar[turn], (uint32_t)(nt / NSLOT) & 1u)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        break;
                    }
                }
                const int first = rank * q, have = min(q, per_tile - first);
                for (int idx0 = 0; idx0 < q * p.m; idx0 += 128) {
                    const int idx = idx0 + r, m = MT == 1 ? 0 : (int)(((uint32_t)idx * p.qinv) >> 20), lp = idx - m * q, row = tile * per_tile + first + lp;
                    const bool live = m < p.m && lp < have && row < p.rows;
                    float v = 0.0f;
                    if (live) {
                        const Acc* from = slot + m * q + lp;
                        const int step = halves * MT * q;
                        auto add_up = [&](const Acc* at0, float scale) -> float {
                            Acc part[8];
#pragma unroll
                            for (int src = 0; src < 8; src++) part[src] = src < C ? at0[src * step] : (Acc)0;
                            Acc sum = part[0];
#pragma unroll
                            for (int src = 1; src < 8; src++)
                                if (src < C) sum += part[src];
                            return F32 ? (float)(sum * scale) : (float)sum;
                        };
                        v = add_up(from, gs0);
                        const float v1 = gu ? add_up(from + MT * q, gs1) : 0.0f;
                        if (gu) v = act_gu(v, v1, p.limit);
                        if (F32 || p.out_f32)
                            ((float*)p.y)[(size_t)m * p.ldy + row] = v;
                        else
                            ((__nv_bfloat16*)p.y)[(size_t)m * p.ldy + row] = __float2bfloat16_rn(v);
                    }
                    if (MT == 1 && !F32 && p.yl_world > 0) {
                        // four rows are one 16-byte line {rows 0-1, number, rows 2-3, number} in every peer's line buffer: plain stores, the receiver polls the number
                        const uint32_t bits = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
                        const uint32_t pair = bits | (__shfl_down_sync(0xffffffffu, bits, 1) << 16), next = __shfl_down_sync(0xffffffffu, pair, 2);
                        const unsigned int seq = epoch * 4096u + (unsigned int)p.yl_tag, buf = (unsigned int)p.yl_buf ^ ((unsigned int)p.yl_flip & epoch & 1u);
                        if (live && (lane & 3) == 0)
                            for (int dst = 0; dst < p.yl_world; dst++)
                                if (p.yl[dst] != 0ull) {
                                    uint4* line = (uint4*)(uintptr_t)(p.yl[dst] + (unsigned long long)buf * p.yl_stride) + ((p.yl_row0 + row) >> 2);
                                    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(line), "r"(pair), "r"(seq), "r"(next), "r"(seq) : "memory");
                                }
                    }
                }
                if (C > 1 && ntl > NSLOT) {
                    __syncwarp();  // every lane has read the slot
                    if (lane == 0) mbar_arrive(&meet[nt & 1]);
                }
            }
#pragma unroll
            for (int m = 0; m < MT; m++) acc[m] = 0;
            c = 0, tile += ncl, nt++;
        }
        tc_before();
        if (warp == 0) { CN_STAMP(4); }
        if (C > 1) {
            // A CTA that has had every sum sent to it may leave: nothing more comes. One that gave up waits for the others.
            if (!met) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
            if (nt < ntl) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    if (C > 1 && warp >= EPI_WARPS) {
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    }
    __syncthreads();
    if (warp == ISSUER) tc_dealloc<1>(tmem, TMEM);
}

// ---------------------------------------------------------------- launch
constexpr int SM_SHARE = (227 * 1024) / 2 - 1024;  // two CTAs per SM
// (asked of a kernel of the same size without tensor memory: for one with it the runtime answers one CTA per SM, whatever its size)
__global__ void __launch_bounds__(THREADS, 2) occupancy_kernel(int* out) {
    extern __shared__ uint8_t smem[];
    if (out) out[0] = smem[threadIdx.x];
}

// clusters of c CTAs that the current device holds at a time, two CTAs per SM: asked once per device (0: an error). How many are launched, and nothing else.
int clusters_of(int c) {
    static std::atomic<int> known[64][9];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    int n = dev < 64 ? known[dev][c].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        if (cn_allow_smem((const void*)occupancy_kernel, SM_SHARE) != cudaSuccess) return 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(c * 512)), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = SM_SHARE;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)c, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
        cfg.attrs = at, cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, occupancy_kernel, &cfg) != cudaSuccess || n < 1) return 0;
        if (dev < 64) known[dev][c].store(n, std::memory_order_relaxed);
    }
    return n;
}

// CTAs per cluster, a rule of the matrix alone, since it fixes the order of a row's sum: the least estimate of the time. Neither the device nor the number of rows has a part in it: the
// clusters that are there at a time are what any B200 holds (parts differ by a few with the way their SMs lie in GPCs; one with more starts more, one with fewer takes a round more).
// A chunk takes a CTA 0.41 us, 0.68 from the tenth on (what lies ready when the activations come is gone by then), more where all CTAs together reach the memory's rate: 0.0032
// for each of them, and 0.92 late in a launch of two to an SM. Without clusters an SM with two CTAs needs 0.86 for a chunk of either however many other SMs have one, and the last
// round counts in full and more. The chunks are otherwise nearer to the mean than to those of the busiest CTA; 0.62 for adding up a tile in a cluster and 0.026 for each of its CTAs. The figures are those that
// made the picks for 130 matrices, each timed with every cut, lose least (1 percent on average; 22 for the estimate that stood here before, which had a matrix of 152 tiles as 152 CTAs on 148 SMs).
// They were taken while the operand
// lay in shared memory; with the codes in tensor memory the picks lose 1.6 percent on average over 33 matrices and one, two and four rows (most: 10240 x 8192 10, one row of 4096 x 14336 9), and stay, since they are
// the order of sums. Measured, us of one row with 1 / 2 / 4 / 6 / 8 CTAs: 16384 x 2048 5.1 / 6.0 / 6.6 / 8.0 / 8.3, 7168 x 5120 9.4 / 6.4 / 6.6 / 7.2 / 7.7, 5120 x 17408 27.7 / 15.6 / 11.7 / 10.8 / 11.3, gate / up of
// 17408 x 5120 17.6 / 17.4 / 17.7 / 19.9 / 22.4, of 9728 x 5120 13.0 / 13.0 / 11.5 / 13.2 / 15.0, of 12288 x 4096 11.6 / 11.8 / 11.8 / 13.8 / 14.4, of 20480 x 2048 10.6 / 10.3 / 12.3. 3, 5 and 7 never were the fastest.
int cut_of(int tiles, int nk) {
    constexpr int AT_ONCE[9] = {0, 296, 148, 0, 70, 0, 46, 0, 32};
    int best_c = 1;
    double best = 1e30;
    for (int c = 1; c <= 8 && c <= nk; c += c == 1 ? 1 : 2) {
        const int n = AT_ONCE[c], used = tiles < n ? tiles : n, ctas = used * c, waves = (tiles + n - 1) / n;
        const double busiest = (double)waves * ((nk + c - 1) / c), mean = (double)tiles * nk / ctas, share = 0.0032 * ctas;
        const double chunks = mean + (c == 1 ? 1.6 : 0.21) * (busiest - mean);
        double early = share > 0.41 ? share : 0.41, late = ctas > 148 ? 0.92 : 0.68;
        if (late < share) late = share;
        if (c == 1 && ctas > 148) early = late = 0.86;
        const double t = early * (chunks < 9.3 ? chunks : 9.3) + (chunks > 9.3 ? (chunks - 9.3) * late : 0.0) + (c > 1 ? 0.62 * waves + 0.026 * c : 0.0);
        if (t < best) best = t, best_c = c;
    }
    return best_c;
}

template <int MT, bool F32>
int launch_tc(const cudaLaunchConfig_t& cfg, const CUtensorMap& map0, const CUtensorMap& map1, const TcParams& p) {
    CN_ALLOW_SMEM((nvfp4_gemv_tc_kernel<MT, F32>), SM_SHARE);
    CN_CUDA(cudaLaunchKernelEx(&cfg, nvfp4_gemv_tc_kernel<MT, F32>, map0, map1, p));
    return CN_OK;
}

}  // namespace

extern "C" int cn_nvfp4_gemv_cut(int rows, int k, int gate_up) { return rows < 1 || k < CH ? 0 : cut_of(gate_up ? (rows + 63) / 64 : (rows + 127) / 128, k / CH); }

int cn_gemv_tc_launch(const GemvCall& a, cudaStream_t stream, const char* who) {
    const bool gu = a.w1 != nullptr, f32 = a.dtype == CN_F32;
    const int m = a.m, mt = m == 1 ? 1 : m == 2 ? 2 : m <= 4 ? 4 : 8;
    const int per_tile = gu ? 64 : 128, tiles = (a.rows + per_tile - 1) / per_tile, nk = a.k / CH;
    const int c = cut_of(tiles, nk), ncl = clusters_of(c);
    if (ncl < 1) CN_FAIL(CN_ERR_CUDA, "%s: the device does not say how many clusters it holds", who);
    const int clusters = tiles < ncl ? tiles : ncl;
    TcParams p = {};
    p.w0 = (const uint8_t*)a.w0, p.w1 = (const uint8_t*)a.w1, p.gs0 = a.gs0, p.gs1 = a.gs1 ? a.gs1 : a.gs0, p.x = a.x, p.y = a.y;
    p.rows = a.rows, p.k = a.k, p.m = m, p.ldy = a.ldy, p.out_f32 = a.out_f32, p.limit = a.limit, p.csize = c, p.tiles = tiles;
    p.share = ((per_tile + c - 1) / c + 3) & ~3;
    p.qinv = ((1u << 20) + (uint32_t)p.share - 1u) / (uint32_t)p.share;
    // sums handed over: a slot per tile in flight, up to NSLOT
    p.ex_bytes = c > 1 || gu || a.line_bases ? c * (gu ? 2 : 1) * p.share * mt * (f32 ? 8 : 4) : 0;
    const int per_cluster = (tiles + clusters - 1) / clusters, front = fixed_smem(mt, f32) + (per_cluster < NSLOT ? per_cluster : NSLOT) * p.ex_bytes;
    p.raw = (SM_SHARE - front) / RAW_STAGE;
    if (p.raw > MAX_RAW) p.raw = MAX_RAW;
    if (p.raw < 1) CN_FAIL(CN_ERR_LIMIT, "%s: %d rows in clusters of %d leave no room for weights", who, m, c);
    if (a.line_bases) {
        if (m != 1 || f32 || a.out_f32 || a.line_world < 2 || a.line_world > 8 || (a.rows & 3) || (a.line_row0 & 3) || !a.line_epoch || a.line_tag < 1 ||
            a.line_tag > 4095 || (a.line_buf & ~1))
            CN_FAIL(CN_ERR_SHAPE, "%s: line output needs one bf16 row, 2..8 ranks and row counts in multiples of 4 (rows %d, first row %d, ranks %d)", who,
                    a.rows, a.line_row0, a.line_world);
        p.yl_world = a.line_world, p.yl_row0 = a.line_row0, p.yl_stride = (unsigned long long)a.line_stride, p.yl_epoch = a.line_epoch;
        p.yl_tag = a.line_tag, p.yl_buf = a.line_buf, p.yl_flip = a.line_flip ? 1 : 0;
        for (int d = 0; d < a.line_world; d++) p.yl[d] = a.line_bases[d];
    }
#ifdef CN_M1_TRACE
    p.trace = cn_trace_slot();
#endif
    CUtensorMap map0, map1;
    const unsigned long long row_bytes = (unsigned long long)nk * 144;
    if (int rc = cn_tmap_words(&map0, a.w0, row_bytes / 4, (unsigned long long)a.rows, 36, (unsigned)per_tile)) return rc;
    if (!gu)
        map1 = map0;
    else if (int rc = cn_tmap_words(&map1, a.w1, row_bytes / 4, (unsigned long long)a.rows, 36, 64))
        return rc;
    // A CTA asks for half of an SM's shared memory, as of its tensor memory: as many of these kernels (or of nvfp4_rows_tc.cu's) as fit an SM find tensor memory there. The pair
    // GEMM, which takes all of it, stands apart by its registers: 640 threads of 72 leave no room for 448 of 64.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * c)), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = SM_SHARE, cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at, cfg.numAttrs = 1;
    if (c > 1) {
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = (unsigned)c, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    if (f32) return mt == 1 ? launch_tc<1, true>(cfg, map0, map1, p) : mt == 2 ? launch_tc<2, true>(cfg, map0, map1, p) : mt == 4 ? launch_tc<4, true>(cfg, map0, map1, p) : launch_tc<8, true>(cfg, map0, map1, p);
    return mt == 1 ? launch_tc<1, false>(cfg, map0, map1, p) : mt == 2 ? launch_tc<2, false>(cfg, map0, map1, p) : mt == 4 ? launch_tc<4, false>(cfg, map0, map1, p) : launch_tc<8, false>(cfg, map0, map1, p);
}
