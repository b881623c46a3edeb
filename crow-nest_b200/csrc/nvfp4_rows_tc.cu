// NVFP4 matrices times groups of up to eight activation rows on tcgen05.mma kind::mxf4nvf4: the routed experts of a step (groups of rows of one expert) and the
// shared expert of more rows than a GEMV takes. Supersedes gemv_fp4_ptrb over the pointer tables (engine/src/kernels.rs:195-233) together with the grouping
// of the reference's prefill path (moe_count / moe_plan / moe_scatter, engine/src/kernels.rs:3334-3420). Arithmetic as in nvfp4_gemv_tc.cu: weights as they
// are, rows as octal digits (blocks that these do not hold well multiplied out), chunks of 256 values of k added in order (f32, for f32 rows 64 bits).
//
// Persistent CTAs, two per SM, walk units of (group, 128-row tile; 64 gate and 64 up rows). The matrices come from device tables, so there is no tensor map:
// a scout warp looks up 32 units at a time (positions, combos, expert, addresses) and hands them to the other warps through a ring, and the warps that lay
// the weights out for the tensor core bring them in themselves, by 16-byte asynchronous copies, past the ends of units. Warps: 0-3 add up and store,
// 4-7 weights, 8-11 activations, 12 scout, 13 issues the MMAs. In the gate / up form a warp's rows are 16 of gate and the same 16 of up.
//
// What bounds it: no unit of the chip but the roles' own loops and hand-overs. A step of 64 tokens, 512 experts of 2048 x 512, top 10, took 165 us; with all copies, stores, digits and sums left
// out 89, with the copies alone left out 139, the stores 167, the digits 148, the sums 158. (With operand A in shared memory that was the nearest bound, 1740 of 2390 cycles of a chunk in both CTAs.)
// us under the profiler, here / mma.sync kernel that decoded to f16 for eight bf16 or two f32 rows: gate / up 85 / 114 (5.0 TB/s), down 63 / 77.
// Tried: a bulk copy for each row piece of 144 bytes (gate / up 105 -> 166 us); copies asked for before the stores of the chunk in hand, one chunk less ahead (109); three or four chunks of
// accumulators and operands in flight (the same); two teams of weight warps, and weight and activation warps on schedulers of their own (slower); digits that stay in their stages while tiles of
// one group follow each other (the same); the operand's bytes taken as they lie in the container (an illegal instruction, whose cause was not found).
#include "nvfp4_digits.cuh"
#include "nvfp4_gemv.cuh"

#include <type_traits>

namespace {

constexpr int RG = 8;        // most rows of a group
constexpr int CH = 256;      // values of k in a chunk
constexpr int PIECE = 32 * 144;  // container bytes of a warp's 32 rows and a chunk
__host__ __device__ constexpr int depth_of(bool f32) { return f32 ? 2 : 3; }  // chunks in flight, as many as fit beside four chunks of digits (two and one chunk more in flight: 64 tokens of f32 179 / 177 us, 288 experts 338 / 331)
constexpr int NA = 2, NB = 4, NX = 16, NDONE = 4, NU = 8;  // operand stages, chunks of digits, chunk factors, finished chunks, units in the ring
constexpr int NBAR = NX + NDONE + 2 * NU;
constexpr int SCOUT = 12, ISSUER = 13, THREADS = 448;
constexpr int FS_OFF = 512, WF_OFF = 1536, UNIT_OFF = 1792, HEADER = 2560;
// columns of the widest MMA, whose N is a multiple of 16: the accumulators lie this far apart in tensor memory (eight f32 rows are 88 columns, and 96 are written)
__host__ __device__ constexpr int ncol(bool f32) { return (RG * digits_of(f32) + 15) / 16 * 16; }
__host__ __device__ constexpr int b_stage(bool f32) { return ncol(f32) * 128 + 4 * 512; }
// accumulators, in half of an SM's tensor memory beside the codes of two chunks and the scales: those of two chunks where they fit
constexpr int TMEM = 256, TM_FIXED = NA * A_COLS + 64;
__host__ __device__ constexpr int nacc(bool f32) { return 2 * ncol(f32) + TM_FIXED <= TMEM ? 2 : 1; }
__host__ __device__ constexpr int smem_of(bool f32) { return NA * A_SCALES + NB * b_stage(f32) + 4 * depth_of(f32) * PIECE + HEADER; }
constexpr int SM_SHARE = (227 * 1024) / 2 - 1024;
static_assert(smem_of(true) <= SM_SHARE && smem_of(false) <= SM_SHARE, "shared memory");

struct Unit {
    unsigned long long w0, w1;
    int tile, nrows;  // nrows < 0: the end
    int combo[RG], xrow[RG];  // rows of results, of activations
};
static_assert(UNIT_OFF + NU * sizeof(Unit) <= HEADER && NBAR * 8 + 8 <= FS_OFF, "header");

template <bool F32, bool KEPT>
__global__ void __launch_bounds__(THREADS, 2) nvfp4_rows_tc_kernel(const RowsCall c) {
    constexpr int D = depth_of(F32), LV = digits_of(F32), ES = F32 ? 4 : 2, N = ncol(F32), B_CODES = N * 128, B_STAGE = b_stage(F32);
    constexpr int NACC = nacc(F32);
    constexpr uint32_t SFA_COL = NACC * N, SFB_COL = NACC * N + 32, A_COL = NACC * N + 64;
    static_assert(NACC * N + TM_FIXED <= TMEM && N % 16 == 0, "tensor memory columns");
    using Acc = typename std::conditional<F32, double, float>::type;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *a0 = smem, *b0 = a0 + NA * A_SCALES, *r0 = b0 + NB * B_STAGE, *head = r0 + (size_t)4 * D * PIECE;
    uint64_t* ready = (uint64_t*)head;        // [NX] weights and digits of a chunk, and its accumulators (those of two chunks before) have been read
    uint64_t* done = ready + NX;              // [NDONE] MMAs of a chunk; the issuer arrives too, and hands on what weight and activation warps wrote beside the operands
    uint64_t* unit_full = done + NDONE;       // [NU]
    uint64_t* unit_empty = unit_full + NU;    // [NU]
    uint32_t* tmem_slot = (uint32_t*)(unit_empty + NU);
    float2* fs = (float2*)(head + FS_OFF);      // [NX][8] {factor, blocks without digits}
    uint32_t* wf = (uint32_t*)(head + WF_OFF);  // [NX][4] scale bytes of 0xFF seen
    Unit* units = (Unit*)(head + UNIT_OFF);     // [NU]
    const int tid = threadIdx.x, warp = (int)warp_uniform((uint32_t)tid >> 5), lane = tid & 31;
    const bool gu = c.tab1 || c.w1 || c.fused_up_rows > 0;
    const int nk = c.k / CH, per_tile = gu ? 64 : 128, T = (c.rows + per_tile - 1) / per_tile;
    const size_t row_bytes = (size_t)nk * 144;

    if (warp == SCOUT) {
        // a barrier a lane and round: chunks (four warps each that bring weights, digits and empty accumulators), finished chunks, units full and empty (four + four + four + one warps read them)
        for (int i = lane; i < NBAR; i += 32) mbar_init(ready + i, i < NX ? 12 : i < NX + NDONE ? 2 : i < NBAR - NU ? 1 : 13);
        mbar_fence_init();
        __syncwarp();
    } else if (warp == ISSUER) {
        tc_alloc<1>(tmem_slot, TMEM);
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    pdl_launch_dependents();  // (behind the allocation of tensor memory)
    pdl_wait();               // groups, ids and activations come from the kernels before this one

    if (warp == SCOUT) {
        // ------------------------------------------------------------ units: a lane looks one up, lane after lane hands them on
        const int n1 = c.count1 ? *c.count1 : 0, ngroups = c.w0 ? (c.m + RG - 1) / RG : (c.order ? n1 + *c.count2 : c.m);
        const long long total = (long long)ngroups * T;
        int q = 0;
        bool ok = true;
        auto room = [&]() {  // the ring has a place for unit q
            if (q >= NU && !mbar_wait(&unit_empty[q % NU], (uint32_t)(q / NU - 1) & 1u)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                ok = false;
            }
            return ok;
        };
        for (long long u0 = blockIdx.x; u0 < total && ok; u0 += 32LL * gridDim.x) {
            const long long u = u0 + (long long)lane * gridDim.x;
            Unit mine = {};
            bool valid = u < total;
            if (valid) {
                const int grp = (int)(u / T);
                mine.tile = (int)(u - (long long)grp * T);
                int pos = grp * RG;
                mine.nrows = min(RG, c.m - pos), mine.w0 = (unsigned long long)c.w0, mine.w1 = (unsigned long long)c.w1;
                if (!c.w0) {
                    if (c.order)
                        pos = grp < n1 ? c.pos1[grp] : c.pos2[grp - n1], mine.nrows = grp < n1 ? 1 : c.rows2[grp - n1];
                    else
                        pos = grp, mine.nrows = 1;  // the combos as they come
                }
#pragma unroll
                for (int r = 0; r < RG; r++) {
                    mine.combo[r] = r < mine.nrows ? (c.order ? c.order[pos + r] : pos + r) : 0;
                    mine.xrow[r] = mine.combo[r] / c.x_div;
                }
                if (!c.w0) {
                    const int e = c.ids[mine.combo[0]];
                    valid = e >= 0 && !(c.experts > 0 && e >= c.experts);
                    if (valid) {
                        mine.w0 = c.tab0[e];
                        mine.w1 = c.tab1 ? c.tab1[e] : (c.fused_up_rows > 0 && mine.w0 ? mine.w0 + (unsigned long long)c.fused_up_rows * row_bytes : 0ull);
                        valid = mine.w0 && (!gu || mine.w1);  // (a matrix that is not resident: nothing to do)
                    }
                }
            }
            for (uint32_t left = __ballot_sync(0xffffffffu, valid); left && room(); left &= left - 1, q++) {
                const int j = __ffs(left) - 1;
                if (lane == j) {
                    units[q % NU] = mine;
                    mbar_arrive(&unit_full[q % NU]);
                }
                __syncwarp();
            }
        }
        if (ok && room() && lane == 0) {
            units[q % NU].nrows = -1;
            mbar_arrive(&unit_full[q % NU]);
        }
        __syncwarp();
    } else if (warp == ISSUER) {
        // ------------------------------------------------------------ scale copies and MMAs
        const uint32_t a_u = warp_uniform(smem_u32(a0)), b_u = warp_uniform(smem_u32(b0));
        bool ok = true;
        for (int q = 0, i = 0; ok; q++) {
            if (!mbar_wait(&unit_full[q % NU], (uint32_t)(q / NU) & 1u)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            const int nrows = (int)warp_uniform((uint32_t)units[q % NU].nrows);
            if (nrows < 0) break;
            const uint32_t idesc = idesc_bs((nrows * LV + 15) & ~15);
            for (int ch = 0; ch < nk; ch++, i++) {
                const int a = i & 1, b = i % NB;
                if (!mbar_wait(&ready[i % NX], (uint32_t)(i / NX) & 1u)) {  // (one wait for all three: each costs some 75 cycles, passed or not)
                    cn_dev_fail(CN_DEV_WAIT_FULL);
                    ok = false;
                    break;
                }
                tc_after();
                const uint64_t db = tc_desc_sw128(b_u + (uint32_t)(b * B_STAGE));
                const uint64_t sa = desc_sf(a_u + (uint32_t)(a * A_SCALES)), sb = desc_sf(b_u + (uint32_t)(b * B_STAGE + B_CODES));
                const uint32_t ta = tmem + SFA_COL + 16 * a, tb = tmem + SFB_COL + 16 * a, td = tmem + N * (i % NACC);
                if (elect_lane()) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        cp_sf(ta + 4 * j, sa + 32 * j);
                        cp_sf(tb + 4 * j, sb + 32 * j);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) umma_bs(td, tmem + A_COL + A_COLS * a + 8 * j, db + 2 * j, idesc, ta + 4 * j, tb + 4 * j, j > 0 ? 1u : 0u);
                    tc_commit<1>(&done[i % NDONE]);
                    mbar_arrive(&done[i % NDONE]);
                }
                __syncwarp();
            }
            if (lane == 0) mbar_arrive(&unit_empty[q % NU]);
        }
    } else if (warp >= 8) {
        // ------------------------------------------------------------ activations -> digits: rows of a chunk and the next chunk's go round the four warps
        const int w = warp - 8;
        int q = 0, ch = 0, nrows = 0;
        using Held = typename std::conditional<KEPT, DigitRecord<F32>, ChunkValues<F32>>::type;
        Held nx[2];
        bool ok = true;
        auto unit = [&](int n) -> int {  // rows of unit n
            if (!mbar_wait(&unit_full[n % NU], (uint32_t)(n / NU) & 1u)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                ok = false;
                return -1;
            }
            return units[n % NU].nrows;
        };
        auto fetch = [&](int n, int rows, int chunk, int i) {
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const int row = ((w - i) & 3) + 4 * t;
                if (row < rows) {
                    if constexpr (KEPT)
                        nx[t].load(c.digits + ((size_t)units[n % NU].xrow[row] * nk + chunk) * digit_record(F32), lane);
                    else
                        nx[t].load((const char*)c.x + ((size_t)units[n % NU].xrow[row] * c.k + (size_t)chunk * CH) * ES, lane);
                }
            }
        };
        nrows = unit(0);
        if (nrows >= 0) fetch(0, nrows, 0, 0);
        for (int i = 0; nrows >= 0; i++) {
            Held now[2] = {nx[0], nx[1]};
            const int at = q;
            int next_rows = nrows;
            if (++ch == nk) ch = 0, q++, next_rows = unit(q);
            if (next_rows >= 0) fetch(q, next_rows, ch, i + 1);
            if (!ok) break;
            // a warp without a row in this chunk only counts itself (64 tokens of 512 experts 176.4 -> 174.0 us). It has one every four chunks at least, so it is no more than six chunks
            // ahead of the MMAs, and there are NX slots.
            if (((w - i) & 3) < nrows) {
                if (i >= NB && !mbar_wait(&done[(i - NB) % NDONE], (uint32_t)((i - NB) / NDONE) & 1u)) {
                    cn_dev_fail(CN_DEV_WAIT_EMPTY);
                    break;
                }
                uint8_t* bs = b0 + (i % NB) * B_STAGE;
                // one copy of the code for both rows of a warp: with two, instructions come late (the roles of a CTA share the instruction cache): us per step with / without, 64 tokens
                // of 512 experts 195.6 / 190.9, 128 tokens 291 / 272, of 64 experts (groups of eight) 148 / 134, f32 rows 171 / 151
#pragma unroll 1
                for (int row = (w - i) & 3; row < nrows; row += 4) {
                    if constexpr (KEPT)
                        now[0].store(lane, bs, bs + B_CODES, row, &fs[(i % NX) * 8 + row]);
                    else
                        to_digits<F32>(now[0].v, lane, bs, bs + B_CODES, row, &fs[(i % NX) * 8 + row]);
                    now[0] = now[1];
                }
                fence_async();
                __syncwarp();
            }
            if (lane == 0) {
                mbar_arrive(&ready[i % NX]);
                if (q != at) mbar_arrive(&unit_empty[at % NU]);
            }
            nrows = next_rows;
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------ weights: 32 rows of the tile to a warp, copied in ahead and laid out as the A operand
        const int w = warp - 4;
        const uint32_t ring = smem_u32(r0) + (uint32_t)(w * D * PIECE);
        const uint64_t pol = l2_policy_evict_first();
        // sixteen-byte pieces, nine to a row and chunk, side by side in the stage; in the gate / up form rows 16-31 of a warp are the up rows of its gate rows
        uint32_t off[9];
#pragma unroll
        for (int j = 0; j < 9; j++) {
            const int id = lane + 32 * j, row = id / 9;
            off[j] = (uint32_t)(gu ? row & 15 : row) * (uint32_t)row_bytes + (uint32_t)(id - 9 * row) * 16u;
        }
        int iq = 0, ic = 0, is = 0, have = 0, asked = 0;  // what is asked for next: unit, chunk, stage; rows there are; chunks so far
        const uint8_t *from = nullptr, *from1 = nullptr;
        bool more = true, ok = true;
        auto issue = [&]() {
            if (more && ic == 0) {
                if (!mbar_wait(&unit_full[iq % NU], (uint32_t)(iq / NU) & 1u)) {
                    cn_dev_fail(CN_DEV_WAIT_FULL);
                    more = ok = false;
                } else {
                    const Unit& u = units[iq % NU];
                    more = u.nrows >= 0;
                    const int first = u.tile * per_tile + w * (gu ? 16 : 32);
                    from = (const uint8_t*)u.w0 + (size_t)first * row_bytes, from1 = (const uint8_t*)u.w1 + (size_t)first * row_bytes;
                    have = c.rows - first;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&unit_empty[iq % NU]);  // (nothing else of the unit is wanted here)
                }
            }
            if (more) {
                const uint32_t dst = ring + (uint32_t)(is * PIECE + lane * 16);
                // piece 32 j + lane: of row 16 and on from piece 144
                const uint8_t *lo = from + (uint32_t)(ic * 144), *hi = gu ? from1 + (uint32_t)(ic * 144) : lo, *mid = lane < 16 ? lo : hi;
                auto copy = [&](int j, uint32_t at) {
                    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst + 512u * j), "l"((j < 4 ? lo : j == 4 ? mid : hi) + at), "l"(pol) : "memory");
                };
                if (have >= (gu ? 16 : 32)) {
#pragma unroll
                    for (int j = 0; j < 9; j++) copy(j, off[j]);
                } else {  // the matrix ends inside these rows
#pragma unroll 1
                    for (int j = 0; j < 9; j++) {
                        const int id = lane + 32 * j, row = id / 9, r = gu ? row & 15 : row;
                        if (r < have) copy(j, (uint32_t)r * (uint32_t)row_bytes + (uint32_t)(id - 9 * row) * 16u);
                    }
                }
                if (++is == D) is = 0;
                if (++ic == nk) ic = 0, iq++;
                asked++;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll 1
        for (int i = 0; i < D; i++) issue();
        // one loop over the chunks that were asked for: what a unit is, is read once, when its first chunk is (us per step, 64 tokens of 512 experts: with a loop over units around a loop over their
        // chunks, and the quotient combo / x_div taken where a row is fetched, 186; so 178.6; f32 rows 208 / 195.5, 288 experts of 4096 x 2048 393 / 386)
        for (int i = 0, s = 0; i < asked && ok; i++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
            __syncwarp();  // the other lanes' copies, too
            const uint4* src = (const uint4*)(r0 + (size_t)(w * D + s) * PIECE) + lane * 9;
            uint32_t v[36];
            const uint32_t odd = load_row(src, v);
            if (i >= NA && !mbar_wait(&done[(i - NA) % NDONE], (uint32_t)((i - NA) / NDONE) & 1u)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                break;
            }
            store_row(tmem + A_COL + A_COLS * (i & 1), a0 + (i & 1) * A_SCALES, w, lane, v);
            if (lane == 0) wf[(i % NX) * 4 + w] = odd;
            fence_async();
            __syncwarp();  // every lane has read the stage
            if (lane == 0) mbar_arrive(&ready[i % NX]);
            issue();
            if (++s == D) s = 0;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------------ sums and output: a thread is a row of the tile
        if (lane < NACC) mbar_arrive(&ready[lane]);  // the accumulators of the first two chunks
        const float gs0 = __ldg(c.gs0), gs1 = gu ? __ldg(c.gs1) : 0.0f, gs = gu && lane >= 16 ? gs1 : gs0;
        bool ok = true;
        for (int q = 0, i = 0; ok; q++) {
            if (!mbar_wait(&unit_full[q % NU], (uint32_t)(q / NU) & 1u)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                break;
            }
            const Unit& u = units[q % NU];
            const int nrows = (int)warp_uniform((uint32_t)u.nrows), row = u.tile * per_tile + (gu ? warp * 16 + (lane & 15) : warp * 32 + lane);
            if (nrows < 0) break;
            Acc acc[RG];  // f32 rows: without the tensor scale
#pragma unroll
            for (int m = 0; m < RG; m++) acc[m] = 0;
            for (int ch = 0; ch < nk; ch++, i++) {
                if (!mbar_wait(&done[i % NDONE], (uint32_t)(i / NDONE) & 1u)) {
                    cn_dev_fail(CN_DEV_WAIT_FULL);
                    ok = false;
                    break;
                }
                tc_after();
                const uint32_t td = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(N * (i % NACC));
                const uint32_t odd = wf[(i % NX) * 4 + warp];
                uint32_t slow = odd;
#pragma unroll
                for (int m0 = 0; m0 < RG; m0 += 2) {
                    if (m0 >= nrows) break;
                    uint32_t d[2 * LV];
#pragma unroll
                    for (int m = 0; m < 2; m++) tc_ld_digits<F32>(td + LV * (m0 + m), d + LV * m);
                    tc_wait_ld();
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        if (m0 + m >= nrows) break;
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
                tc_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ready[(i + NACC) % NX]);
                if (slow && row < c.rows) {
                    const uint8_t* wr = (const uint8_t*)(gu && lane >= 16 ? u.w1 : u.w0) + ((size_t)row * nk + ch) * 144;
#pragma unroll 1
                    for (int m = 0; m < nrows; m++) {
                        const uint32_t blocks = __float_as_uint(fs[(i % NX) * 8 + m].y);
                        if (!(blocks | odd)) continue;
                        Acc v = whole_blocks<F32>(wr, blocks, odd != 0u, (const char*)c.x + ((size_t)u.xrow[m] * c.k + (size_t)ch * CH) * ES);
                        if (!F32) v *= gs;
#pragma unroll
                        for (int j = 0; j < RG; j++)
                            if (j == m) acc[j] += v;
                    }
                }
            }
            if (!ok) break;
#pragma unroll
            for (int m = 0; m < RG; m++) {
                if (m >= nrows) break;
                float v = F32 ? (float)(acc[m] * gs) : (float)acc[m];
                if (gu) v = act_gu(v, __shfl_down_sync(0xffffffffu, v, 16), c.limit);
                if (row >= c.rows || (gu && lane >= 16)) continue;
                const int combo = u.combo[m];
                float* y = c.yptrs ? (float*)c.yptrs[combo] : c.y + (size_t)combo * c.ldy;
                y[row] = v;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&unit_empty[q % NU]);
        }
        tc_before();
    }
    __syncthreads();
    if (warp == ISSUER) tc_dealloc<1>(tmem, TMEM);
}

template <bool F32, bool KEPT>
int launch(const RowsCall& p, dim3 grid, cudaStream_t stream) {
    CN_ALLOW_SMEM((nvfp4_rows_tc_kernel<F32, KEPT>), SM_SHARE);
    CN_CUDA(cn_launch_pdl(nvfp4_rows_tc_kernel<F32, KEPT>, grid, dim3(THREADS), SM_SHARE, stream, p));
    return CN_OK;
}

}  // namespace

int cn_rows_launch(const RowsCall& a, cudaStream_t stream, const char* who) {
    if (a.rows <= 0 || a.k <= 0 || a.k % 256 != 0) CN_FAIL(CN_ERR_SHAPE, "%s: k = %d must be a positive multiple of 256", who, a.k);
    if (((uintptr_t)a.w0 | (uintptr_t)a.w1 | (uintptr_t)a.x) & 15)  // 16-byte asynchronous copies and 128-bit loads
        CN_FAIL(CN_ERR_SHAPE, "%s: weight and activation pointers must be 16-byte aligned", who);
    RowsCall p = a;
    if (!p.gs1) p.gs1 = a.gs0;
    const bool gu = a.tab1 || a.w1 || a.fused_up_rows > 0, f32 = a.x_f32 != 0;
    const long long units = (long long)a.max_groups * ((a.rows + (gu ? 63 : 127)) / (gu ? 64 : 128));
    const dim3 grid((unsigned)(units < 2 * 148 ? units : 2 * 148));
    // (all of an SM's half, so that two CTAs and no more share its tensor memory)
    return f32 ? (p.digits ? launch<true, true>(p, grid, stream) : launch<true, false>(p, grid, stream)) : p.digits ? launch<false, true>(p, grid, stream) : launch<false, false>(p, grid, stream);
}
