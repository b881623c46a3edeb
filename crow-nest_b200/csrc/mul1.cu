// EXL3 "MUL1" trellis GEMV / expert FFN on sm_100a: y = x W with W = diag(suh) H W_hat H diag(svh) / 128,
// W_hat decoded from the 16-bit trellis states in the inner loop.
//
// Supersedes mul1_had_in / mul1_gemv / mul1_gemv2 / mul1_had_out / mul1_act_had_in
// (engine/src/kernels_mul1.cu:114, :280, :553, :669, :688) behind the plan interface of
// kernels::mul1::GemvPlan / FfnPlan (engine/src/kernels.rs:6644-6850); CPU twin cpu_mul1::gemv
// (engine/src/cpu_mul1.rs:1626). Format: converter/src/mul1.rs:10-34.
//
// Three steps per GEMV, none of which writes a dequantised weight:
//   had_in   xh = H128(x * suh) per 128-block, stored f16 with a power-of-two scale per block
//   gemv     y' = xh W_hat over a k-split: each CTA owns 8 adjacent tile columns (128 outputs) and
//            k/(16 S) tile rows; the 768-byte run of 8 tiles per tile row arrives by 1-D bulk copy
//            (TMA) into a shared-memory ring; warp w decodes tile column w: lane g extracts its 8
//            states from one to three 32-bit windows (every bitrate has its shifts at compile time), multiplies by 0x83DCD12D,
//            sums the bytes with dp4a (+0x6400 = the f16 pattern of 1024 + s), maps pairs through
//            one HFMA2 to the codec's f16 weights (bit-exact) and accumulates with f16 x f16 -> f32
//            mixed FMAs; partial sums of the k-split go to scratch
//   had_out  y = H128(sum of partials) / 128 * svh
// The first step is part of the GEMV launch for x where there are few rows (every CTA transforms its k-split) and a launch of its own for more
// (staged_rows), and a kernel of its own, with the activation, for h; the last one carries the weighted combine of a routed step. One token, four experts
// of 4096 x 1536: eight launches 52.5 us, five 43.4.
// The inner loop is instruction-bound, not HBM-bound: about 6 issue slots per weight. us per step in a graph of six, 64 experts of 4096 x 1536, top 4, the words of every state looked up on their own
// (at K = 3: three words a lane) and two loads a B operand / so, one token and 16: K = 1 58.9 / 36.3 and 416 / 238, 1.5 58.3 / 36.7 and 429 / 246, 2 58.9 / 37.8 and 437 / 251, 2.5 59.2 / 38.6 and 422 / 246,
// 3 40.8 / 39.0 and 258.5 / 248.2, 3.5 59.8 / 40.0 and 436 / 261, 4 59.4 / 38.2 and 425 / 239, 5 63.0 / 40.7 and 467 / 266, 6 62.9 / 41.4 and 473 / 280, 7 63.6 / 42.0 and 453 / 269, 8 63.7 / 40.1 and 472 / 262;
// gate of 16 slots of eight rows, K = 2.5 78.9 / 48.0, K = 6 88.2 / 51.8. Measured and not kept: pairs
// of sums put together by a multiplication in place of a byte permute (260.1 at K = 3), shifts by multiplications (270 and more): IMAD and dp4a share a pipe that is as full as the one
// of shifts and masks. A stage is a whole 128-row block of eight tiles: with
// four the waits and counters of a stage took a step of 16 tokens from 280 to 296 us.
// Three helpers restate reference text because their operation order defines the bits the parity contract asks for:
// fwht128 follows mul1_fwht128 (engine/src/kernels_mul1.cu:74-88: the stage order and the a+b / a-b pairing), out_block
// follows mul1_out_block (:98-110: partial sums left to right, then the transform, 1/128 and the scale), mul1_pair follows
// the first half of mul1_w2 (:500-510: the multiply-hash byte sum and the f16 FMA constants of the codec).
#include "common.cuh"
#include "nvfp4_gemv.cuh"

namespace {

constexpr int MUL1_MAXT = CN_MAX_M;  // activation rows per slot
constexpr int MUL1_GT = 8;           // most rows of a group when the MoE step bundles the combos of an expert (groups of 4 or 8)
constexpr int RING = 2;              // stages of the tile ring
constexpr int UROWS = 8;             // tile rows per stage: one 128-row block of the input
constexpr int XPAD = 16;             // f16 elements added to the pitch of a staged activation row
constexpr int SMEM_MOST = 160 * 1024, PAD_MORE = 16;  // shared memory of a GEMV call with a pad of eight; bytes of a pad beyond that

struct Mul1Spec {
    int k, n;        // in, out
    int bits, half;  // bitrate
    int n32;         // u32 words per tile
    long long tr_off, suh_off, svh_off;  // byte offsets into the record
};

// What differs between the matrices of one launch (gate and up read the same rows): the staged activations of the matrix, its
// partial sums, and where its trellis and input scales lie in a record.
struct Mul1Side {
    uint16_t* xh;
    float* xinv;
    float* part;
    long long tr_off, suh_off;
};

__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }

// natural-order FWHT of 128 values over one warp, element 4*lane + j in v[j]; stages (a+b, a-b)
__device__ __forceinline__ void fwht128(float v[4], int lane) {
    const float a0 = __fadd_rn(v[0], v[1]), a1 = __fsub_rn(v[0], v[1]), a2 = __fadd_rn(v[2], v[3]), a3 = __fsub_rn(v[2], v[3]);
    v[0] = __fadd_rn(a0, a2), v[1] = __fadd_rn(a1, a3), v[2] = __fsub_rn(a0, a2), v[3] = __fsub_rn(a1, a3);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float o = __shfl_xor_sync(0xffffffffu, v[j], m);
            v[j] = (lane & m) ? __fsub_rn(o, v[j]) : __fadd_rn(v[j], o);
        }
    }
}

// power-of-two scale of a 128-block so that |v| * mul < 2^15 (f16 exact range); returns mul, sets inv
__device__ __forceinline__ float block_scale(float amax, float& inv) {
    uint32_t e = (__float_as_uint(amax) >> 23) & 0xFF;
    inv = 1.0f;
    if (!(amax > 0.0f) || e == 255) return 1.0f;
    e = e < 15 ? 15 : e;
    inv = __uint_as_float((e - 14u) << 23);
    return __uint_as_float((268u - e) << 23);
}

// Four scaled values as two f16 planes: hi = f16(v * mul), lo = f16((v * mul - hi) * 2^11). hi + lo * 2^-11
// carries 22 significand bits, so the f16 x f16 products lose nothing that an f32 activation would keep.
__device__ __forceinline__ void store_hi_lo(uint16_t* xh, size_t plane, size_t at, const float v[4], float mul) {
    uint16_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float s = v[j] * mul;
        const __half h = __float2half_rn(s);
        hi[j] = __half_as_ushort(h);
        lo[j] = __half_as_ushort(__float2half_rn((s - __half2float(h)) * 2048.0f));
    }
    *(uint2*)(xh + at) = make_uint2(hi[0] | ((uint32_t)hi[1] << 16), hi[2] | ((uint32_t)hi[3] << 16));
    *(uint2*)(xh + plane + at) = make_uint2(lo[0] | ((uint32_t)lo[1] << 16), lo[2] | ((uint32_t)lo[3] << 16));
}

// where word i of a staged row lies: see mul1_gemv_kernel
__device__ __forceinline__ int word_at(int i) { return (i & ~7) | ((i & 3) << 1) | ((i >> 2) & 1); }
// the same planes for four values (4 lane .. 4 lane + 3) of a 128-block in shared memory
__device__ __forceinline__ void store_planes(uint16_t* blk, int plane, int lane, const float v[4], float mul) {
    uint32_t* w = (uint32_t*)blk;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        uint16_t hi[2], lo[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const float s = v[2 * j + q] * mul;
            const __half h = __float2half_rn(s);
            hi[q] = __half_as_ushort(h), lo[q] = __half_as_ushort(__float2half_rn((s - __half2float(h)) * 2048.0f));
        }
        const int at = word_at(2 * lane + j);
        w[at] = hi[0] | ((uint32_t)hi[1] << 16), w[plane / 2 + at] = lo[0] | ((uint32_t)lo[1] << 16);
    }
}

// Where the activation rows of a GEMV come from: row t of slot s is row (s / x_div) * T + t of x, or rowsrc[s * T + t] (negative = an
// unused row of a group: zeros). And where the records come from when the launch is the first of its chain: record s is table[ids[s]],
// written to ptrs for the kernels behind it (table null: ptrs is filled already).
struct Mul1In {
    const void* x;  // null: the side's staged planes are read instead
    int bf16, x_div;
    const int* rowsrc;
    const unsigned long long* table;
    const int32_t* ids;
    int experts;
};
// elements at .. at + 3 of a row; `wide`: the row's address allows one load
__device__ __forceinline__ void load_x4(const void* x, int bf16, bool wide, size_t at, float v[4]) {
    if (bf16) {
        const uint16_t* p = (const uint16_t*)x + at;
        uint32_t a, b;
        if (wide) {
            const uint2 u = *(const uint2*)p;
            a = u.x, b = u.y;
        } else {
            a = p[0] | ((uint32_t)p[1] << 16), b = p[2] | ((uint32_t)p[3] << 16);
        }
        v[0] = __uint_as_float(a << 16), v[1] = __uint_as_float(a & 0xffff0000u), v[2] = __uint_as_float(b << 16), v[3] = __uint_as_float(b & 0xffff0000u);
    } else {
        const float* p = (const float*)x + at;
        if (wide) {
            const float4 f = *(const float4*)p;
            v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
        } else {
            v[0] = p[0], v[1] = p[1], v[2] = p[2], v[3] = p[3];
        }
    }
}

// The input transform of 128 values of row t of a slot, by one warp: v = H128(x * suh), four values a lane; returns the power of two that
// brings them into f16 and, in inv, its inverse.
struct Mul1Block {
    const Mul1In& in;
    const uint16_t* suh;
    bool wide_x, wide_s;
    __device__ __forceinline__ Mul1Block(const Mul1In& in_, unsigned long long rec, long long suh_off)
        : in(in_), suh((const uint16_t*)(rec + (unsigned long long)suh_off)), wide_x(((uintptr_t)in_.x & 15) == 0), wide_s(((uintptr_t)suh & 7) == 0) {}
    __device__ __forceinline__ float operator()(int slot, int t, int T, int k, int c0, int lane, float v[4], float& inv) const {
        const int src = in.rowsrc ? in.rowsrc[slot * T + t] : 0;
        const size_t xrow = (in.rowsrc ? (size_t)(src < 0 ? 0 : src) : (size_t)(slot / in.x_div) * T + t) * k;
        load_x4(in.x, in.bf16, wide_x, xrow + c0, v);
        uint16_t sc[4];
        if (wide_s) {
            const uint2 u = *(const uint2*)(suh + c0);
            sc[0] = (uint16_t)u.x, sc[1] = (uint16_t)(u.x >> 16), sc[2] = (uint16_t)u.y, sc[3] = (uint16_t)(u.y >> 16);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) sc[j] = suh[c0 + j];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = __fmul_rn(src < 0 ? 0.0f : v[j], h2f(sc[j]));
        fwht128(v, lane);
        float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        return block_scale(amax, inv);
    }
};
// the record of a slot: of the combo's expert where the launch is the first of its chain
__device__ __forceinline__ unsigned long long slot_record(const unsigned long long* ptrs, const Mul1In& in, int slot) {
    if (!in.table) return ptrs[slot];
    const int e = in.ids[slot];
    return (e < 0 || (in.experts > 0 && e >= in.experts)) ? 0ull : in.table[e];
}

// The input transform as a launch of its own: xh = the hi / lo planes, xinv = the inverse scales. grid (k/128, matrices, slots), block 32 T (warp t =
// activation row t). Taken where the CTAs of the GEMV would repeat it too often (see staged_rows).
__global__ void mul1_had_in_kernel(unsigned long long* __restrict__ ptrs, Mul1Side side_a, Mul1Side side_b, int k, int T, size_t plane, Mul1In in) {
    pdl_launch_dependents();
    pdl_wait();  // everything below may read what earlier kernels of the stream wrote
    const int slot = blockIdx.z, t = threadIdx.x >> 5, blk = blockIdx.x, lane = threadIdx.x & 31;
    const unsigned long long rec = slot_record(ptrs, in, slot);
    if (in.table && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ptrs[slot] = rec;
    if (rec == 0ull) return;  // a null record: nothing to read or write
    const Mul1Side& sd = blockIdx.y ? side_b : side_a;
    const size_t row = (size_t)slot * T + t;
    const int c0 = blk * 128 + 4 * lane;
    float v[4], inv;
    const float mul = Mul1Block(in, rec, sd.suh_off)(slot, t, T, k, c0, lane, v, inv);
    store_hi_lo(sd.xh, plane, row * k + c0, v, mul);
    if (lane == 0) sd.xinv[row * (k / 128) + blk] = inv;
}

// the codec's f16 weights of two states (bit-exact): sum16 = 0x6400 + bytesum(state * 0x83DCD12D) is the
// f16 pattern of 1024 + s; w = fma(sum16, 0x1eee, 0xc931) in f16 with one rounding (converter/src/mul1.rs:135-143)
__device__ __forceinline__ uint32_t mul1_pair(uint32_t s0, uint32_t s1) {
    const uint32_t a = __dp4a(s0 * 0x83DCD12Du, 0x01010101u, 0x6400u), b = __dp4a(s1 * 0x83DCD12Du, 0x01010101u, 0x6400u);
    const uint32_t packed = __byte_perm(a, b, 0x5410);
    uint32_t w;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(w) : "r"(packed), "r"(0x1eee1eeeu), "r"(0xc931c931u));
    return w;
}

// A lane's eight states at a bitrate of K2 / 2. They lie in 16 + off(7) bits of the tile, which start at one of a few bits of a word: those that end within the first 32 of them are cut out of
// the window `hi` of these, those within the last 32 out of `lw`, and what neither has (above five bits) out of a third, `md`, that starts with the first of them. Where no lane starts so late that the second
// window goes beyond the next word (ALONE), both come from the same two words; else each has two of its own.
template <int K2>
struct Rate {
    static constexpr int words = 4 * K2;  // of a tile
    __host__ __device__ static constexpr int off(int j) { return K2 % 2 == 0 ? K2 / 2 * j : j / 2 * K2 + (j & 1 ? K2 / 2 + 1 : 0); }
    static constexpr int second = off(7) > 16 ? off(7) - 16 : 0;  // first bit of `lw`
    __host__ __device__ static constexpr int between() {          // of `md`; 0: none
        for (int j = 0; j < 8; j++)
            if (off(j) > 16 && off(j) < second) return off(j);
        return 0;
    }
    static constexpr int third = between();
    __host__ __device__ static constexpr bool alone() {
        for (int g = 0; g < 32; g++)
            if (((4 * K2 * g + K2 / 2 - 16) & 31) + second > 32) return false;
        return true;
    }
    __host__ __device__ static constexpr bool fits() {
        for (int j = 0; j < 8; j++)
            if (off(j) > 16 && off(j) < second && off(j) - third > 16) return false;
        return true;
    }
};
// 16 bits of x from bit `at` on, the most significant bit being 0
template <int AT>
__device__ __forceinline__ uint32_t field(uint32_t x) {
    return AT == 0 ? x >> 16 : (x >> (16 - AT)) & 0xffffu;
}
template <int K2, int J>
__device__ __forceinline__ uint32_t state(uint32_t hi, uint32_t md, uint32_t lw) {
    using R = Rate<K2>;
    constexpr int at = R::off(J);
    constexpr bool first = at <= 16, last = at >= R::second;
    return field<first ? at : last ? at - R::second : at - R::third>(first ? hi : last ? lw : md);
}

// y' partials of one k-split. grid (matrices n/128, S, slots), block 288 = 8 decode warps + 1 copy warp.
// part[slot][sp][t][n]; xh16 [slot][T][k] f16, xinv [slot][T][k/128].
// MT: activation rows the register allocation is built for (1, 2, 4 or 8; T <= MT of them live)
// HAD: the input transform is part of the launch: xh = H128(x * suh) per 128-block as hi / lo planes and 1 / scale, one warp per (row, block), straight
// into shared memory. The CTAs of one k-split repeat it (some 150 instructions a block), which costs less than a launch before this one
// and the planes' way through memory.
// K2: twice the bitrate
template <int K2, int MT, bool HAD>
__global__ void __launch_bounds__(288, 4) mul1_gemv_kernel(unsigned long long* __restrict__ ptrs, Mul1Side side_a, Mul1Side side_b, Mul1Spec sp_,
                                                        int S, int T, size_t plane, int SPC, Mul1In in) {
    pdl_launch_dependents();
    pdl_wait();  // everything below may read what earlier kernels of the stream wrote
    // SPC consecutive k-splits per CTA (blockIdx.y walks groups of SPC): the splits keep their own partial sums, so
    // the arithmetic does not depend on SPC; a CTA that takes several streams them through one ring without a drain
    extern __shared__ __align__(128) uint8_t smem[];
    const int slot = blockIdx.z, sp0 = blockIdx.y * SPC;
    const unsigned long long rec = HAD ? slot_record(ptrs, in, slot) : ptrs[slot];
    if (HAD && in.table && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ptrs[slot] = rec;
    if (rec == 0ull) return;  // uniform, before any barrier
    const int k = sp_.k, n = sp_.n, n32 = sp_.n32;
    const int tiles_n = n >> 4, tps = (k >> 4) / S, kb0 = sp0 * tps, rows = SPC * tps * 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool second = (int)blockIdx.x >= (n >> 7);  // the CTAs of the second matrix follow those of the first
    const Mul1Side& sd = second ? side_b : side_a;
    const uint16_t* __restrict__ xh = sd.xh;
    const float* __restrict__ xinv = sd.xinv;
    float* __restrict__ part = sd.part;
    const int nb0 = ((int)blockIdx.x - (second ? n >> 7 : 0)) * 8;
    const int run_bytes = 32 * n32;  // 8 tiles of one tile row
    uint64_t* full = (uint64_t*)smem;
    uint64_t* empty = full + RING;
    uint32_t* ring = (uint32_t*)(smem + 128);                                   // [RING][UROWS][8][n32]
    // [T][2][pitch] f16, hi and lo plane of a row beside each other, the words of every 16 values in the order 0 4 1 5 2 6 3 7: a lane's two words of a B operand are one 64-bit load. A pitch of
    // 32 bytes more than a multiple of 256 keeps the four columns that half a warp reads at once on distinct banks
    const int pitch = rows + XPAD;
    uint16_t* xs = (uint16_t*)(smem + 128 + (size_t)RING * UROWS * run_bytes);
    float* xi = (float*)(xs + (size_t)2 * T * pitch);  // [T][rows/128]
    if (threadIdx.x == 0) {
        for (int s = 0; s < RING; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 8);
        }
        mbar_fence_init();
    }
    __syncthreads();
    const int nst1 = (tps + UROWS - 1) / UROWS;  // stages of one split
    const int nst = SPC * nst1;
    if (warp == 8) {
        const uint8_t* base = (const uint8_t*)(rec + (unsigned long long)sd.tr_off);
        if (((uintptr_t)base & 15) != 0) {
            cn_dev_fail(103);  // a trellis that is not 16-byte aligned cannot be bulk-copied
            return;
        }
        for (int c = 0; c < nst; c++) {
            const int s = c % RING;
            if (c >= RING && !mbar_wait(&empty[s], ((c / RING) - 1) & 1)) {
                cn_dev_fail(CN_DEV_WAIT_EMPTY);
                return;
            }
            const int spi = c / nst1, cs = c - spi * nst1;  // split within the CTA, stage within the split
            const int live = min(UROWS, tps - cs * UROWS);
            if (lane == 0) {
                mbar_expect_tx(&full[s], (uint32_t)(live * run_bytes));
                mbar_arrive(&full[s]);
            }
            __syncwarp();
            if (lane < live) {
                const size_t off = ((size_t)(kb0 + spi * tps + cs * UROWS + lane) * tiles_n + nb0) * n32 * 4;
                bulk_g2s((uint8_t*)ring + ((size_t)s * UROWS + lane) * run_bytes, base + off, (uint32_t)run_bytes, &full[s]);
            }
        }
        return;
    }
    // the activation rows of this k-split, and their block scales
    const int nblk = rows / 128;
    if (HAD) {
        const Mul1Block block(in, rec, sd.suh_off);
        for (int i = warp; i < T * nblk; i += 8) {
            const int t = i / nblk, b = i - t * nblk;
            float v[4], inv;
            const float mul = block(slot, t, T, k, kb0 * 16 + b * 128 + 4 * lane, lane, v, inv);
            store_planes(xs + (size_t)2 * t * pitch + b * 128, pitch, lane, v, mul);
            if (lane == 0) xi[i] = inv;
        }
    } else {
        for (int i = threadIdx.x; i < T * rows / 2; i += 256) {
            const int t = i / (rows / 2), r = i - t * (rows / 2);
            const size_t at = ((size_t)slot * T + t) * k + (size_t)kb0 * 16;
            ((uint32_t*)(xs + (size_t)2 * t * pitch))[word_at(r)] = ((const uint32_t*)(xh + at))[r];
            ((uint32_t*)(xs + (size_t)(2 * t + 1) * pitch))[word_at(r)] = ((const uint32_t*)(xh + plane + at))[r];
        }
        for (int i = threadIdx.x; i < T * nblk; i += 256) {
            const int t = i / nblk, b = i - t * nblk;
            xi[i] = xinv[((size_t)slot * T + t) * (k / 128) + kb0 / 8 + b];
        }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");

    using R = Rate<K2>;
    static_assert(R::fits(), "states that lie in no window");
    constexpr int TW = R::words;  // words of a tile
    const int first_bit = (4 * K2 * lane + K2 / 2 - 16 + 32 * TW) % (32 * TW), wi0 = first_bit >> 5, sh0 = first_bit & 31;
    // Multiply-accumulate on the tensor cores. The eight weights a lane decodes from a tile are the A fragment of one
    // mma.m16n8k16 as they stand (MMA row = output column g / g + 8 of the tile, MMA k = the tile's k): w01 | w45 | w23 |
    // w67. Column c of the B operand is activation row c >> 1, plane c & 1 (hi, lo), so one MMA serves four activation
    // rows and a lane (g, t) ends up with the hi and lo sums of activation row t for outputs g and g + 8: nothing is
    // exchanged between lanes. Columns of rows beyond T repeat the last live row and are never stored.
    const int g = lane >> 2, t4 = lane & 3;
    constexpr int NM = MT > 4 ? 2 : 1;  // MMAs per tile: four activation rows each
    const uint16_t* xb[NM];
    const float* xil[NM];
#pragma unroll
    for (int i = 0; i < NM; i++) {
        const int rb = min(4 * i + (g >> 1), T - 1), rc = min(4 * i + t4, T - 1);
        xb[i] = xs + (size_t)(2 * rb + (g & 1)) * pitch + 4 * t4;
        xil[i] = xi + rc * nblk;
    }
    float acc[NM][4], tot0[NM], tot1[NM];
#pragma unroll
    for (int i = 0; i < NM; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = tot0[i] = tot1[i] = 0.0f;
    // Everything a tile needs beyond its own words is a constant offset from pointers that move once per stage, and a split is a whole number of stages and of 128-row
    // blocks (tps % 8 == 0, which the launcher guarantees), so the loop carries no division, no bounds test and no address arithmetic per tile.
    constexpr bool ALONE = R::alone();
    auto after = [](int w) { return w + 1 == TW ? 0 : w + 1; };
    const int o1 = after(wi0), wi1 = (wi0 + ((sh0 + R::second) >> 5)) % TW, o2 = after(wi1), sh1 = ALONE ? sh0 + R::second : (sh0 + R::second) & 31;
    const int wi2 = (wi0 + ((sh0 + R::third) >> 5)) % TW, o3 = after(wi2), sh2 = (sh0 + R::third) & 31;
    const uint32_t* lane_tile = ring + (size_t)warp * TW;  // this warp's tile of the ring's first tile row
    int s = 0, cs = 0, spi = 0;
    uint32_t ph = 0;
    for (int c = 0; c < nst; c++) {
        if (!mbar_wait(&full[s], ph)) {
            cn_dev_fail(CN_DEV_WAIT_FULL);
            return;
        }
        const uint32_t* tb = lane_tile + (size_t)s * (UROWS * 8) * TW;
        const int kx = (spi * tps + cs * UROWS) * 16;  // first k of the stage within the staged activations
#pragma unroll
        for (int u = 0; u < UROWS; u++) {
            const uint32_t* tl = tb + u * 8 * TW;
            const uint32_t w0 = tl[wi0], w1 = tl[o1];
            // (a shift of 32 is the second word itself)
            const uint32_t hi = __funnelshift_l(w1, w0, sh0), lw = R::second == 0 ? hi : ALONE ? __funnelshift_lc(w1, w0, sh1) : __funnelshift_l(tl[o2], tl[wi1], sh1);
            const uint32_t md = R::third == 0 ? hi : __funnelshift_l(tl[o3], tl[wi2], sh2);
            const uint32_t w01 = mul1_pair(state<K2, 0>(hi, md, lw), state<K2, 1>(hi, md, lw)), w23 = mul1_pair(state<K2, 2>(hi, md, lw), state<K2, 3>(hi, md, lw));
            const uint32_t w45 = mul1_pair(state<K2, 4>(hi, md, lw), state<K2, 5>(hi, md, lw)), w67 = mul1_pair(state<K2, 6>(hi, md, lw), state<K2, 7>(hi, md, lw));
#pragma unroll
            for (int i = 0; i < NM; i++) {
                const uint2 xr = *(const uint2*)(xb[i] + kx + u * 16);
                mma16816(acc[i], w01, w45, w23, w67, xr.x, xr.y);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == RING) s = 0, ph ^= 1u;
        // the stage was a 128-row block: hi + lo * 2^-11, then the block's activation scale
#pragma unroll
        for (int i = 0; i < NM; i++) {
            const float inv = xil[i][c];
            tot0[i] = fmaf(fmaf(acc[i][1], 4.8828125e-4f, acc[i][0]), inv, tot0[i]);
            tot1[i] = fmaf(fmaf(acc[i][3], 4.8828125e-4f, acc[i][2]), inv, tot1[i]);
            acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
        }
        if (++cs == nst1) {
            // end of a split: lane (g, t) stores outputs g and g + 8 of its tile column for activation row t (+ 4)
#pragma unroll
            for (int i = 0; i < NM; i++) {
                const int t = 4 * i + t4;
                if (t < T) {
                    float* pp = part + (((size_t)slot * S + sp0 + spi) * T + t) * n + (size_t)(nb0 + warp) * 16 + g;
                    pp[0] = tot0[i];
                    pp[8] = tot1[i];
                }
                tot0[i] = tot1[i] = 0.0f;
            }
            cs = 0;
            spi++;
        }
    }
}

// v = H128(sum_sp part[slot][sp][t][blk*128 ..]) / 128 * svh
__device__ __forceinline__ void out_block(float v[4], const float* __restrict__ part, const uint16_t* __restrict__ svh, int slot, int S, int T,
                                          int t, int n, int blk, int lane) {
    const int c0 = blk * 128 + 4 * lane;
    // the splits are added one after the other, but eight 16-byte loads are in flight at a time (one trip to L2 for each split
    // of each value made this the longest step of a one-token FFN after the GEMVs: 13 us of 64 with sixteen splits twice)
    const float4* src = (const float4*)(part + ((size_t)slot * S * T + t) * n + c0);
    const size_t step = (size_t)T * n / 4;
    float4 a = src[0];
    for (int q0 = 1; q0 < S; q0 += 8) {
        float4 r[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (q0 + i < S) r[i] = src[(size_t)(q0 + i) * step];
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (q0 + i < S) a.x = __fadd_rn(a.x, r[i].x), a.y = __fadd_rn(a.y, r[i].y), a.z = __fadd_rn(a.z, r[i].z), a.w = __fadd_rn(a.w, r[i].w);
    }
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    fwht128(v, lane);
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = __fmul_rn(__fmul_rn(v[j], 0.0078125f), h2f(svh[c0 + j]));
}

// grid (n/128, 1, slots), block 32 T (warp t = activation row t). YT: 0 f32, 1 bf16 output; y row = slot * T + t
// rowdst (optional): the y row of (slot, t) as an index into y [rows][n], negative = nothing to store
template <int YT>
__global__ void mul1_had_out_kernel(const unsigned long long* __restrict__ ptrs, const float* __restrict__ part, void* __restrict__ y, int n,
                                    int S, int T, long long svh_off, const int* __restrict__ rowdst) {
    pdl_launch_dependents();
    pdl_wait();  // everything below may read what earlier kernels of the stream wrote
    const int slot = blockIdx.z, t = threadIdx.x >> 5, blk = blockIdx.x, lane = threadIdx.x & 31;  // one warp per activation row
    if (ptrs[slot] == 0ull) return;
    const int dst = rowdst ? rowdst[slot * T + t] : 0;
    if (dst < 0) return;
    float v[4];
    out_block(v, part, (const uint16_t*)(ptrs[slot] + (unsigned long long)svh_off), slot, S, T, t, n, blk, lane);
    const size_t at = (rowdst ? (size_t)dst : (size_t)slot * T + t) * n + blk * 128 + 4 * lane;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (YT == 1)
            ((__nv_bfloat16*)y)[at + j] = __float2bfloat16_rn(v[j]);
        else
            ((float*)y)[at + j] = v[j];
    }
}

// had_out and the weighted combine of the routed step in one launch: y[tok][c] = base + sum_j w_j * had_out(combo tok * K + j)[c], j in pick
// order, with the arithmetic of moe_combine_kernel; base = shared[tok][c] or 0. grid (n/128, tokens), one warp per pick (K <= 32), which
// transforms its combo's 128 values into shared memory. place (optional): the (slot * T + t) of a combo, else slot = combo, T = 1.
template <int YT>
__global__ void __launch_bounds__(1024) mul1_out_combine_kernel(const unsigned long long* __restrict__ table, const int32_t* __restrict__ ids, const float* __restrict__ wts,
                                                                const float* __restrict__ part, const float* __restrict__ shared, void* __restrict__ y, int n, int S,
                                                                int T, int K, int experts, long long svh_off, const int* __restrict__ place) {
    extern __shared__ float sv[];  // [K][128], then the weights
    pdl_launch_dependents();
    pdl_wait();
    const int tok = blockIdx.y, j = threadIdx.x >> 5, blk = blockIdx.x, lane = threadIdx.x & 31;
    const int c = tok * K + j, e = ids[c];
    const unsigned long long rec = (e < 0 || (experts > 0 && e >= experts)) ? 0ull : table[e];
    float* ws = sv + K * 128;
    if (lane == 0) ws[j] = wts[c], ws[K + j] = rec ? 1.0f : 0.0f;
    if (rec) {
        const int at = place ? place[c] : c, slot = at / T, t = at - slot * T;
        float v[4];
        out_block(v, part, (const uint16_t*)(rec + (unsigned long long)svh_off), slot, S, T, t, n, blk, lane);
        *(float4*)(sv + j * 128 + 4 * lane) = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 128; i += blockDim.x) {
        float acc = 0.0f;
        for (int q = 0; q < K; q++)
            if (ws[K + q] != 0.0f) acc = __fadd_rn(acc, __fmul_rn(ws[q], sv[q * 128 + i]));
        const size_t to = (size_t)tok * n + blk * 128 + i;
        const float r = __fadd_rn(shared ? shared[to] : 0.0f, acc);
        if (YT == 1)
            ((__nv_bfloat16*)y)[to] = __float2bfloat16_rn(r);
        else
            ((float*)y)[to] = r;
    }
}

// The middle of the FFN in one launch: had_out of gate and of up, h = act(g, u), had_in of down.
// grid (inter/128, 1, slots), block 32 T (warp t = activation row t).
__global__ void mul1_act_had_in_kernel(const unsigned long long* __restrict__ ptrs, const float* __restrict__ part_g,
                                       const float* __restrict__ part_u, uint16_t* __restrict__ xh_d, float* __restrict__ xinv_d, int inter, int S,
                                       int T, long long svh_g, long long svh_u, long long suh_d, float limit, size_t plane) {
    pdl_launch_dependents();
    pdl_wait();  // everything below may read what earlier kernels of the stream wrote
    const int slot = blockIdx.z, t = threadIdx.x >> 5, blk = blockIdx.x, lane = threadIdx.x & 31;  // one warp per activation row
    if (ptrs[slot] == 0ull) return;
    float g[4], u[4], v[4];
    out_block(g, part_g, (const uint16_t*)(ptrs[slot] + (unsigned long long)svh_g), slot, S, T, t, inter, blk, lane);
    out_block(u, part_u, (const uint16_t*)(ptrs[slot] + (unsigned long long)svh_u), slot, S, T, t, inter, blk, lane);
    const uint16_t* suh = (const uint16_t*)(ptrs[slot] + (unsigned long long)suh_d);
    const int c0 = blk * 128 + 4 * lane;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float gv = g[j], uv = u[j];
        if (limit > 0.0f) {
            gv = gv > limit ? limit : gv;
            uv = uv > limit ? limit : (uv < -limit ? -limit : uv);
        }
        const float h = __fmul_rn(gv / (1.0f + expf(-gv)), uv);
        v[j] = __fmul_rn(h, h2f(suh[c0 + j]));
    }
    fwht128(v, lane);
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    float inv;
    const float mul = block_scale(amax, inv);
    const size_t row = ((size_t)slot * T + t) * inter;
    store_hi_lo(xh_d, plane, row + c0, v, mul);
    if (lane == 0) xinv_d[((size_t)slot * T + t) * (inter / 128) + blk] = inv;
}

// W_hat as fp16 bits, row major [k][n]: one thread per (tile, position) - the codec self-check
__global__ void mul1_reconstruct_kernel(const uint32_t* __restrict__ trellis, uint16_t* __restrict__ w, int k, int n, int bits, int half, int n32) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)(k / 16) * (n / 16) * 256;
    if (i >= total) return;
    const int p = (int)(i & 255);
    const long long tile = i >> 8;
    const int kb = (int)(tile / (n / 16)), nb = (int)(tile % (n / 16));
    const int sbits = n32 * 32;
    const int eb = !half ? (p + 1) * bits : ((p & 1) ? (p / 2 + 1) * (2 * bits + 1) : (p / 2) * (2 * bits + 1) + bits);
    const int lo = (eb - 16 + sbits) % sbits;
    const uint32_t* t = trellis + tile * n32;
    const int wi = lo >> 5, o = lo & 31, w1 = wi + 1 == n32 ? 0 : wi + 1;
    const uint32_t st = __funnelshift_l(t[w1], t[wi], o) >> 16;
    const uint32_t pr = mul1_pair(st, st);
    const int lane = p >> 3, j = p & 7;
    const int off[4] = {0, 1, 8, 9};
    const int row = 2 * (lane & 3) + off[j & 3], col = (lane >> 2) + 8 * (j >> 2);
    w[(size_t)(kb * 16 + row) * n + nb * 16 + col] = (uint16_t)(pr & 0xffff);
}

}  // namespace

// ---------------------------------------------------------------- host side
namespace {

struct Mul1Plan {
    int hidden, inter, bits, half, n32, max_slots, max_t;
    size_t kmax;
    uint16_t *xh, *xh_up;   // [2 planes][slots][T][kmax] f16: staged rows (of the down projection; of gate and of up where they are staged)
    size_t plane;           // elements of one plane
    float *xinv, *xinv_up;  // [slots][T][kmax/128]
    float *part_a, *part_b;  // [slots][16][T][kmax]
    unsigned long long* ptrs;  // [slots] gathered record addresses (MoE form)
    int32_t* order;            // [slots] combos sorted by expert (grouped MoE form)
    int* groups;               // [3 * slots + 8] the group lists and counts of cn_moe_group_launch
    int* rowsrc;               // [slots * MUL1_GT] x row of every (group slot, row), -1 = unused
    int* rowdst;               // [slots * MUL1_GT] combo (output row) of every (group slot, row), -1 = unused
    int* place;                // [slots] (group slot * rows + row) of every combo
    int grp_rows;              // rows the scratch holds per slot: max(max_t, 4)
    float* eo;                 // [slots][T][hidden] expert outputs (MoE form)
};

int ksplit(int k) {
    // the largest divisor of k/128 that is <= 16: k-splits end on Hadamard blocks
    const int blocks = k / 128;
    for (int s = 16; s >= 1; s--)
        if (blocks % s == 0) return s;
    return 1;
}

long long trellis_bytes(int k, int n, int n32) { return (long long)(k / 16) * (n / 16) * n32 * 4; }

Mul1Spec spec_of(const Mul1Plan* p, int which) {
    const long long tb = trellis_bytes(p->hidden, p->inter, p->n32), h2 = 2LL * p->hidden, i2 = 2LL * p->inter;
    Mul1Spec s;
    s.bits = p->bits, s.half = p->half, s.n32 = p->n32;
    if (which == 0) s.k = p->hidden, s.n = p->inter, s.tr_off = 0, s.suh_off = 3 * tb, s.svh_off = 3 * tb + h2;
    if (which == 1) s.k = p->hidden, s.n = p->inter, s.tr_off = tb, s.suh_off = 3 * tb + h2 + i2, s.svh_off = 3 * tb + 2 * h2 + i2;
    if (which == 2) s.k = p->inter, s.n = p->hidden, s.tr_off = 2 * tb, s.suh_off = 3 * tb + 2 * h2 + 2 * i2, s.svh_off = 3 * tb + 2 * h2 + 3 * i2;
    return s;
}

// live: how many of the slots are expected to hold a record (the grouped MoE form launches more slots than it fills)
// sb: the second matrix of the launch (up beside gate), or null. in: the rows to transform, or null where the side holds them staged
int launch_gemv(const unsigned long long* ptrs, const Mul1Side& sa, const Mul1Side* sb, const Mul1Spec& s, int slots, int T, size_t plane,
                cudaStream_t st, const Mul1In* in, int live = 0) {
    if (live < 1 || live > slots) live = slots;
    const int mats = sb ? 2 : 1;
    const int S = ksplit(s.k), tps = (s.k / 16) / S;
    if (tps % 8 != 0) CN_FAIL(CN_ERR_SHAPE, "mul1 gemv: k = %d does not split into whole 128-row blocks", s.k);  // the kernel's stage / block counters rely on it
    // k-splits per CTA: as many as still leave about four CTAs per SM (the splits keep separate partial sums, so
    // this only moves work between CTAs) and fit the staged activations
    int spc = 1;
    const size_t most = SMEM_MOST + (size_t)2 * T * PAD_MORE;  // (a limit of the calls, which has no part of the pad in it that a row got later)
    for (int c = S; c > 1; c--) {
        if (S % c) continue;
        const long long ctas = (long long)mats * (s.n / 128) * (S / c) * live;
        const size_t need = 128 + (size_t)RING * UROWS * 32 * s.n32 + (size_t)2 * T * (c * tps * 16 + XPAD) * 2 + 8 + (size_t)T * (c * tps / 8) * 4;
        if (ctas >= 592 && need <= most) {
            spc = c;
            break;
        }
    }
    const int rows = spc * tps * 16;
    const size_t smem = 128 + (size_t)RING * UROWS * 32 * s.n32 + (size_t)2 * T * (rows + XPAD) * 2 + 8 + (size_t)T * (rows / 128) * 4;
    dim3 grid(mats * (s.n / 128), S / spc, slots);
    if (smem > most) CN_FAIL(CN_ERR_LIMIT, "mul1 gemv: %zu B of shared memory per block", smem);
    const int k2 = 2 * s.bits + (s.half ? 1 : 0);
    const int mt = T == 1 ? 1 : (T == 2 ? 2 : (T <= 4 ? 4 : 8));
    const Mul1In none = {};
#define CN_MUL1_CASE(K2V, MTV, HADV)                                                                                                \
    if (k2 == K2V && mt == MTV && (in != nullptr) == HADV) {                                                                        \
        CN_ALLOW_SMEM((mul1_gemv_kernel<K2V, MTV, HADV>), SMEM_MOST + 2 * MUL1_MAXT * PAD_MORE);                                    \
        CN_CUDA(cn_launch_pdl((mul1_gemv_kernel<K2V, MTV, HADV>), grid, dim3(288), smem, st, const_cast<unsigned long long*>(ptrs), sa, sb ? *sb : sa, s, S, T, plane, spc, in ? *in : none)); \
    }
#define CN_MUL1_CASES(K2V) CN_MUL1_CASE(K2V, 1, true) CN_MUL1_CASE(K2V, 2, true) CN_MUL1_CASE(K2V, 4, true) CN_MUL1_CASE(K2V, 8, true) \
    CN_MUL1_CASE(K2V, 1, false) CN_MUL1_CASE(K2V, 2, false) CN_MUL1_CASE(K2V, 4, false) CN_MUL1_CASE(K2V, 8, false)
    CN_MUL1_CASES(2) CN_MUL1_CASES(3) CN_MUL1_CASES(4) CN_MUL1_CASES(5) CN_MUL1_CASES(6) CN_MUL1_CASES(7) CN_MUL1_CASES(8) CN_MUL1_CASES(10) CN_MUL1_CASES(12) CN_MUL1_CASES(14)
    CN_MUL1_CASES(16)
#undef CN_MUL1_CASES
#undef CN_MUL1_CASE
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

// Whether the rows are transformed by a launch of their own. Inside the GEMV every CTA of a k-split repeats the transform of its part: (n / 128) x (k / 128)
// block transforms for a row and matrix, against a launch more. us per call inside / apart, hidden 4096, inter 1536, one matrix (384 transforms a row) or
// gate and up (768) and the whole FFN: gate of 4 slots, 1 row each 16.4 / 18.4 (1.5 k), 4 rows 16.4 / 18.4 (6.1 k), 8 rows 20.5 / 20.5 (12.3 k); 16 slots, 2 rows
// 42.6 / 42.5 (12.3 k), 8 rows 57.4 / 52.8; 48 slots, 8 rows 166 / 135; FFN of 4 slots, 1 row 41.0 / 43.0 (3.1 k), 4 rows 45.1 / 45.1 (12.3 k); 16 slots, 8 rows
// 170 / 149; a routed step of 16 tokens 268 / 256, of 64 tokens 575 / 516.
bool staged_rows(const Mul1Spec& s, int matrices, int slots, int T) { return (long long)matrices * slots * T * (s.n / 128) * (s.k / 128) > 12288; }

// sb: the second matrix of the launch (up beside gate), or null
int launch_had_in(unsigned long long* ptrs, const Mul1In& in, const Mul1Side& sa, const Mul1Side* sb, int k, int slots, int T, size_t plane, cudaStream_t st) {
    CN_CUDA(cn_launch_pdl(mul1_had_in_kernel, dim3(k / 128, sb ? 2 : 1, slots), dim3(32 * T), 0, st, ptrs, sa, sb ? *sb : sa, k, T, plane, in));
    return CN_OK;
}

int check_run(const Mul1Plan* p, int slots, int T, const char* who) {
    if (!p) CN_FAIL(CN_ERR_SHAPE, "%s: null plan", who);
    if (slots < 1 || slots > p->max_slots || T < 1 || T > p->max_t)
        CN_FAIL(CN_ERR_LIMIT, "%s: %d slots x %d rows, the plan holds %d x %d", who, slots, T, p->max_slots, p->max_t);
    return CN_OK;
}

// Slot s of the grouped MoE form (gt rows per slot, 4 or 8): the groups of two or more rows first, then the one-row
// groups, then empty slots (null record). Fills the slot's record address and, per row, where its x row comes from and
// which combo's output row it is.
__global__ void mul1_slots_kernel(const unsigned long long* __restrict__ table, const int32_t* __restrict__ ids, const int32_t* __restrict__ order,
                                  const int* __restrict__ ga, const int* __restrict__ gb, const int* __restrict__ gbrows, const int* __restrict__ counts,
                                  unsigned long long* __restrict__ ptrs, int* __restrict__ rowsrc, int* __restrict__ rowdst, int* __restrict__ place, int slots, int x_div, int gt) {
    pdl_launch_dependents();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slots) return;
    const int na = counts[0], nb = counts[1];
    int pos = -1, rows = 0;
    if (s < nb) pos = gb[s], rows = gbrows[s];
    else if (s < nb + na) pos = ga[s - nb], rows = 1;
    ptrs[s] = pos < 0 ? 0ull : table[ids[order[pos]]];
    for (int t = 0; t < gt; t++) {
        const int c = t < rows ? order[pos + t] : -1;
        rowsrc[s * gt + t] = c < 0 ? -1 : c / x_div;
        rowdst[s * gt + t] = c;
        if (c >= 0) place[c] = s * gt + t;
    }
}

}  // namespace

extern "C" int cn_mul1_plan_destroy(void* plan);

extern "C" int cn_mul1_plan_create(void** plan_out, int hidden, int inter, int bits, int half, int max_slots, int max_t) {
    if (!plan_out || hidden <= 0 || inter <= 0 || hidden % 128 || inter % 128)
        CN_FAIL(CN_ERR_SHAPE, "cn_mul1_plan_create: [%d, %d] is not a positive multiple of 128 on both sides", hidden, inter);
    if (bits < 1 || bits > 8 || (half && bits > 3)) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_plan_create: unsupported bitrate %d%s", bits, half ? ".5" : "");
    if (max_slots < 1 || max_t < 1 || max_t > MUL1_MAXT) CN_FAIL(CN_ERR_LIMIT, "cn_mul1_plan_create: %d slots, %d rows (rows <= %d)", max_slots, max_t, MUL1_MAXT);
    Mul1Plan* p = new Mul1Plan();
    p->hidden = hidden, p->inter = inter, p->bits = bits, p->half = half, p->n32 = 8 * bits + (half ? 4 : 0), p->max_slots = max_slots, p->max_t = max_t;
    p->kmax = hidden > inter ? hidden : inter;
    // the grouped MoE form runs its slots with four or eight rows: the scratch holds four rows per slot, which covers
    // eight-row groups whenever there are few enough of them (see cn_moe_mul1_experts)
    p->grp_rows = max_t > 4 ? max_t : 4;
    const size_t rows = (size_t)max_slots * p->grp_rows;
    p->plane = rows * p->kmax;
    // a failure part-way frees what the earlier steps got (the destroy call takes a half-built plan)
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    step(cudaMalloc(&p->xh, 2 * p->plane * 2));
    step(cudaMalloc(&p->xh_up, 2 * p->plane * 2));
    step(cudaMalloc(&p->xinv, rows * (p->kmax / 128) * 4));
    step(cudaMalloc(&p->xinv_up, rows * (p->kmax / 128) * 4));
    step(cudaMalloc(&p->part_a, rows * 16 * p->kmax * 4));
    step(cudaMalloc(&p->part_b, rows * 16 * p->kmax * 4));
    step(cudaMalloc(&p->ptrs, (size_t)max_slots * 8));
    step(cudaMalloc(&p->order, (size_t)max_slots * 4));
    step(cudaMalloc(&p->groups, ((size_t)3 * max_slots + 8) * 4));
    step(cudaMalloc(&p->rowsrc, (size_t)max_slots * MUL1_GT * 4));
    step(cudaMalloc(&p->rowdst, (size_t)max_slots * MUL1_GT * 4));
    step(cudaMalloc(&p->place, (size_t)max_slots * 4));
    step(cudaMalloc(&p->eo, rows * hidden * 4));
    if (e != cudaSuccess) {
        cn_mul1_plan_destroy(p);
        CN_FAIL(CN_ERR_CUDA, "cn_mul1_plan_create: %s", cudaGetErrorString(e));
    }
    *plan_out = p;
    return CN_OK;
}

extern "C" int cn_mul1_plan_destroy(void* plan) {
    Mul1Plan* p = (Mul1Plan*)plan;
    if (!p) return CN_OK;
    cudaFree(p->xh), cudaFree(p->xh_up), cudaFree(p->xinv), cudaFree(p->xinv_up), cudaFree(p->place), cudaFree(p->part_a), cudaFree(p->part_b), cudaFree(p->ptrs),
        cudaFree(p->eo), cudaFree(p->order), cudaFree(p->groups), cudaFree(p->rowsrc), cudaFree(p->rowdst);
    delete p;
    return CN_OK;
}

extern "C" int cn_mul1_gemv(void* plan, int which, const unsigned long long* ptrs, const void* x, void* y, int slots, int t, int x_div, int dtype,
                            cn_stream_t stream) {
    Mul1Plan* p = (Mul1Plan*)plan;
    if (int rc = check_run(p, slots, t, "cn_mul1_gemv")) return rc;
    if (which < 0 || which > 2 || x_div < 1) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv: matrix %d (0 gate, 1 up, 2 down), x_div %d", which, x_div);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    cudaStream_t st = (cudaStream_t)stream;
    const Mul1Spec s = spec_of(p, which);
    const Mul1Side side = {p->xh, p->xinv, p->part_a, s.tr_off, s.suh_off};
    const Mul1In in = {x, dtype == CN_BF16, x_div, nullptr, nullptr, nullptr, 0};
    const bool staged = staged_rows(s, 1, slots, t);
    if (staged)
        if (int rc = launch_had_in(const_cast<unsigned long long*>(ptrs), in, side, nullptr, s.k, slots, t, p->plane, st)) return rc;  // (table null: ptrs is read)
    if (int rc = launch_gemv(ptrs, side, nullptr, s, slots, t, p->plane, st, staged ? nullptr : &in)) return rc;
    dim3 grid(s.n / 128, 1, slots);
    if (dtype == CN_BF16)
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<1>), dim3(grid), dim3(32 * t), 0, st, ptrs, p->part_a, y, s.n, ksplit(s.k), t, s.svh_off, (const int*)nullptr));
    else
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<0>), dim3(grid), dim3(32 * t), 0, st, ptrs, p->part_a, y, s.n, ksplit(s.k), t, s.svh_off, (const int*)nullptr));
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

// The FFN up to the partial sums of the down projection (p->part_a): gate and up with the input transform, the middle, down.
static int mul1_ffn_parts(Mul1Plan* p, const unsigned long long* ptrs, const Mul1In& in, int slots, int t, float limit, cudaStream_t st, int live = 0) {
    const Mul1Spec g = spec_of(p, 0), u = spec_of(p, 1), d = spec_of(p, 2);
    // gate and up share each launch: two small grids on two streams cost an event fork and join and ran one after the other
    // anyway (one token, four experts of 4096 x 1536: 65 -> 55 us with out_block's wide loads; 16 tokens: 295 us, no difference beyond noise)
    const Mul1Side ga = {p->xh, p->xinv, p->part_a, g.tr_off, g.suh_off}, up = {p->xh_up, p->xinv_up, p->part_b, u.tr_off, u.suh_off};
    const Mul1Side dn = {p->xh, p->xinv, p->part_a, d.tr_off, d.suh_off};
    const bool staged = staged_rows(g, 2, slots, t);
    if (staged)
        if (int rc = launch_had_in(const_cast<unsigned long long*>(ptrs), in, ga, &up, g.k, slots, t, p->plane, st)) return rc;
    if (int rc = launch_gemv(ptrs, ga, &up, g, slots, t, p->plane, st, staged ? nullptr : &in, live)) return rc;
    CN_CUDA(cn_launch_pdl(mul1_act_had_in_kernel, dim3(p->inter / 128, 1, slots), dim3(32 * t), 0, st, ptrs, p->part_a, p->part_b, p->xh, p->xinv, p->inter, ksplit(p->hidden), t,
                                                                         g.svh_off, u.svh_off, d.suh_off, limit, p->plane));
    return launch_gemv(ptrs, dn, nullptr, d, slots, t, p->plane, st, nullptr, live);
}

// y[slot][t] = down(act(gate x, up x)) as f32 when out_f32, else in the type of the rows; rowdst: see mul1_had_out_kernel
static int mul1_ffn(Mul1Plan* p, const unsigned long long* ptrs, const Mul1In& in, void* y, int slots, int t, float limit, int out_f32, cudaStream_t st,
                    const int* rowdst = nullptr, int live = 0) {
    if (int rc = mul1_ffn_parts(p, ptrs, in, slots, t, limit, st, live)) return rc;
    const Mul1Spec d = spec_of(p, 2);
    dim3 grid(d.n / 128, 1, slots);
    if (in.bf16 && !out_f32)
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<1>), dim3(grid), dim3(32 * t), 0, st, ptrs, p->part_a, y, d.n, ksplit(d.k), t, d.svh_off, rowdst));
    else
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<0>), dim3(grid), dim3(32 * t), 0, st, ptrs, p->part_a, y, d.n, ksplit(d.k), t, d.svh_off, rowdst));
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

extern "C" int cn_mul1_ffn(void* plan, const unsigned long long* ptrs, const void* x, void* y, int slots, int t, int x_div, float limit, int dtype,
                           cn_stream_t stream) {
    Mul1Plan* p = (Mul1Plan*)plan;
    if (int rc = check_run(p, slots, t, "cn_mul1_ffn")) return rc;
    if (x_div < 1) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_ffn: x_div %d", x_div);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_ffn: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    const Mul1In in = {x, dtype == CN_BF16, x_div, nullptr, nullptr, nullptr, 0};
    return mul1_ffn(p, ptrs, in, y, slots, t, limit, 0, (cudaStream_t)stream);
}

extern "C" int cn_moe_combine(const float* eo, const float* wts, const int32_t* ids, const unsigned long long* table, const float* shared,
                              const float* sgate, void* y, int tokens, int hidden, int topk, int experts, int dtype, cn_stream_t stream);

namespace {

// How the combos of a routed step run: one slot each, or bundled by expert into slots of T rows (place: see mul1_out_combine_kernel)
struct Mul1Slots {
    Mul1In in;
    int slots, T, live;
    const int *rowdst, *place;
};

int mul1_slots(Mul1Plan* p, const unsigned long long* table, const int32_t* ids, const void* x, int combos, int x_div, int experts, int dtype, cudaStream_t st,
               Mul1Slots& r) {
    r = {};
    r.in.x = x, r.in.bf16 = dtype == CN_BF16, r.in.x_div = x_div, r.slots = combos, r.T = 1;
    if (experts > 0 && 2 * combos >= experts) {
        // Enough combos that experts repeat: the combos are sorted by expert and bundled into groups that share one
        // decode of the expert's trellis (a group of up to four rows is one MMA per tile like a single row, eight rows
        // are two). Groups of eight when the batch is long (four combo slots per expert or more) and the plan's scratch
        // holds them; the slots launched are bounded by experts + combos / rows, the rest of the combo slots do not exist.
        const long long cap_rows = (long long)p->max_slots * p->grp_rows;
        int gt = 4;
        if (combos >= 4 * experts && ((long long)experts + combos / 8) * 8 <= cap_rows) gt = 8;
        long long ng = (long long)experts + combos / gt;  // every expert ends in at most one short group
        if (ng > combos) ng = combos;
        if (ng * gt <= cap_rows && ng <= p->max_slots) {
            int* ga = p->groups;
            int* gb = ga + combos;
            int* gbrows = gb + combos;
            int* counts = gbrows + combos;
            if (int rc = cn_moe_group_launch(ids, table, combos, experts, p->order, ga, gb, gbrows, counts, gt, st)) return rc;
            CN_CUDA(cn_launch_pdl(mul1_slots_kernel, dim3(((int)ng + 127) / 128), dim3(128), 0, st, table, ids, p->order, ga, gb, gbrows, counts, p->ptrs,
                                  p->rowsrc, p->rowdst, p->place, (int)ng, x_div, gt));
            // a slot beyond the groups is a null record, which all kernels skip; a group's unused rows are zero rows
            // (the work per CTA is sized as if a quarter of the launched slots were filled: measured best at 45 of 64 and at 8 of 128)
            r.in.rowsrc = p->rowsrc, r.in.x_div = 1, r.slots = (int)ng, r.T = gt, r.live = (int)((ng + 3) / 4), r.rowdst = p->rowdst, r.place = p->place;
            return CN_OK;
        }
    }
    r.in.table = table, r.in.ids = ids, r.in.experts = experts;
    return CN_OK;
}

}  // namespace

extern "C" int cn_moe_mul1_experts(void* plan, const unsigned long long* table, const int32_t* ids, const void* x, float* eo, int combos, int x_div,
                                   int experts, float limit, int dtype, cn_stream_t stream) {
    Mul1Plan* p = (Mul1Plan*)plan;
    if (int rc = check_run(p, combos, 1, "cn_moe_mul1_experts")) return rc;
    if (x_div < 1 || !eo) CN_FAIL(CN_ERR_SHAPE, "cn_moe_mul1_experts: x_div %d, eo %p", x_div, (void*)eo);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_mul1_experts: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    cudaStream_t st = (cudaStream_t)stream;
    Mul1Slots r;
    if (int rc = mul1_slots(p, table, ids, x, combos, x_div, experts, dtype, st, r)) return rc;
    return mul1_ffn(p, p->ptrs, r.in, eo, r.slots, r.T, limit, 1, st, r.rowdst, r.live);
}

extern "C" int cn_moe_mul1_run(void* plan, const unsigned long long* table, const int32_t* ids, const float* wts, const float* shared, const void* x,
                               void* y, int tokens, int topk, int experts, float limit, int dtype, cn_stream_t stream) {
    Mul1Plan* p = (Mul1Plan*)plan;
    if (topk > 32 || topk < 1 || tokens < 1 || tokens > 65535) {  // the fused combine takes a warp per pick
        if (int rc = cn_moe_mul1_experts(plan, table, ids, x, p ? p->eo : nullptr, tokens * topk, topk, experts, limit, dtype, stream)) return rc;
        return cn_moe_combine(p->eo, wts, ids, table, shared, nullptr, y, tokens, p->hidden, topk, experts, dtype, stream);
    }
    if (int rc = check_run(p, tokens * topk, 1, "cn_moe_mul1_run")) return rc;
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_mul1_run: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    cudaStream_t st = (cudaStream_t)stream;
    Mul1Slots r;
    if (int rc = mul1_slots(p, table, ids, x, tokens * topk, topk, experts, dtype, st, r)) return rc;
    if (int rc = mul1_ffn_parts(p, p->ptrs, r.in, r.slots, r.T, limit, st, r.live)) return rc;
    const Mul1Spec d = spec_of(p, 2);
    const dim3 grid(d.n / 128, tokens), block(32 * topk);
    const size_t smem = (size_t)topk * (128 + 2) * 4;
    if (dtype == CN_BF16)
        CN_CUDA(cn_launch_pdl((mul1_out_combine_kernel<1>), grid, block, smem, st, table, ids, wts, p->part_a, shared, y, d.n, ksplit(d.k), r.T, topk, experts, d.svh_off, r.place));
    else
        CN_CUDA(cn_launch_pdl((mul1_out_combine_kernel<0>), grid, block, smem, st, table, ids, wts, p->part_a, shared, y, d.n, ksplit(d.k), r.T, topk, experts, d.svh_off, r.place));
    return CN_OK;
}

extern "C" int cn_mul1_reconstruct(const void* trellis, void* w_out, int k, int n, int bits, int half, cn_stream_t stream) {
    if (k <= 0 || n <= 0 || k % 16 || n % 16) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_reconstruct: [%d, %d] is not a multiple of 16", k, n);
    const int n32 = 8 * bits + (half ? 4 : 0);
    const long long total = (long long)(k / 16) * (n / 16) * 256;
    mul1_reconstruct_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint32_t*)trellis, (uint16_t*)w_out, k, n, bits, half, n32);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

// ---------------------------------------------------------------- allocation-free MUL1 GEMV
// For callers that may not allocate device memory at the point of the call - an engine thread that
// already runs inside a latency-critical decode loop, a plugin host that forbids cudaMalloc after
// start-up because an allocation synchronises the whole device, or code that holds a memory budget
// it has fully handed out. The scratch of the GEMV (the k-split partial sums) lives in a fixed array inside the library image instead of a plan.
//
// Limits: slots * t <= CN_MUL1_STATIC_ROWS (8) activation rows per call, hidden and inter <=
// CN_MUL1_STATIC_DIM (4096). The array is 2 MB and every GPU that loads the library holds
// it until the process exits.
namespace {

constexpr size_t NA_ROWS = 8, NA_DIM = 4096, NA_SPLITS = 16;
constexpr size_t NA_BYTES = NA_ROWS * NA_SPLITS * NA_DIM * 4;  // f32 partial sums of the k-split

// File-scope device array: in host code this name is only a handle for the runtime, never an
// address a kernel may be given; the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_mul1_static_scratch[NA_BYTES];

constexpr int NA_MAX_DEVICES = 64;
unsigned char* g_static_ptr[NA_MAX_DEVICES] = {};

// The device address of the scratch array on the current device, looked up once per device.
int static_scratch(unsigned char** out) {
    int dev = -1;
    CN_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NA_MAX_DEVICES) CN_FAIL(CN_ERR_LIMIT, "cn_mul1_gemv_noalloc: device ordinal %d beyond %d", dev, NA_MAX_DEVICES);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_mul1_static_scratch);
        if (e != cudaSuccess || !p) CN_FAIL(CN_ERR_CUDA, "cn_mul1_gemv_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_static_ptr[dev] = (unsigned char*)p;
    }
    *out = g_static_ptr[dev];
    return CN_OK;
}

}  // namespace

extern "C" int cn_mul1_gemv_noalloc(int which, int hidden, int inter, int bits, int half, const unsigned long long* ptrs, const void* x, void* y,
                                    int slots, int t, int x_div, int dtype, cn_stream_t stream) {
    if (hidden <= 0 || inter <= 0 || hidden % 128 || inter % 128)
        CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv_noalloc: [%d, %d] is not a positive multiple of 128 on both sides", hidden, inter);
    if (bits < 1 || bits > 8 || (half && bits > 3)) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv_noalloc: unsupported bitrate %d%s", bits, half ? ".5" : "");
    if (which < 0 || which > 2 || x_div < 1) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv_noalloc: matrix %d (0 gate, 1 up, 2 down), x_div %d", which, x_div);
    if (slots < 1 || t < 1 || t > MUL1_MAXT || (size_t)slots * t > NA_ROWS)
        CN_FAIL(CN_ERR_LIMIT, "cn_mul1_gemv_noalloc: %d slots x %d rows; the fixed scratch holds %zu rows in all (use a plan for more)", slots, t, NA_ROWS);
    if ((size_t)hidden > NA_DIM || (size_t)inter > NA_DIM)
        CN_FAIL(CN_ERR_LIMIT, "cn_mul1_gemv_noalloc: hidden %d / inter %d beyond the fixed scratch's %zu (use a plan for more)", hidden, inter, NA_DIM);
    // before the first launch: the kernels read x in this type
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_mul1_gemv_noalloc: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    unsigned char* base = nullptr;
    if (int rc = static_scratch(&base)) return rc;
    Mul1Plan view = {};
    view.hidden = hidden, view.inter = inter, view.bits = bits, view.half = half, view.n32 = 8 * bits + (half ? 4 : 0);
    const Mul1Spec s = spec_of(&view, which);
    float* part = (float*)base;
    cudaStream_t st = (cudaStream_t)stream;
    // the GEMV fills every partial that had_out sums, so nothing has to start at zero
    const Mul1Side side = {nullptr, nullptr, part, s.tr_off, s.suh_off};
    const Mul1In in = {x, dtype == CN_BF16, x_div, nullptr, nullptr, nullptr, 0};
    if (int rc = launch_gemv(ptrs, side, nullptr, s, slots, t, 0, st, &in)) return rc;
    dim3 grid(s.n / 128, 1, slots);
    if (dtype == CN_BF16)
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<1>), dim3(grid), dim3(32 * t), 0, st, ptrs, part, y, s.n, ksplit(s.k), t, s.svh_off, (const int*)nullptr));
    else
        CN_CUDA(cn_launch_pdl((mul1_had_out_kernel<0>), dim3(grid), dim3(32 * t), 0, st, ptrs, part, y, s.n, ksplit(s.k), t, s.svh_off, (const int*)nullptr));
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}
