// Shared by the kernels that multiply NVFP4 weights as they are on tcgen05.mma kind::mxf4nvf4 (nvfp4_gemv_tc.cu, nvfp4_rows_tc.cu): PTX wrappers, 256 values
// of an activation row as octal digits, and blocks of 16 multiplied out.
#pragma once
#include "tc5.cuh"

#include <type_traits>

__host__ __device__ constexpr int digits_of(bool f32) { return f32 ? 11 : 8; }

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ uint64_t desc_sf(uint32_t smem_addr) {  // a scale chunk: 32 rows of 16 bytes, no swizzle, 8-row groups 128 B apart
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
// kind::mxf4nvf4: A and B E2M1 (format 1) K-major, UE4M3 scales (0), N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t idesc_bs(int n) { return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }
__device__ __forceinline__ void cp_sf(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// A in tensor memory: a row's 64 values in eight columns of its lane
__device__ __forceinline__ void umma_bs(uint32_t tmem_d, uint32_t ta, uint64_t db, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], [%1], %2, %3, [%4], [%5], p;\n\t}"
        ::"r"(tmem_d), "r"(ta), "l"(db), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_ld2(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld1(uint32_t taddr, uint32_t* v) { asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v[0]) : "r"(taddr) : "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// a row's digits of one chunk
template <bool F32>
__device__ __forceinline__ void tc_ld_digits(uint32_t taddr, uint32_t* v) {
    tc_ld8(taddr, v);
    if (F32) tc_ld2(taddr + 8, v + 8), tc_ld1(taddr + 10, v + 10);
}

// ---------------------------------------------------------------- 256 values of an activation row as digits (a warp; a lane holds eight values)
// bs: the B tile; the row's lines are `row` x the digits of a value + j for digit j. With E the exponent of a block's largest value, a value is q x 2^(E - 21), |q| <= 2^22
// (f32: q x 2^(E - 30), |q| <= 2^31): its digits are the octal digits of q + 44444444 (octal; f32: eleven fours), less four each. The scale byte is 2^(8 - (Emax - E)), Emax
// that of the chunk.
//
// A bf16 value is whole in its digits from 2^-14 of 2^E on, an f32 value from 2^-7 on; smaller ones are off by 2^-22 (f32: 2^-31) of 2^E at most. That is nothing beside the
// large values of a block, but much where one or two stand alone and meet small weights. So a block of which one half (eight values) has none that reaches 2^-8 of the
// largest and the other fewer than three has no digits: the threads that add the chunk multiply it out (`whole_blocks`). So f32 values are off by 2^-24 of the third largest (or of the largest of a half) at most, bf16 ones by 2^-15.
// Rows of 1e4 beside values of size 1, one to a block, weights zero there: f32 3.4e-8 off, with ten digits and no such rule 1.6e-5; such a block is less than one in 1e5 of an FFN's hidden rows (SiLU of deviation 7 times its like; the look at its values one in 300), none of normally distributed ones. The same goes for blocks below
// 2^-17 of their chunk's largest value or below 2^-99, and for those with an infinity or NaN.
// fs[row]: 2^(Emax - 8) and the blocks without digits (block b: bit 2 b).
constexpr float TO_INT = 12582912.0f;  // 3 x 2^22: a sum with it has the nearest whole number in its mantissa (ties to even)

template <bool F32, bool RECORD = false>
__device__ __forceinline__ void to_digits(const uint4* raw, int lane, uint8_t* bs, uint8_t* sf, int row, float2* fs) {
    constexpr int LV = digits_of(F32);
    constexpr uint32_t LEAST = 28u, EXP = F32 ? 23u : 7u;  // least biased E: all scales are numbers
    uint32_t u[F32 ? 8 : 4], mine;  // the lane's largest value
    u[0] = raw[0].x, u[1] = raw[0].y, u[2] = raw[0].z, u[3] = raw[0].w;
    if constexpr (F32) {
        u[4] = raw[1].x, u[5] = raw[1].y, u[6] = raw[1].z, u[7] = raw[1].w;
        mine = u[0] & 0x7fffffffu;
#pragma unroll
        for (int i = 1; i < 8; i++) mine = max(mine, u[i] & 0x7fffffffu);
    } else {
        mine = __vmaxu2(__vmaxu2(u[0] & 0x7fff7fffu, u[1] & 0x7fff7fffu), __vmaxu2(u[2] & 0x7fff7fffu, u[3] & 0x7fff7fffu));
        mine = max(mine >> 16, mine & 0xffffu);
    }
    const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1), top = max(mine, other);  // two lanes hold a block of 16
    uint32_t e = top >> EXP;
    bool none = e == 255u;  // infinity, NaN
    const uint32_t emax = max(__reduce_max_sync(0xffffffffu, none ? 0u : e), LEAST);
    const uint32_t limit = (max(e, 9u) - 8u) << EXP;
    none |= top != 0u && (e + 17u < emax || e < LEAST);
    uint32_t blocks = 0u;
    if (__any_sync(0xffffffffu, none || (top != 0u && min(mine, other) < limit))) {
        int large = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) large += (F32 ? u[i] & 0x7fffffffu : (u[i >> 1] >> (16 * (i & 1))) & 0x7fffu) >= limit;
        large += __shfl_xor_sync(0xffffffffu, large, 1);
        none |= top != 0u && min(mine, other) < limit && large < 3;
        blocks = __ballot_sync(0xffffffffu, none) & 0x55555555u;
#pragma unroll
        for (int i = 0; i < (F32 ? 8 : 4); i++) u[i] = none ? 0u : u[i];
    }
    if (none || top == 0u) e = emax;
    const float scale = __uint_as_float(((F32 ? 266u : 275u) - e) << 23);  // 2^(21 - (e - 127)), f32: 12
    uint32_t lo[4], hi[4], over[4];  // value pair p: byte j = digits j (hi: 4 + j; over: 8 + j) of both
#pragma unroll
    for (int p = 0; p < 4; p++) {
        uint32_t sel[2], up[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float v = __uint_as_float(F32 ? u[F32 ? 2 * p + h : p] : h ? u[p] & 0xffff0000u : u[p] << 16);
            uint32_t q;
            if constexpr (F32) {
                // five digits of the value in units of 2^(E - 12), six of what is left, which may reach beyond them by one
                const float t = fmaf(v, scale, TO_INT), w = fmaf(fmaf(v, scale, TO_INT - t), 262144.0f, TO_INT);
                const uint32_t lq = __float_as_uint(w) + (0444444u - 0x4b400000u), hq = __float_as_uint(t) + (044444u - 0x4b400000u) + (lq >> 18);
                q = (lq & 0x3ffffu) | ((hq & 0x3fu) << 18);
                uint32_t x = hq >> 6;
                x += (x & 0xfc0u) * 3u;
                up[h] = x + (x & 0x3838u);
            } else {
                q = __float_as_uint(fmaf(v, scale, TO_INT)) + (044444444u - 0x4b400000u);
            }
            q += (q & 0x00fff000u) * 15u;  // octal digits apart: four to sixteen bits, two to eight, one to four
            q += (q & 0x0fc00fc0u) * 3u;
            q += q & 0x38383838u;
            sel[h] = q;
        }
        // digit d - 4 as E2M1: -4 .. 3 = E D C A 0 2 4 5; the even value's in the low nibble
        lo[p] = __byte_perm(0x0A0C0D0Eu, 0x05040200u, sel[0]) | __byte_perm(0xA0C0D0E0u, 0x50402000u, sel[1]);
        hi[p] = __byte_perm(0x0A0C0D0Eu, 0x05040200u, sel[0] >> 16) | __byte_perm(0xA0C0D0E0u, 0x50402000u, sel[1] >> 16);
        if constexpr (F32) over[p] = __byte_perm(0x0A0C0D0Eu, 0x05040200u, up[0]) | __byte_perm(0xA0C0D0E0u, 0x50402000u, up[1]);
    }
    const uint32_t at = (uint32_t)(lane >> 2), in = (uint32_t)(lane & 3) * 4u;
    auto put = [&](int j, uint32_t w) {
        const uint32_t n = (uint32_t)(row * LV + j);
        *(uint32_t*)(bs + n * 128u + ((at ^ (F32 ? n & 7u : (uint32_t)j)) << 4) + in) = w;
    };
#pragma unroll
    for (int h = 0; h < (F32 ? 3 : 2); h++) {
        const uint32_t* s = h == 0 ? lo : h == 1 ? hi : over;
        const uint32_t a = __byte_perm(s[0], s[1], 0x5140), b = __byte_perm(s[2], s[3], 0x5140);
        const uint32_t c = __byte_perm(s[0], s[1], 0x7362), d = __byte_perm(s[2], s[3], 0x7362);
        put(4 * h, __byte_perm(a, b, 0x5410));
        put(4 * h + 1, __byte_perm(a, b, 0x7632));
        put(4 * h + 2, __byte_perm(c, d, 0x5410));
        if (4 * h + 3 < LV) put(4 * h + 3, __byte_perm(c, d, 0x7632));
    }
    const uint32_t under = emax - e;  // 0..17: 2^8 .. 2^-9, the last three subnormal
    uint32_t sw = (under <= 14u ? (15u - under) << 3 : 32u >> (under - 12u)) << (8 * ((lane >> 1) & 3));
    sw |= __shfl_xor_sync(0xffffffffu, sw, 2);
    sw |= __shfl_xor_sync(0xffffffffu, sw, 4);
    if constexpr (RECORD) {
        if ((lane & 7) == 0) ((uint32_t*)sf)[lane >> 3] = sw;
    } else {
        int n = row * LV + (lane & 7);
        *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = sw;
        if ((lane & 7) < LV - 8) {
            n += 8;
            *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = sw;
        }
    }
    if (lane == 0) *fs = make_float2(__uint_as_float((emax - 8u) << 23), __uint_as_float(blocks));
}

// The same kept in global memory, for matrices of many tiles, which would each make the digits of their rows: the lines as of row 0, four words of scales, factor and blocks without digits.
__host__ __device__ constexpr int digit_record(bool f32) { return digits_of(f32) * 128 + 32; }
template <bool F32>
struct ChunkValues {  // a lane's eight values of a chunk
    static constexpr int XR = F32 ? 2 : 1;
    uint4 v[XR];
    __device__ __forceinline__ void load(const void* x, int lane) {  // x: the chunk's 256 values
#pragma unroll
        for (int j = 0; j < XR; j++) v[j] = __ldcg((const uint4*)x + lane * XR + j);
    }
};
template <bool F32>
__device__ __forceinline__ void put_record(const ChunkValues<F32>& c, int lane, uint8_t* rec) {
    to_digits<F32, true>(c.v, lane, rec, rec + digits_of(F32) * 128, 0, (float2*)(rec + digits_of(F32) * 128 + 16));
}
template <bool F32>
struct DigitRecord {  // a lane's part of one
    static constexpr int PIECES = digits_of(F32) * 8, PER = (PIECES + 31) / 32;
    uint4 code[PER];
    uint32_t scales;
    float2 f;
    __device__ __forceinline__ void load(const uint8_t* rec, int lane) {
#pragma unroll
        for (int p = 0; p < PER; p++)
            if (lane + 32 * p < PIECES) code[p] = __ldcg((const uint4*)rec + lane + 32 * p);
        scales = __ldcg((const uint32_t*)(rec + PIECES * 16) + (lane >> 3));
        f = __ldcg((const float2*)(rec + PIECES * 16 + 16));
    }
    __device__ __forceinline__ void store(int lane, uint8_t* bs, uint8_t* sf, int row, float2* fs) const {
        constexpr int LV = digits_of(F32);
#pragma unroll
        for (int p = 0; p < PER; p++) {
            const int id = lane + 32 * p, j = id >> 3, n = row * LV + j;
            if (id < PIECES) *(uint4*)(bs + n * 128 + ((((id & 7) ^ j ^ n) & 7) << 4)) = code[p];
        }
        int n = row * LV + (lane & 7);
        *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = scales;
        if ((lane & 7) < LV - 8) {
            n += 8;
            *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = scales;
        }
        if (lane == 0) *fs = f;
    }
};

// a chunk's factor in 64 bits (a normal power of two)
__device__ __forceinline__ double power_of_two(float f) { return __hiloint2double((int)((__float_as_uint(f) >> 3) + (896u << 20)), 0); }

// ---------------------------------------------------------------- container blocks -> operand layout (a lane: the four blocks of a row)
constexpr int A_COLS = 32, A_SCALES = 4 * 512;  // a chunk of 128 rows as operand A: columns of tensor memory with its codes, bytes of the four MMAs' scales

// A row's 144 bytes at src into registers, scale bytes as the tensor core is to read them; whether any row of the warp has one of 0xFF: that stands for 480, which it does not know, and is
// nothing here (`whole_blocks` multiplies the block out).
__device__ __forceinline__ uint32_t load_row(const uint4* src, uint32_t (&v)[36]) {
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const uint4 q = src[j];
        v[4 * j] = q.x, v[4 * j + 1] = q.y, v[4 * j + 2] = q.z, v[4 * j + 3] = q.w;
    }
    uint32_t odd = 0u;
#pragma unroll
    for (int b = 0; b < 4; b++) odd |= v[9 * b] & ((v[9 * b] & 0x7f7f7f7fu) + 0x01010101u);
    odd = __any_sync(0xffffffffu, (odd & 0x80808080u) != 0u);
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const uint32_t sc = v[9 * b];
        v[9 * b] = scale_bytes_rule(sc);
        if (odd) {
            const uint32_t ff = sc & ((sc & 0x7f7f7f7fu) + 0x01010101u) & 0x80808080u;
            v[9 * b] &= ~(ff - (ff >> 7));
        }
    }
    return odd;
}
__device__ __forceinline__ void store_scales(uint8_t* dst, int row, const uint32_t (&v)[36]) {
#pragma unroll
    for (int b = 0; b < 4; b++) *(uint32_t*)(dst + b * 512 + (row & 31) * 16 + (row >> 5) * 4) = v[9 * b];
}
// Row 32 w + lane of the operand: its codes into A_COLS columns of tensor memory, of which a warp reaches 32 lanes, its scales into shared memory, from where the issuing thread has them copied.
// Laid out in shared memory, as operand A by descriptor, the codes went through it twice more (stored, read by the MMA), and it was what a chunk used most: us, so / now, one row of gate / up of
// 17408 x 5120 19.1 / 17.6, four rows 23.9 / 22.1; 4096 x 4096 4.6 / 4.2; 64 layers of 5120 x 17408 2811 / 2488.
__device__ __forceinline__ void store_row(uint32_t taddr, uint8_t* scales, int w, int lane, const uint32_t (&v)[36]) {
    uint32_t codes[32];
#pragma unroll
    for (int i = 0; i < 32; i++) codes[i] = v[9 * (i >> 3) + 1 + (i & 7)];
    tc_after();  // (the MMAs that read these columns are done)
    tc_st32(taddr + ((uint32_t)(w * 32) << 16), codes);
    store_scales(scales, 32 * w + lane, v);
    tc_wait_st();
    tc_before();
}

// ---------------------------------------------------------------- sums
// A row's columns of digits into its sum over the chunk, in units of the highest digit: from the smallest up; f32: what the last two additions round off into `rest`.
template <bool F32>
__device__ __forceinline__ float sum_digits(const uint32_t* d, float& rest) {
    constexpr int LV = digits_of(F32), PLAIN = F32 ? LV - 2 : LV;
    float s = __uint_as_float(d[0]);
    rest = 0.0f;
#pragma unroll
    for (int j = 1; j < PLAIN; j++) s = fmaf(s, 0.125f, __uint_as_float(d[j]));
#pragma unroll
    for (int j = PLAIN; j < LV; j++) {
        const float a = s * 0.125f, b = __uint_as_float(d[j]);
        s = a + b;
        const float bb = s - a;
        rest = rest * 0.125f + ((a - (s - bb)) + (b - bb));
    }
    return s;
}

// Blocks of 16 without digits (`blocks`, bit 2 b) and, where `odd`, those whose scale byte is 0xFF (480, which the tensor core does not know and is given as nothing), from global memory: the
// row's 144 container bytes at wr times 256 values at x. All that a block (bf16: two blocks) needs is
// asked for at once: what it costs is the way to memory. f32: products and sums in 64 bits. One row of gate / up 17408 x 5120 with a NaN 21.9 -> 22.6 us, 4096 x 4096 4.7 -> 6.3;
// eight rows with a value of 1e4 in the same place 37 -> 49 us.
template <bool F32>
static __device__ __noinline__ typename std::conditional<F32, double, float>::type whole_blocks(const uint8_t* wr, uint32_t blocks, bool odd, const void* x) {
    using Acc = typename std::conditional<F32, double, float>::type;
    constexpr int XR = F32 ? 4 : 2, NB = F32 ? 1 : 2;
    if (odd) {
        uint32_t s[4];
#pragma unroll
        for (int g = 0; g < 4; g++) s[g] = __ldcg((const uint32_t*)(wr + 36 * g));
#pragma unroll
        for (int b = 0; b < 16; b++) blocks |= ((s[b >> 2] >> (8 * (b & 3))) & 0xffu) == 0xffu ? 1u << (2 * b) : 0u;
    }
    Acc sum = 0;
    while (blocks) {
        uint32_t scale[NB], code[NB][2];
        uint4 v[NB][XR];
#pragma unroll
        for (int h = 0; h < NB; h++) {
            const int b = blocks ? (__ffs(blocks) - 1) >> 1 : -1;
            blocks &= blocks - 1u;
            if (b >= 0) {
                const uint8_t* blk = wr + 36 * (b >> 2);
                scale[h] = __ldcg((const uint32_t*)blk) >> (8 * (b & 3)) & 0xffu;
                code[h][0] = __ldcg((const uint32_t*)(blk + 4) + 2 * (b & 3)), code[h][1] = __ldcg((const uint32_t*)(blk + 4) + 2 * (b & 3) + 1);
#pragma unroll
                for (int i = 0; i < XR; i++) v[h][i] = __ldcg((const uint4*)x + b * XR + i);
            } else {
                scale[h] = code[h][0] = code[h][1] = 0u;
#pragma unroll
                for (int i = 0; i < XR; i++) v[h][i] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
#pragma unroll
        for (int h = 0; h < NB; h++) {
            Acc t = 0;
            uint32_t w[8];
            e2m1x8_to_f16x2(code[h][0], w), e2m1x8_to_f16x2(code[h][1], w + 4);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const uint4 q = v[h][i / (F32 ? 4 : 8)];
                const int wd = F32 ? i & 3 : (i >> 1) & 3;
                const uint32_t bits = wd == 0 ? q.x : wd == 1 ? q.y : wd == 2 ? q.z : q.w;
                const float xv = __uint_as_float(F32 ? bits : (i & 1) ? bits & 0xffff0000u : bits << 16);
                t += (Acc)((i & 1) ? f16hi_to_f32(w[i >> 1]) : f16lo_to_f32(w[i >> 1])) * (Acc)xv;
            }
            sum += t * (Acc)ue4m3_f32(scale[h], true);
        }
    }
    return sum;
}
