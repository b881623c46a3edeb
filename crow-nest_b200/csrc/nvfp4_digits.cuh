// Shared by the kernels that multiply NVFP4 weights as they are on tcgen05.mma kind::mxf4nvf4 (nvfp4_gemv_tc.cu, nvfp4_rows_tc.cu): PTX wrappers, 256 values
// of an activation row as octal digits, and a block of 16 multiplied out in f32.
#pragma once
#include "tc5.cuh"

__host__ __device__ constexpr int digits_of(bool f32) { return f32 ? 10 : 8; }

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ uint64_t desc_sf(uint32_t smem_addr) {  // a scale chunk: 32 rows of 16 bytes, no swizzle, 8-row groups 128 B apart
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
// kind::mxf4nvf4: A and B E2M1 (format 1) K-major, UE4M3 scales (0), N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t idesc_bs(int n) { return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }
__device__ __forceinline__ void cp_sf(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_bs(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
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
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---------------------------------------------------------------- 256 values of an activation row as digits (a warp; a lane holds eight values)
// bs: the B tile; the row's lines are `row` x the digits of a value + j for digit j. With E the exponent of a block's largest value, a value is
// q x 2^(E - 21), |q| <= 2^22 (f32: q x 2^(E - 27), |q| <= 2^28): its digits are the octal digits of q + 44444444 (octal; f32: ten fours), less four
// each. The scale byte is 2^(8 - (Emax - E)), Emax that of the chunk.
template <bool F32>
__device__ __forceinline__ void to_digits(const uint4* raw, int lane, uint8_t* bs, uint8_t* sf, int row, float2* fs) {
    constexpr int LV = digits_of(F32);
    constexpr uint32_t LEAST = F32 ? 28u : 22u;  // biased exponent below which the scale of a block would be no number
    uint32_t u[F32 ? 8 : 4], top;
    u[0] = raw[0].x, u[1] = raw[0].y, u[2] = raw[0].z, u[3] = raw[0].w;
    if constexpr (F32) {
        u[4] = raw[1].x, u[5] = raw[1].y, u[6] = raw[1].z, u[7] = raw[1].w;
        top = u[0] & 0x7fffffffu;
#pragma unroll
        for (int i = 1; i < 8; i++) top = max(top, u[i] & 0x7fffffffu);
    } else {
        top = __vmaxu2(__vmaxu2(u[0] & 0x7fff7fffu, u[1] & 0x7fff7fffu), __vmaxu2(u[2] & 0x7fff7fffu, u[3] & 0x7fff7fffu));
        top = max(top >> 16, top & 0xffffu);
    }
    top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));  // two lanes hold a block of 16
    uint32_t e = top >> (F32 ? 23 : 7);
    const bool odd = top != 0u && (e < LEAST || e == 255u);  // too small, infinity, NaN
    const uint32_t emax = max(__reduce_max_sync(0xffffffffu, odd ? 0u : e), LEAST);
    const bool slow = odd || (top != 0u && emax - e > 17u);
    const uint32_t slow_lanes = __ballot_sync(0xffffffffu, slow);
    if (slow || top == 0u) {
        e = emax;
#pragma unroll
        for (int i = 0; i < (F32 ? 8 : 4); i++) u[i] = 0u;
    }
    const float scale = __uint_as_float(((F32 ? 281u : 275u) - e) << 23);  // 2^(21 - (e - 127)), f32: 27
    uint32_t lo[4], hi[4], over[4];  // value pair p: byte j = digits j (hi: 4 + j; over: 8 + j) of both
#pragma unroll
    for (int p = 0; p < 4; p++) {
        uint32_t sel[2], up[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t q;
            if constexpr (F32) {
                q = (uint32_t)(__float2int_rn(__uint_as_float(u[2 * p + h]) * scale) + 04444444444);
                up[h] = q >> 24;
                up[h] += up[h] & 0x38u;
                q &= 0x00ffffffu;
            } else {
                const float v = __uint_as_float(h ? u[p] & 0xffff0000u : u[p] << 16);
                q = __float_as_uint(fmaf(v, scale, 12582912.0f)) + (044444444u - 0x4b400000u);  // (q + 2^22 is the sum's mantissa: rounded to nearest even)
            }
            q += (q & 0x00fff000u) * 15u;  // octal digits apart: four to sixteen bits, two to eight, one to four
            q += (q & 0x0fc00fc0u) * 3u;
            q += q & 0x38383838u;
            sel[h] = q;
        }
        // digit d - 4 as E2M1: -4 .. 3 = E D C A 0 2 4 5; the even value's in the low nibble
        lo[p] = __byte_perm(0x0A0C0D0Eu, 0x05040200u, sel[0]) | __byte_perm(0xA0C0D0E0u, 0x50402000u, sel[1]);
        hi[p] = __byte_perm(0x0A0C0D0Eu, 0x05040200u, sel[0] >> 16) | __byte_perm(0xA0C0D0E0u, 0x50402000u, sel[1] >> 16);
        if constexpr (F32) {
            const uint32_t c = __byte_perm(0x0A0C0D0Eu, 0x05040200u, up[0] | (up[1] << 8));  // even 8, even 9, odd 8, odd 9
            over[p] = c | (c >> 12);
        }
    }
    const uint32_t at = (uint32_t)(lane >> 2), in = (uint32_t)(lane & 3) * 4u;
    auto put = [&](int j, uint32_t w) {
        if constexpr (F32) {
            const uint32_t n = (uint32_t)(row * LV + j), r = n & 7u;
            *(uint32_t*)(bs + n * 128u + ((at ^ r) << 4) + in) = w;
        } else {
            *(uint32_t*)(bs + row * 1024 + j * 128 + ((at ^ (uint32_t)j) << 4) + in) = w;
        }
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t* s = h ? hi : lo;
        const uint32_t a = __byte_perm(s[0], s[1], 0x5140), b = __byte_perm(s[2], s[3], 0x5140);
        const uint32_t c = __byte_perm(s[0], s[1], 0x7362), d = __byte_perm(s[2], s[3], 0x7362);
        put(4 * h, __byte_perm(a, b, 0x5410));
        put(4 * h + 1, __byte_perm(a, b, 0x7632));
        put(4 * h + 2, __byte_perm(c, d, 0x5410));
        put(4 * h + 3, __byte_perm(c, d, 0x7632));
    }
    if constexpr (F32) {
        const uint32_t a = __byte_perm(over[0], over[1], 0x5140), b = __byte_perm(over[2], over[3], 0x5140);
        put(8, __byte_perm(a, b, 0x5410));
        put(9, __byte_perm(a, b, 0x7632));
    }
    const uint32_t under = emax - e;  // 0..17: 2^8 .. 2^-9, the last three subnormal
    uint32_t sw = (under <= 14u ? (15u - under) << 3 : 32u >> (under - 12u)) << (8 * ((lane >> 1) & 3));
    sw |= __shfl_xor_sync(0xffffffffu, sw, 2);
    sw |= __shfl_xor_sync(0xffffffffu, sw, 4);
    int n = row * LV + (lane & 7);
    *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = sw;
    if (F32 && (lane & 7) < LV - 8) {
        n += 8;
        *(uint32_t*)(sf + (lane >> 3) * 512 + (n & 31) * 16 + (n >> 5) * 4) = sw;
    }
    if (lane == 0) *fs = make_float2(__uint_as_float((emax - 8u) << 23), __uint_as_float(slow_lanes));  // 2^(Emax - 8)
}

// one block of 16 values from global memory: sum of code x activation, times the block's scale
template <bool F32>
static __device__ __noinline__ float slow_block(const uint8_t* wblk, int sub, const void* x) {
    float sum = 0.0f;
    for (int i = 0; i < 16; i++) {
        const uint32_t b = wblk[4 + sub * 8 + (i >> 1)], n = (i & 1) ? b >> 4 : b & 15u, c = n & 7u;
        const float v = c < 2u ? 0.5f * (float)c : __uint_as_float(((126u + (c >> 1)) << 23) | ((c & 1u) << 22));
        const float xv = F32 ? __ldcg((const float*)x + i) : __uint_as_float((uint32_t)__ldcg((const unsigned short*)x + i) << 16);
        sum = fmaf((n & 8u) ? -v : v, xv, sum);
    }
    return sum * ue4m3_f32(wblk[sub], true);
}

