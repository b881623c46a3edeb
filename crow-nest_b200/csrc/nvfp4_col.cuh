// Device helpers of the kernels whose activation rows are MMA columns (moe_step.cu): weights with their scale
// applied in f16 (exact), f32 activations as three f16 planes.
#pragma once
#include "common.cuh"

// Two scale bytes of a word, `shift` = 8 (t >> 1): bytes t >> 1 and 2 + (t >> 1), as f16x2 of scale x 2^-8: an E4M3 byte shifted left by
// seven is that f16 as it stands, subnormals included. The engine's reading: bit 7 ignored, 0x7F read as 0x7E.
__device__ __forceinline__ __half2 lane_scales(uint32_t w, uint32_t shift) {
    uint32_t r = (w >> shift) & 0x007f007fu;
    asm("min.u16x2 %0, %0, %1;" : "+r"(r) : "r"(0x007e007eu));
    r <<= 7;
    return *(const __half2*)&r;
}
// One 64-value block of 16 weight rows times NP groups of eight columns -> cc. Inside an MMA the order of k is free as long as
// A and B agree: lane (g, t) takes code words t and t + 4 of rows g (pa, the block's start + 4 t) and g + 8 (pb) - one 32-bit load of
// eight codes feeds half of two MMAs - and x(ps, half) gives the matching eight activations of column g of group ps. A word's
// eight values share a scale, so the two words' scales are made in one register (four instructions) and the multiplies take its halves
// (measured in a kernel for groups of rows: a step of 64 tokens 258 us with one scale at a time, 245 with two).
template <int NP, typename X>
__device__ __forceinline__ void block_mma(float (&cc)[NP][4], const uint8_t* pa, const uint8_t* pb, int t, X x) {
    const __half2 sa = lane_scales(*(const uint32_t*)(pa - 4 * t), 8u * (t >> 1)), sb = lane_scales(*(const uint32_t*)(pb - 4 * t), 8u * (t >> 1));
#pragma unroll
    for (int ps = 0; ps < NP; ps++) cc[ps][0] = cc[ps][1] = cc[ps][2] = cc[ps][3] = 0.0f;
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
        uint32_t ha[4], hb[4];
        e2m1x8_to_f16x2(*(const uint32_t*)(pa + 4 + 16 * hf), ha);
        e2m1x8_to_f16x2(*(const uint32_t*)(pb + 4 + 16 * hf), hb);
        const __half2 fa = hf ? __high2half2(sa) : __low2half2(sa), fb = hf ? __high2half2(sb) : __low2half2(sb);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const __half2 va = __hmul2(*(const __half2*)&ha[i], fa), vb = __hmul2(*(const __half2*)&hb[i], fb);
            ha[i] = *(const uint32_t*)&va, hb[i] = *(const uint32_t*)&vb;
        }
#pragma unroll
        for (int ps = 0; ps < NP; ps++) {
            const uint4 xv = x(ps, hf);
            mma16816(cc[ps], ha[0], hb[0], ha[1], hb[1], xv.x, xv.y);
            mma16816(cc[ps], ha[2], hb[2], ha[3], hb[3], xv.z, xv.w);
        }
    }
}
// the power of two of a tensor scale (1 where it has none)
__device__ __forceinline__ float gs_pow2(float gs) {
    const uint32_t e = (__float_as_uint(gs) >> 23) & 0xFF;
    return e > 0 && e < 255 ? __uint_as_float(e << 23) : 1.0f;
}

// Eight f32 values of a 64-value block, eight consecutive lanes (lane & 24 the same) holding the block: the block's power-of-two
// scale, and three f16 planes: the value on the block's own grid of 2^5 (values below 2^15 after scaling), then what is left as
// f16, twice. An infinity or a NaN goes into the first plane and leaves nothing. Returns the inverse scale, times the 2^8 that
// lane_scales leaves out.
__device__ __forceinline__ float f32_planes(const uint4& lo, const uint4& hi, int lane, uint32_t h[3][4]) {
    const uint32_t u[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t e = 0;  // largest exponent of the block's finite values
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t ev = (u[q] >> 23) & 0xFF;
        e = max(e, ev == 255u ? 0u : ev);
    }
    const uint32_t gm = 0xffu << (lane & 24);
    e = max(e, __shfl_xor_sync(gm, e, 1));
    e = max(e, __shfl_xor_sync(gm, e, 2));
    e = max(e, __shfl_xor_sync(gm, e, 4));
    e = e < 15 ? 15 : e;
    const float mul = __uint_as_float((268u - e) << 23);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float a = __uint_as_float(u[2 * q]) * mul, c = __uint_as_float(u[2 * q + 1]) * mul;
        const bool fa = fabsf(a) < 65536.0f, fc = fabsf(c) < 65536.0f;
        const float ga = fa ? __fsub_rn(__fadd_rn(a, 402653184.0f), 402653184.0f) : a;  // 1.5 x 2^28
        const float gc = fc ? __fsub_rn(__fadd_rn(c, 402653184.0f), 402653184.0f) : c;
        const __half2 h0 = __floats2half2_rn(ga, gc);
        a = fa ? (a - ga) * 2048.0f : 0.0f, c = fc ? (c - gc) * 2048.0f : 0.0f;
        const __half2 h1 = __floats2half2_rn(a, c);
        const __half2 h2 = __floats2half2_rn((a - __low2float(h1)) * 2048.0f, (c - __high2float(h1)) * 2048.0f);
        h[0][q] = *(const uint32_t*)&h0, h[1][q] = *(const uint32_t*)&h1, h[2][q] = *(const uint32_t*)&h2;
    }
    return __uint_as_float((e - 6u) << 23);
}
