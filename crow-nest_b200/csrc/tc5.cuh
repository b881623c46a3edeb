// Fifth-generation tensor-core helpers shared by the kernels that decode NVFP4 weights into tensor memory: tcgen05 and
// TMA PTX wrappers, the host side of a 2-D tensor map, and the register decode of one 64-value NVFP4 block.
#pragma once
#include <cuda.h>

#include "common.cuh"

// ---------------------------------------------------------------- host: tensor maps (elements beyond the matrix read as zero)
// Rows of `words` 32-bit words (a multiple of four) one after another, in boxes of box_words words x box_rows rows, no swizzle: NVFP4 container bytes.
int cn_tmap_words(CUtensorMap* map, const void* base, unsigned long long words, unsigned long long rows, unsigned box_words, unsigned box_rows);
// A row-major matrix of 16-bit values (bf16 or f16), rows row_bytes apart (a multiple of 16), as blocks of 64 columns: coordinates (column of a block, row, block), boxes of box_rows rows
// and box_blocks blocks with 128-byte swizzle, each block a K-major operand tile of an MMA.
int cn_tmap_blocks(CUtensorMap* map, const void* base, bool bf16, unsigned long long blocks, unsigned long long rows, unsigned long long row_bytes, unsigned box_rows,
                   unsigned box_blocks);

// ---------------------------------------------------------------- device: TMA and clusters
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* m) { asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory"); }
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(m), "r"(x),
                 "r"(y), "r"(bar)
                 : "memory");
}
// from either CTA of a pair; `bar` may name the even CTA's barrier (peer bit cleared)
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* m, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(m), "r"(x),
        "r"(y), "r"(z), "r"(bar)
        : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_ctas() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }
// shared::cluster address of a local shared address in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// Arrival on another CTA's barrier for work that the tensor core orders itself (tensor-memory stores before
// tcgen05.fence::before_thread_sync): no generic-memory data rides on it, so CTA scope is enough. A cluster-scope release
// here and cluster-scope acquires in the waits cost a fence each, several hundred cycles per 64 values of K.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// ---------------------------------------------------------------- device: tcgen05
// shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: start address >> 4, leading byte offset 1
// (unused by swizzled K-major tiles), stride byte offset = 8 rows * 128 B, descriptor version 1, layout 2
__device__ __forceinline__ uint64_t tc_desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// instruction descriptor of kind::f16: D f32 (bit 4), A and B both f16 (0) or both bf16 (1) at bits 7 and 10, K-major,
// N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t tc_idesc_f16(int m, int n, bool bf16) {
    return (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// D (tensor memory) (+)= A (tensor memory: lane = row, 32-bit column = two K values) x B (shared memory)
template <int CG>
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if (CG == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(accumulate)
            : "memory");
}
// One lane of a converged warp, chosen in hardware. The issuing warp runs its loop as a whole, with operands that are
// uniform over the warp, and only the instruction itself sits behind this predicate: the descriptors then stay in uniform
// registers. A loop behind `lane == 0` moves every operand there one by one: 78 cycles per MMA measured against 27.
__device__ __forceinline__ bool elect_lane() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
// arrive on `bar` (of both CTAs of a pair for CG = 2) when the MMAs issued so far are done
template <int CG>
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                     "h"((uint16_t)3)
                     : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <int CG>
__device__ __forceinline__ void tc_alloc(uint32_t* slot, uint32_t cols) {
    if (CG == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <int CG>
__device__ __forceinline__ void tc_dealloc(uint32_t tmem, uint32_t cols) {
    if (CG == 2)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    else
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
// 32 lanes x 32 columns, asynchronous until tc_wait_ld
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t v[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// the calling warp's 32 lanes x 32 columns <- registers, asynchronous until tc_wait_st
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t v[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
        "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
        "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- device: one 64-value block -> 32 registers of two values
// w[0] = the four UE4M3 scale bytes, w[1..8] = the code words. Scale byte 0x7F reads as 0x7E; of the others bit 7 is ignored.
__device__ __forceinline__ uint32_t scale_bytes_rule(uint32_t s) {
    const uint32_t t = s & 0x7f7f7f7fu;
    return t - ((((t + 0x01010101u) & ~s) >> 7) & 0x01010101u);
}
// f16: code x scale x 2^-8, exact: cvt to f16x2 and one HMUL2 per pair; a scale byte shifted left by seven IS the f16 of
// scale x 2^-8, subnormals included. The caller multiplies the sums by F16_UNSCALE.
constexpr float F16_UNSCALE = 256.0f;
__device__ __forceinline__ void decode64_f16(const uint32_t w[9], uint32_t v[32]) {
    const uint32_t sw = scale_bytes_rule(w[0]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t sb = __byte_perm(sw, 0u, 0x4040 | (i >> 1) | ((i >> 1) << 8)) << 7;
        e2m1x8_to_f16x2(w[1 + i], v + 4 * i);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const __half2 p = __hmul2(*(const __half2*)&v[4 * i + q], *(const __half2*)&sb);
            v[4 * i + q] = *(const uint32_t*)&p;
        }
    }
}
// bf16: code x scale x 2^-12, exact (six significant bits at most). A code's magnitude x 2^108 comes from two byte-permute
// tables (high and low byte of the bf16), its sign from the nibble's top bit; a scale byte shifted left by four IS the
// bf16 of scale x 2^-120, subnormals included. The caller multiplies the sums by BF16_UNSCALE.
// Why 2^-12: the activations are not scaled per row, so the f32 sums see them as they are. The largest weight becomes 2688 x 2^-12 < 1:
// no sum of 2^15 products overflows for rows up to 2^113; and rows down to 2^-112 keep 20 bits and more above the last subnormal f32
// (the tensor core keeps subnormals; measured with 2^-60, where rows of 2^-80 lost a percent and rows below 2^-96 all). Those are
// the rows that a power of two per row could bring to f16.
constexpr float BF16_UNSCALE = 4096.0f;  // 2^12
__device__ __forceinline__ void decode64_bf16(const uint32_t w[9], uint32_t v[32]) {
    const uint32_t sw = scale_bytes_rule(w[0]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int sbi = i >> 1;
        const uint32_t sb = __byte_perm(sw, 0u, 0x4040 | sbi | (sbi << 8)) << 4;
        const uint32_t cw = w[1 + i], mag = cw & 0x77777777u, up = cw << 4;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t sel = h ? mag >> 16 : mag;
            const uint32_t hi = __byte_perm(0x75757500u, 0x76767676u, sel);
            const uint32_t lo = __byte_perm(0xC0800000u, 0xC0804000u, sel);
            const uint32_t sg = __byte_perm(up, cw, h ? 0x7362 : 0x5140);
            const uint32_t hs = hi | (sg & 0x80808080u);
            const uint32_t a = __byte_perm(lo, hs, 0x5140), b = __byte_perm(lo, hs, 0x7362);
            const __nv_bfloat162 pa = __hmul2(*(const __nv_bfloat162*)&a, *(const __nv_bfloat162*)&sb);
            const __nv_bfloat162 pb = __hmul2(*(const __nv_bfloat162*)&b, *(const __nv_bfloat162*)&sb);
            v[4 * i + 2 * h] = *(const uint32_t*)&pa;
            v[4 * i + 2 * h + 1] = *(const uint32_t*)&pb;
        }
    }
}
