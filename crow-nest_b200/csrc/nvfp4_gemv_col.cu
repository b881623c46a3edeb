// NVFP4 GEMV whose activation rows are columns of the tensor-core tile: Y[m][n] = sum_k W[n][k] X[m][k], m = 1..8 f32 rows.
//
// Supersedes gemv_nvfp4_w / _gu / _wm / _gum (engine/src/kernels_p2.rs:355-530) for f32 activations.
//
// Arithmetic. An E2M1 code times its UE4M3 scale has six significant bits and is exact in f16, so a weight enters the MMA
// with its scale applied (one HMUL2 per two weights) and a 64-value block needs a single f32 scale step per column. An f32
// activation is split into three f16 planes over a power-of-two scale per 64-value block: the value on a grid of 2^-10 of
// the block's largest binade, then what is left rounded to f16, twice: all 24 bits of a value within 2^10 of the block's largest, 23
// of one within 2^38, and below that (the last plane is a subnormal f16) an error of at most 2^-60 of the largest. Each plane is a column and the three sums are added at the end. Products are exact,
// accumulation is the tensor core's f32 inside a block and f32 FMAs across blocks; the tensor core cuts every product at
// 2^-24 of the largest, which the coarse grid keeps the first plane clear of (as a rounded f16 it cost half the accuracy where
// one value dominates a block). Relative error against 64 bits, k = 4096: 3.6e-8 on N(0,1) rows, 4.5e-8 .. 8e-8 on rows with
// heavy tails or outliers of 1e4; the f32 FMA kernel of nvfp4_gemv.cu: 9.9e-8 and 9.3e-8 .. 1.0e-7.
//
// Order of a sum, the same for every m and launch shape: k is cut into parts (parts_log2), a part into units of 128 values;
// unit u of a part belongs to sum u % 8; a part is its eight sums in order, plane by plane; a row is its parts in order.
//
// Shape of the kernel: persistent CTAs over 16-row tiles; warp 8 streams row pieces through a ring of bulk copies (it starts
// before the activations are ready), warps 0-7 are dealt units of 16 rows x 128 values round robin across tiles, so that no
// warp idles at a part's ragged end, warp 9 adds the eight sums of a part and stores. Clusters of two or four CTAs share a
// tile by parts where that fills the machine better; the others hand a part's sums to the first CTA through distributed
// shared memory.
// What bounds it: issue slots, at 0.63 of them in gate/up of one row (206 warp instructions a unit in all; 5120 x 17408 in clusters of two 0.47 and
// 250). The FMA kernel that it replaces for k >= 2048 spends 3.2 slots per weight AND row.
#include "common.cuh"
#include "nvfp4_col.cuh"
#include "nvfp4_gemv.cuh"

namespace {

constexpr int NW = 8;  // consumer warps = sums of a part
constexpr int NTHREADS = (NW + 2) * 32;
constexpr int NPL = 3;  // columns (f16 planes) of an activation row
constexpr int MAX_STAGES = 12;
constexpr int RD = 3;  // parts in flight between the consumers and the adding warp
constexpr int XD = 4;  // parts in flight between the CTAs of a cluster
constexpr int ROWS = 16;
constexpr int HDR = 512;  // barriers
constexpr int MAX_KS = 4;

// log2 of the parts of a row, at most 72 blocks (4608 values) each: a function of k alone.
inline int parts_log2(int bpr) {
    int lg = 0;
    while (lg < 6 && bpr > 72 << lg) lg++;
    return lg;
}
// first block of part i of 2^lg (whole groups of four blocks: 16-byte pieces)
__host__ __device__ inline int part_start(int i, int lg, int bpr) { return (int)(((long long)(bpr >> 2) * i) >> lg) * 4; }

struct ColParams {
    GemvParams g;
    int lg, ks, tx, pitch;  // log2 of the parts of a row; CTAs per cluster; blocks per row and stage; bytes of a row in a stage
    uint32_t xch_off, red_off, inv_off, x_off, ring_off;
};

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void arrive_peer(uint32_t bar_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_addr) : "memory");
}
// bounded wait that acquires what another CTA of the cluster released
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
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
// NP: MMA column groups, 8 NP >= 3 m. CPS: CTAs per SM the register allocation must allow.
template <int NP, int CPS>
__global__ void __launch_bounds__(NTHREADS, CPS) nvfp4_gemv_col_kernel(const ColParams cp) {
    extern __shared__ __align__(128) uint8_t smem[];
    const GemvParams& p = cp.g;
    const int KS = cp.ks, crank = (int)(blockIdx.x % KS), cid = (int)(blockIdx.x / KS), ncl = (int)(gridDim.x / KS);
    const int bpr = p.k >> 6, lg = cp.lg, mine = (1 << lg) / KS, part0 = crank * mine;
    const int b0 = part_start(part0, lg, bpr), nblk = part_start(part0 + mine, lg, bpr) - b0;  // this CTA's blocks of every row
    const size_t row_bytes = (size_t)bpr * 36;
    const float gs0 = __ldg(p.gs0), gs1 = __ldg(p.gs1);
    const float gp = gs_pow2(gs0);
    const float* xbase = (const float*)p.x + (size_t)b0 * 64;
    float* y = (float*)p.y;
    const bool gu = p.w1 != nullptr;
    const int m = p.m, ncol = NPL * m;
    const int per_cta = gu ? ROWS / 2 : ROWS;  // gate/up: 8 indices, row slots 0-7 gate, 8-15 up
    const int ntiles = (p.rows + per_cta - 1) / per_cta;
    const int S = p.stages, TX = cp.tx, pitch = cp.pitch, stage_bytes = ROWS * pitch;

    uint64_t* full = (uint64_t*)smem;
    uint64_t* empty = full + MAX_STAGES;
    uint64_t* tbar = empty + MAX_STAGES;         // [RD] a part's sums are posted
    uint64_t* tfree = tbar + RD;                 // [RD] ... and have been read
    uint64_t* xbar = tfree + RD;                 // [MAX_KS - 1][XD] first CTA: a part of another CTA has arrived
    uint64_t* xfree = xbar + (MAX_KS - 1) * XD;  // [XD] other CTAs: ... and has been read
    static_assert((2 * MAX_STAGES + 2 * RD + MAX_KS * XD) * 8 <= HDR, "barriers overlap");
    const uint32_t base = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int posts = min(NW, part_start(1, lg, bpr) >> 1);  // sums of a part that hold any unit

    if (warp == NW) {
        if (lane < S) {
            mbar_init(&full[lane], 1);
            mbar_init(&empty[lane], NW);
        }
        if (lane < RD) {
            mbar_init(&tbar[lane], posts);
            mbar_init(&tfree[lane], 1);
        }
        if (KS > 1 && lane < MAX_KS * XD) mbar_init(&xbar[lane], 1);  // xbar and xfree lie side by side
        mbar_fence_init();
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(NTHREADS) : "memory");
    }
    pdl_launch_dependents();
    if (KS > 1) cluster_sync_all();  // every CTA's barriers exist before anything is sent to them

    if (warp == NW) {
        // ------------------------------------------------------------ weights in
        const uint64_t pol = l2_policy_evict_first();
        int s = 0;
        uint32_t par = 1;  // parity of "empty": the first round passes at once
        bool ok = true;
        for (int tile = cid; tile < ntiles && ok; tile += ncl) {
            const int row0 = tile * per_cta;
            const int row = gu ? row0 + (lane & 7) : row0 + lane;
            const uint8_t* wb = (gu && ((lane >> 3) & 1)) ? p.w1 : p.w0;
            const uint8_t* src = (lane < ROWS && row < p.rows) ? wb + (size_t)row * row_bytes : nullptr;
            const uint32_t nvalid = (uint32_t)__popc(__ballot_sync(0xffffffffu, src != nullptr));
            for (int pt = part0; pt < part0 + mine && ok; pt++) {
                const int pb = part_start(pt, lg, bpr), pe = part_start(pt + 1, lg, bpr);
                for (int b = pb; b < pe; b += TX) {
                    const uint32_t piece = (uint32_t)min(TX, pe - b) * 36u;
                    if (!mbar_wait(&empty[s], par)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    if (lane == 0) {
                        mbar_expect_tx(&full[s], nvalid * piece);
                        mbar_arrive(&full[s]);
                    }
                    __syncwarp();
                    if (src) bulk_g2s_stream(smem + cp.ring_off + (size_t)s * stage_bytes + (size_t)lane * pitch, src + (size_t)b * 36, piece, &full[s], pol);
                    if (++s == S) s = 0, par ^= 1u;
                }
            }
        }
    } else if (warp < NW) {
        // ------------------------------------------------------------ activations: f16 planes over a power-of-two scale per
        // 64-value block; eight lanes per block, eight values each. Column c, block b, 16-byte chunk i at
        // ((c nblk + b) 8 + (i ^ 4 (c & 1))) 16: the two columns that a quarter-warp reads at once lie on distinct banks.
        // The power of two of the tensor scale goes into the block scales (exact), the rest is applied to the sums.
        pdl_wait();  // the activations may come from the previous kernel of the stream
        const int ntask = nblk * 8;
        constexpr int PF = 3;  // loads of a thread in flight, twice 16 bytes each
        for (int r = 0; r < m; r++) {
            const uint4* xr = (const uint4*)(xbase + (size_t)r * p.k);
            for (int t0 = tid; t0 < ntask; t0 += PF * NW * 32) {
                uint4 raw[PF][2];
#pragma unroll
                for (int i = 0; i < PF; i++) {
                    const int task = t0 + i * (NW * 32);
                    if (task < ntask) raw[i][0] = __ldcg(xr + (size_t)task * 2), raw[i][1] = __ldcg(xr + (size_t)task * 2 + 1);
                }
#pragma unroll
                for (int i = 0; i < PF; i++) {
                    const int task = t0 + i * (NW * 32);
                    if (task >= ntask) break;  // uniform over eight lanes
                    const int b = task >> 3, ch = task & 7;
                    uint32_t h[NPL][4];
                    const float inv = f32_planes(raw[i][0], raw[i][1], lane, h);
#pragma unroll
                    for (int pl = 0; pl < NPL; pl++) {
                        const int c = r * NPL + pl;
                        *(uint4*)(smem + cp.x_off + ((size_t)(c * nblk + b) * 8 + (ch ^ (4 * (c & 1)))) * 16) = make_uint4(h[pl][0], h[pl][1], h[pl][2], h[pl][3]);
                        if (ch == pl) *(float*)(smem + cp.inv_off + ((size_t)b * (8 * NP) + c) * 4) = inv * gp;
                    }
                }
            }
        }
        asm volatile("bar.sync 2, %0;" ::"n"(NTHREADS) : "memory");  // staged, and the barriers are initialised

        // ------------------------------------------------------------ units of 16 rows x 128 values
        // Inside an MMA the order of k is free as long as A and B agree: thread t of a quad takes word t (8 codes) of 32
        // consecutive values of a row and activations 8 t .. 8 t + 7 of column g: one 32-bit load per row, one 128-bit load
        // per column group, two MMAs.
        const int g = lane >> 2, t = lane & 3;
        const uint32_t ring = base + cp.ring_off + (uint32_t)(g * pitch + 4 * t);
        const uint32_t xflip = (g & 1) ? (uint32_t)-64 : 64u;  // from the first half of a block to the second
        uint32_t xa[NP];
#pragma unroll
        for (int ps = 0; ps < NP; ps++) {
            int c = ps * 8 + g;
            if (c >= ncol) c = g & 1;  // a column beyond the live ones repeats one of them and is not read
            xa[ps] = base + cp.x_off + (uint32_t)(c * nblk * 128 + (c & 1) * 64 + t * 16);
        }
        const uint32_t xi0 = base + cp.inv_off + 8u * (uint32_t)t;
        int s = 0, rs = 0, dealt = 0;
        uint32_t par = 0, rpar = 1;
        bool ok = true;
        for (int tile = cid; tile < ntiles && ok; tile += ncl) {
            for (int pt = part0; pt < part0 + mine && ok; pt++) {
                const int pb = part_start(pt, lg, bpr), pe = part_start(pt + 1, lg, bpr), nu = (pe - pb) >> 1;
                const int v = (warp - dealt) & (NW - 1);
                dealt += nu;
                float acc[NP][4];
#pragma unroll
                for (int ps = 0; ps < NP; ps++) acc[ps][0] = acc[ps][1] = acc[ps][2] = acc[ps][3] = 0.0f;
                int u = v;
                for (int b = pb; b < pe; b += TX) {
                    if (!mbar_wait(&full[s], par)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        ok = false;
                        break;
                    }
                    const int ub = (b - pb) >> 1, ue = min(ub + (TX >> 1), nu);
                    for (; u < ue; u += NW) {
                        const uint32_t pa = ring + (uint32_t)(s * stage_bytes + (u - ub) * 72);
                        const uint32_t lb = (uint32_t)(pb - b0 + 2 * u);  // block within this CTA's activations
#pragma unroll
                        for (int bl = 0; bl < 2; bl++) {
                            const uint32_t pw = pa + 36u * bl, pw8 = pw + 8u * (uint32_t)pitch;
                            const __half2 sa = lane_scales(lds32(pw - 4u * t), 8u * (t >> 1)), sb = lane_scales(lds32(pw8 - 4u * t), 8u * (t >> 1));
                            float cc[NP][4];
#pragma unroll
                            for (int ps = 0; ps < NP; ps++) cc[ps][0] = cc[ps][1] = cc[ps][2] = cc[ps][3] = 0.0f;
#pragma unroll
                            for (int hf = 0; hf < 2; hf++) {
                                uint32_t ha[4], hb[4];
                                e2m1x8_to_f16x2(lds32(pw + 4u + 16u * hf), ha);
                                e2m1x8_to_f16x2(lds32(pw8 + 4u + 16u * hf), hb);
                                const __half2 fha = hf ? __high2half2(sa) : __low2half2(sa), fhb = hf ? __high2half2(sb) : __low2half2(sb);
                                const uint32_t fa = *(const uint32_t*)&fha, fb = *(const uint32_t*)&fhb;
#pragma unroll
                                for (int i = 0; i < 4; i++) ha[i] = hmul2u(ha[i], fa), hb[i] = hmul2u(hb[i], fb);
#pragma unroll
                                for (int ps = 0; ps < NP; ps++) {
                                    const uint4 xv = lds128(xa[ps] + (lb + bl) * 128u + (hf ? xflip : 0u));
                                    mma16816(cc[ps], ha[0], hb[0], ha[1], hb[1], xv.x, xv.y);
                                    mma16816(cc[ps], ha[2], hb[2], ha[3], hb[3], xv.z, xv.w);
                                }
                            }
#pragma unroll
                            for (int ps = 0; ps < NP; ps++) {
                                const float2 xi = lds64f(xi0 + ((lb + bl) * NP + ps) * 32u);
                                acc[ps][0] = fmaf(cc[ps][0], xi.x, acc[ps][0]);
                                acc[ps][1] = fmaf(cc[ps][1], xi.y, acc[ps][1]);
                                acc[ps][2] = fmaf(cc[ps][2], xi.x, acc[ps][2]);
                                acc[ps][3] = fmaf(cc[ps][3], xi.y, acc[ps][3]);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[s]);
                    if (++s == S) s = 0, par ^= 1u;
                }
                if (!ok) break;
                if (!mbar_wait(&tfree[rs], rpar)) {  // also by a warp with nothing to post: nobody gets two rounds ahead of a slot
                    cn_dev_fail(CN_DEV_WAIT_EMPTY);
                    ok = false;
                    break;
                }
                if (v < posts) {
                    // sums [v][column][16 rows]
                    float* rb = (float*)(smem + cp.red_off) + (size_t)(rs * NW + v) * ncol * 16;
#pragma unroll
                    for (int ps = 0; ps < NP; ps++) {
                        const int c = ps * 8 + 2 * t;
                        if (c < ncol) rb[c * 16 + g] = acc[ps][0], rb[c * 16 + g + 8] = acc[ps][2];
                        if (c + 1 < ncol) rb[c * 16 + 16 + g] = acc[ps][1], rb[c * 16 + 16 + g + 8] = acc[ps][3];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tbar[rs]);
                }
                if (++rs == RD) rs = 0, rpar ^= 1u;
            }
        }
    } else {
        // ------------------------------------------------------------ a part's sums, the parts of a row, results out
        asm volatile("bar.sync 2, %0;" ::"n"(NTHREADS) : "memory");
        pdl_wait();  // a kernel two places ahead in the stream may still read what this one overwrites
        constexpr int NO = NP == 1 ? 1 : (NP == 2 ? 3 : 4);  // outputs per lane: 16 m / 32 rounded up
        const float f0 = gs0 / gp, f1 = gs1 / gp;            // exact: gp is a power of two
        int rs = 0, seq = 0;
        uint32_t rpar = 0;
        bool ok = true;
        // outputs lane + 32 i of the part in slot rs: row slot o & 15 of activation row o >> 4
        auto collect = [&](float out[NO]) -> bool {
            if (!mbar_wait(&tbar[rs], rpar)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                return false;
            }
            const float* rb = (const float*)(smem + cp.red_off) + (size_t)rs * NW * ncol * 16;
#pragma unroll
            for (int i = 0; i < NO; i++) {
                const int o = lane + 32 * i;
                out[i] = 0.0f;
                if (o < 16 * m) {
                    const float* q = rb + (o >> 4) * (NPL * 16) + (o & 15);
                    float s0 = q[0], s1 = q[16], s2 = q[32];
                    for (int v = 1; v < posts; v++) s0 += q[v * ncol * 16], s1 += q[v * ncol * 16 + 16], s2 += q[v * ncol * 16 + 32];
                    out[i] = fmaf(s2, 0x1p-22f, fmaf(s1, 0x1p-11f, s0));
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&tfree[rs]);
            if (++rs == RD) rs = 0, rpar ^= 1u;
            return true;
        };
        for (int tile = cid; tile < ntiles && ok; tile += ncl) {
            float tot[NO], cur[NO];
            for (int i = 0; i < mine && ok; i++) {
                if (!collect(cur)) {
                    ok = false;
                    break;
                }
                if (crank == 0) {
#pragma unroll
                    for (int j = 0; j < NO; j++) tot[j] = i == 0 ? cur[j] : tot[j] + cur[j];
                } else {
                    const int xs = seq % XD;
                    if (seq >= XD && !mbar_wait_cluster(&xfree[xs], ((seq / XD) - 1) & 1)) {
                        cn_dev_fail(CN_DEV_WAIT_EMPTY);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = base + cp.xch_off + (uint32_t)(((crank - 1) * XD + xs) * m * 64);
#pragma unroll
                    for (int j = 0; j < NO; j++)
                        if (lane + 32 * j < 16 * m) st_peer_f32(peer_addr(dst + 4u * (uint32_t)(lane + 32 * j), 0), cur[j]);
                    __syncwarp();
                    if (lane == 0) arrive_peer(peer_addr(smem_u32(&xbar[(crank - 1) * XD + xs]), 0));
                    seq++;
                }
            }
            if (crank != 0 || !ok) continue;
            for (int src = 1; src < KS && ok; src++) {
                for (int i = 0; i < mine; i++) {
                    const int n = seq + i, xs = n % XD;
                    if (!mbar_wait_cluster(&xbar[(src - 1) * XD + xs], (n / XD) & 1)) {
                        cn_dev_fail(CN_DEV_WAIT_FULL);
                        ok = false;
                        break;
                    }
                    const float* q = (const float*)(smem + cp.xch_off) + ((src - 1) * XD + xs) * m * 16;
#pragma unroll
                    for (int j = 0; j < NO; j++)
                        if (lane + 32 * j < 16 * m) tot[j] += q[lane + 32 * j];
                    __syncwarp();
                    if (lane == 0) arrive_peer(peer_addr(smem_u32(&xfree[xs]), (uint32_t)src));
                }
            }
            seq += mine;
            if (!ok) break;
#pragma unroll
            for (int j = 0; j < NO; j++) {
                const int o = lane + 32 * j, slot = o & 15, r = o >> 4;
                const float a = tot[j] * ((gu && slot >= 8) ? f1 : f0);
                const float up = __shfl_down_sync(0xffffffffu, a, 8);
                const int row = tile * per_cta + slot;
                if (slot < per_cta && row < p.rows && r < m) y[(size_t)r * p.ldy + row] = gu ? act_gu(a, up, p.limit) : a;
            }
        }
    }
    if (KS > 1) cluster_sync_all();  // nobody leaves while a CTA of the cluster may still send or receive
}

template <int NP, int CPS>
int launch_col(const cudaLaunchConfig_t& cfg, const ColParams& p) {
    CN_ALLOW_SMEM((nvfp4_gemv_col_kernel<NP, CPS>), 226 * 1024);
    CN_CUDA(cudaLaunchKernelEx(&cfg, nvfp4_gemv_col_kernel<NP, CPS>, p));
    return CN_OK;
}

}  // namespace

int cn_gemv_col_launch(const GemvCall& a, cudaStream_t stream, const char* who) {
    const int rows = a.rows, k = a.k, m = a.m, bpr = k / 64;
    const bool gu = a.w1 != nullptr;
    const int ncol = NPL * m, np = (ncol + 7) / 8;
    const int per_cta = gu ? ROWS / 2 : ROWS;
    const int ntiles = (rows + per_cta - 1) / per_cta;
    ColParams p = {};
    p.lg = parts_log2(bpr);
    const int parts = 1 << p.lg;
    int pmax = 0;
    for (int i = 0; i < parts; i++) {
        const int n = part_start(i + 1, p.lg, bpr) - part_start(i, p.lg, bpr);
        pmax = n > pmax ? n : pmax;
    }
    // a part in as few equal chunks as have `most` blocks or fewer
    long long stage_bytes = 0;
    auto chunks_of = [&](int most) {
        const int nch = (pmax + most - 1) / most;
        p.tx = ((pmax + nch - 1) / nch + 3) & ~3;
        p.pitch = p.tx * 36 + ((p.tx / 4) % 2 == 0 ? 16 : 0);  // an odd number of 16-byte units: the eight rows of a load on distinct banks
        stage_bytes = (long long)ROWS * p.pitch;
    };
    chunks_of(32);
    auto layout = [&](int ks, ColParams& q) {  // returns the shared memory in front of the ring for clusters of ks
        int bmax = 0;
        for (int r = 0; r < ks; r++) {
            const int n = part_start((r + 1) * (parts / ks), p.lg, bpr) - part_start(r * (parts / ks), p.lg, bpr);
            bmax = n > bmax ? n : bmax;
        }
        q.xch_off = HDR;
        q.red_off = q.xch_off + (ks > 1 ? (uint32_t)((ks - 1) * XD * m * 64) : 0u);
        q.inv_off = q.red_off + (uint32_t)(RD * NW * ncol * 64);
        q.x_off = (q.inv_off + (uint32_t)(bmax * np * 32) + 127u) & ~127u;
        const long long end = (long long)q.x_off + (long long)ncol * bmax * 128;
        q.ring_off = (uint32_t)((end + 127) & ~127LL);
        return (end + 127) & ~127LL;
    };
    // CTAs per cluster and per SM, by the tiles of the busiest SM in whole matrix rows (half way between the mean and its next
    // whole number: short queues are evened out by whoever starts late), dearer with one CTA's warps alone or with sums handed
    // on. Measured, CTAs per cluster / per SM: 5120 x 17408, one row: 2/2 22.6 us, 1/1 32.1, 4/2 36.5; 5120 x 5120, four rows:
    // 1/1 14.4 us, 2/1 16.1, 1/2 (two calls) 22.8; gate/up 17408 x 5120, one row: 1/2 37.1 us, 1/3 37.4, 2/2 39.4, 1/1 52.9.
    int ks = 0, cps = 0;
    double best = 1e30;
    for (int c = np == 1 ? 3 : 2; c >= 1; c--) {
        for (int n = 1; n <= MAX_KS && n <= parts; n *= 2) {
            ColParams q = p;
            if ((227 * 1024) / c - 1024 - layout(n, q) < 3 * stage_bytes) continue;
            const double mean = (double)ntiles * n / 148, t0 = 0.5 * (mean + (double)(long long)(mean + 0.999999)) / n;
            const double t = t0 * (c == 1 ? 1.3 : (c == 3 ? 1.05 : 1.0)) * (n == 1 ? 1.0 : (n == 2 ? 1.25 : 1.7));
            if (t < best) best = t, ks = n, cps = c;
        }
    }
    if (!ks) {
        if (m == 1) CN_FAIL(CN_ERR_LIMIT, "%s: k = %d leaves no room for a weight ring beside the activations", who, k);
        // the staged activations of all m rows do not fit beside a ring: two calls over half the rows each
        const int m0 = m / 2;
        GemvCall lo = a, hi = a;
        lo.m = m0, hi.m = m - m0;
        hi.x = (const float*)a.x + (size_t)m0 * k;
        hi.y = (float*)a.y + (size_t)m0 * a.ldy;
        const int rc = cn_gemv_col_launch(lo, stream, who);
        return rc ? rc : cn_gemv_col_launch(hi, stream, who);
    }
    // Longer chunks, up to a whole part, where three stages of them fit as well: a chunk's wait and release cost every warp some forty
    // instructions for the one to three units that it has there. FFN 5120 - 17408, one row: 59.1 us with chunks of 20 and 24 blocks, 51.4 of 40
    // and 36; 162853 x 3584, eight rows: 306 and 251.
    const int tx32 = p.tx;
    chunks_of(72);
    while (p.tx > tx32 && (227 * 1024) / cps - 1024 - layout(ks, p) < 3 * stage_bytes) chunks_of(p.tx - 4);
    p.ks = ks;
    const long long front = layout(ks, p);
    const int clusters = 148 * cps / ks, grid = ks * (ntiles < clusters ? ntiles : clusters);
    const long long chunks = (long long)((ntiles + grid / ks - 1) / (grid / ks)) * (parts / ks) * ((pmax + p.tx - 1) / p.tx);
    long long stages = ((227 * 1024) / cps - 1024 - front) / stage_bytes;
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    if (stages > chunks) stages = chunks;
    GemvParams& g = p.g;
    g.w0 = (const uint8_t*)a.w0, g.w1 = (const uint8_t*)a.w1, g.gs0 = a.gs0, g.gs1 = a.gs1 ? a.gs1 : a.gs0, g.x = a.x, g.y = a.y;
    g.rows = rows, g.k = k, g.m = m, g.ldy = a.ldy, g.limit = a.limit, g.stages = (int)stages;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = (size_t)(front + stages * stage_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at, cfg.numAttrs = 1;
    if (ks > 1) {
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = (unsigned)ks, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
#define CN_COL_CASE(NPV, CPSV) \
    if (np == NPV && cps == CPSV) return launch_col<NPV, CPSV>(cfg, p);
    CN_COL_CASE(1, 3) CN_COL_CASE(1, 2) CN_COL_CASE(1, 1) CN_COL_CASE(2, 2) CN_COL_CASE(2, 1) CN_COL_CASE(3, 2) CN_COL_CASE(3, 1)
#undef CN_COL_CASE
    CN_FAIL(CN_ERR_SHAPE, "%s: no kernel for %d columns, %d CTAs per SM", who, ncol, cps);
}
