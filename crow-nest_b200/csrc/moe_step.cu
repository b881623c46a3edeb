// The second half of a small routed-expert step in one launch: down projections of a token's experts and of the shared expert, and the
// weighted combine. Supersedes gemv_fp4_ptrb over the down table, acc_combo and gate_shared (engine/src/kernels.rs:195-233, :1583-1599)
// for steps of few combos; many share experts and run in groups instead (nvfp4_rows_tc.cu).
//
// A CTA owns 16 rows of one token's result. Its work is cut into units - an expert's down matrix, eight 64-value blocks of k - and every
// warp keeps its units to itself: it brings 16 row pieces in by its own bulk copies, cuts 512 values of h into f16 planes (three columns of
// an MMA: nvfp4_col.cuh) and leaves 16 sums in shared memory. The CTA meets once; then a lane per row adds the units of an expert, the
// experts in pick order, and the shared expert, as moe_combine_kernel does: no expert output goes through memory.
//
// Measured, one token of 512 experts of 2048 x 512, top 10, with a shared expert, captured: 28.8 -> 20.5 us against four launches and a fork to a
// side stream and back.
//
// What bounds it: latency. The ids are older than the kernel before this one (which waits for whatever wrote them before it lets this one
// start), so the first weights are on their way while gate / up still runs; after it there is one trip to L2 for h, the
// unit itself (some 1450 warp instructions with its loads and planes), and a barrier.
#include "moe_step.cuh"
#include "nvfp4_col.cuh"

namespace {

constexpr int CB = 8;  // blocks of a unit
constexpr int PITCH = CB * 36 + 16;
constexpr int CHUNK = 16 * PITCH;
constexpr int NWMAX = 12;
constexpr int X_BYTES = 3 * CB * 128;  // three planes of a unit's activations
constexpr int INV_BYTES = CB * 32;     // [block][column] scales
constexpr int MAX_UNITS = 256;
constexpr int MAX_PICKS = 64;
constexpr int WT_OFF = 128, SUM_OFF = WT_OFF + MAX_PICKS * 8;  // behind the barriers: weight and "has a matrix" of every pick, [units][16] sums, the warps' own memory
constexpr int WARP_BYTES = CHUNK + X_BYTES + INV_BYTES;
static_assert(NWMAX * 8 <= WT_OFF && WARP_BYTES % 128 == 0, "layout");
__host__ __device__ constexpr int warp_off(int units) { return (SUM_OFF + units * 64 + 127) & ~127; }

__global__ void __launch_bounds__(NWMAX * 32, 2) moe_down_combine_kernel(const MoeDownCall c) {
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int tile = blockIdx.x, tok = blockIdx.y;
    const int cr = (c.inter / 64 + CB - 1) / CB, cs = c.shared ? (c.shared_inter / 64 + CB - 1) / CB : 0;
    const int nr = c.topk * cr, units = nr + cs;
    uint64_t* full = (uint64_t*)smem + warp;
    float* sums = (float*)(smem + SUM_OFF);
    uint8_t* mine = smem + warp_off(units) + (size_t)warp * WARP_BYTES;
    if (lane == 0) {
        mbar_init(full, 1);
        mbar_fence_init();
    }
    __syncwarp();
    // an expert's down matrix, null where it is not resident
    auto matrix = [&](int j) -> const uint8_t* {
        const int e = __ldcg(c.ids + (size_t)tok * c.topk + j);
        if (e < 0 || (c.experts > 0 && e >= c.experts)) return nullptr;
        return (const uint8_t*)__ldcg(c.table + e);
    };
    const uint64_t pol = l2_policy_evict_first();
    // unit u's weights on their way; false where there are none
    auto issue = [&](int u) -> bool {
        const bool sh = u >= nr;
        const uint8_t* w = sh ? (const uint8_t*)c.shared : matrix(u / cr);
        if (!w) return false;
        const int bpr = (sh ? c.shared_inter : c.inter) >> 6, ch = sh ? u - nr : u % cr;
        const uint32_t piece = (uint32_t)min(CB, bpr - ch * CB) * 36u;
        const int row = tile * 16 + lane;
        const bool have = lane < 16 && row < c.hidden;
        const uint32_t n = (uint32_t)__popc(__ballot_sync(0xffffffffu, have));
        if (lane == 0) {
            mbar_expect_tx(full, n * piece);
            mbar_arrive(full);
        }
        __syncwarp();
        if (have) bulk_g2s_stream(mine + (size_t)lane * PITCH, w + (size_t)row * bpr * 36 + (size_t)ch * (CB * 36), piece, full, pol);
        return true;
    };
    bool live = warp < units && issue(warp);
    // a pick's weight (0: no matrix) for the sums at the end: two dependent trips to L2 each, one after another, if they were made there
    float2* wt = (float2*)(smem + WT_OFF);
    for (int j = (int)blockDim.x - 1 - (int)threadIdx.x; j < c.topk; j += blockDim.x)
        wt[j] = make_float2(__ldcg(c.wts + (size_t)tok * c.topk + j), matrix(j) ? 1.0f : 0.0f);

    pdl_wait();  // h comes from the kernel before this one
    uint8_t *xs = mine + CHUNK, *inv = xs + X_BYTES;
    const int g = lane >> 2, t = lane & 3, col = g < 3 ? g : g & 1;  // a column beyond the three planes repeats one and is not read
    const uint8_t* xa = xs + col * (CB * 128) + (col & 1) * 64 + t * 16;
    const int xflip = (col & 1) ? -64 : 64;
    bool ok = true;
    uint32_t par = 0;
    for (int u = warp; u < units && ok; u += nw) {
        if (u != warp) live = issue(u);
        const bool sh = u >= nr;
        float v[2] = {0.0f, 0.0f};
        if (live) {
            const int k = sh ? c.shared_inter : c.inter, ch = sh ? u - nr : u % cr, nb = min(CB, (k >> 6) - ch * CB);
            const float gs = __ldg(sh ? c.shared_gs : c.gs), gp = gs_pow2(gs);
            const uint4* x = (const uint4*)((sh ? c.hs + (size_t)tok * k : c.h + ((size_t)tok * c.topk + u / cr) * k) + ch * (CB * 64));
            uint4 lo[2], hi[2];
#pragma unroll
            for (int i = 0; i < 2; i++)
                if (i * 4 < nb) lo[i] = __ldcg(x + 2 * (32 * i + lane)), hi[i] = __ldcg(x + 2 * (32 * i + lane) + 1);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (i * 4 >= nb) break;  // nb is 4 or 8
                const int b = 4 * i + (lane >> 3), chn = lane & 7;
                uint32_t h[3][4];
                const float iv = f32_planes(lo[i], hi[i], lane, h);
#pragma unroll
                for (int pl = 0; pl < 3; pl++) {
                    *(uint4*)(xs + (size_t)((pl * CB + b) * 8 + (chn ^ (4 * (pl & 1)))) * 16) = make_uint4(h[pl][0], h[pl][1], h[pl][2], h[pl][3]);
                    if (chn == pl) *(float*)(inv + (b * 8 + pl) * 4) = iv * gp;
                }
            }
            __syncwarp();
            if (!mbar_wait(full, par)) {
                cn_dev_fail(CN_DEV_WAIT_FULL);
                ok = false;
            } else {
                par ^= 1u;
                const uint8_t* cbase = mine + g * PITCH + 4 * t;
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
                for (int b = 0; b < nb; b++) {
                    float cc[1][4];
                    block_mma<1>(cc, cbase + 36 * b, cbase + 36 * b + 8 * PITCH, t, [&](int, int hf) { return *(const uint4*)(xa + b * 128 + (hf ? xflip : 0)); });
                    const float2 xi = *(const float2*)(inv + b * 32 + 8 * t);
                    acc[0] = fmaf(cc[0][0], xi.x, acc[0]), acc[1] = fmaf(cc[0][1], xi.y, acc[1]);
                    acc[2] = fmaf(cc[0][2], xi.x, acc[2]), acc[3] = fmaf(cc[0][3], xi.y, acc[3]);
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float na = __shfl_down_sync(0xffffffffu, acc[2 * i], 1);
                    v[i] = fmaf(na, 0x1p-22f, fmaf(acc[2 * i + 1], 0x1p-11f, acc[2 * i])) * (gs / gp);  // gp is a power of two
                }
            }
        }
        if (t == 0) sums[u * 16 + g] = v[0], sums[u * 16 + g + 8] = v[1];
        __syncwarp();  // the unit's weights and planes have been read
    }
    if (__syncthreads_or(!ok)) return;
    const int row = tile * 16 + (int)threadIdx.x;
    if (threadIdx.x >= 16 || row >= c.hidden) return;
    float acc = 0.0f;
    for (int j = 0; j < c.topk; j++) {
        const float2 w = wt[j];
        if (w.y == 0.0f) continue;
        float e = sums[j * cr * 16 + threadIdx.x];
        for (int i = 1; i < cr; i++) e += sums[(j * cr + i) * 16 + threadIdx.x];
        acc = __fadd_rn(acc, __fmul_rn(w.x, e));
    }
    float base = 0.0f;
    if (c.shared) {
        base = sums[nr * 16 + threadIdx.x];
        for (int i = 1; i < cs; i++) base += sums[(nr + i) * 16 + threadIdx.x];
        if (c.sgate) base = __fmul_rn(1.0f / (1.0f + expf(-__ldg(c.sgate + tok))), base);
    }
    const float r = __fadd_rn(base, acc);
    if (c.out_bf16)
        ((__nv_bfloat16*)c.y)[(size_t)tok * c.hidden + row] = __float2bfloat16_rn(r);
    else
        ((float*)c.y)[(size_t)tok * c.hidden + row] = r;
}

int units_of(const MoeDownCall& c) { return c.topk * ((c.inter / 64 + CB - 1) / CB) + (c.shared ? (c.shared_inter / 64 + CB - 1) / CB : 0); }

}  // namespace

bool cn_moe_down_combine_fits(const MoeDownCall& c) {
    return c.inter % 256 == 0 && (!c.shared || (c.shared_inter > 0 && c.shared_inter % 256 == 0)) && units_of(c) <= MAX_UNITS && c.topk <= MAX_PICKS && c.tokens <= 65535 &&
           !(((uintptr_t)c.shared | (uintptr_t)c.h | (uintptr_t)c.hs) & 15);
}

long long cn_moe_down_combine_units(const MoeDownCall& c) { return (long long)((c.hidden + 15) / 16) * c.tokens * units_of(c); }

int cn_moe_down_combine_launch(const MoeDownCall& c, cudaStream_t stream) {
    if (!cn_moe_down_combine_fits(c)) CN_FAIL(CN_ERR_SHAPE, "moe down projections: inter %d, shared inter %d, %d picks", c.inter, c.shared_inter, c.topk);
    const int units = units_of(c);
    const int rounds = (units + NWMAX - 1) / NWMAX, nw = (units + rounds - 1) / rounds;  // as few rounds of units as twelve warps allow, level
    const size_t smem = (size_t)warp_off(units) + (size_t)nw * WARP_BYTES;
    CN_ALLOW_SMEM(moe_down_combine_kernel, 226 * 1024);
    CN_CUDA(cn_launch_pdl(moe_down_combine_kernel, dim3((unsigned)((c.hidden + 15) / 16), (unsigned)c.tokens), dim3((unsigned)nw * 32), smem, stream, c));
    return CN_OK;
}
