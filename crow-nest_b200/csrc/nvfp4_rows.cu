// Routed-expert NVFP4 rows: groups of activation rows of one expert as the columns of the tensor-core tile, one warp per tile.
//
// Supersedes gemv_fp4_ptrb over the pointer tables (engine/src/kernels.rs:195-233) together with the grouping idea of the
// reference's prefill path (moe_count / moe_plan / moe_scatter, engine/src/kernels.rs:3334-3420). Arithmetic: weights
// with their scale in f16 (exact), f32 rows as three f16 planes, f32 sums.
//
// An expert's matrices are small (2048 x 512: a row is 288 bytes), so what a GEMV kernel spends per tile - handing sums between
// warps, staging and scale tables per CTA - outweighs the tile. Here a warp keeps a 16-row tile to itself: it brings the tile in
// by its own asynchronous copies (16 row pieces of up to eight blocks, two to four chunks ahead; as a bulk copy for every piece they were what the
// kernel waited for: 64 tokens 244 us a step, 224 with 16-byte copies), holds all its sums in registers and stores them; warps meet only once, when the group's rows have been staged. Up to eight bf16 rows or two f32 rows of an expert (six
// columns) share one decode of its weights; a row's sum does not depend on the rows it is grouped with. Bound by issue slots:
// some 175 warp instructions per 16 x 128 values in all (200 with one scale made at a time: 258 us a step against 245). Measured at 64 tokens, 512 experts of 2048 x 512, top 10 (under
// the profiler): gate/up 157 -> 114 us, down 203 -> 77 us against one CTA set per combo.
#include "nvfp4_col.cuh"
#include "nvfp4_gemv.cuh"

namespace {

constexpr int NW = 8;
constexpr int CB = 8;  // blocks per row and chunk
constexpr int PITCH = PIECE_PITCH, CHUNK = PIECE_TILE;
constexpr int MAX_D = 4;
static_assert(PITCH == CB * 36 + 16, "pieces of a chunk");

struct RowsParams {
    RowsCall c;
    int parts, depth;
    uint32_t inv_off, x_off, ring_off;
};

// NPL: columns per activation row (1: bf16, 3: f32)
template <int NPL, int CPS>
__global__ void __launch_bounds__(NW * 32, CPS) nvfp4_rows_kernel(const RowsParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int XE = NPL == 1 ? 2 : 4;
    const RowsCall& c = p.c;
    pdl_launch_dependents();
    pdl_wait();  // the groups, ids and activations come from the kernels before this one
    constexpr int RG = NPL == 1 ? 8 : 2;  // most rows of a group
    const int bpr = c.k >> 6;
    const size_t row_bytes = (size_t)bpr * 36;
    const bool gu = c.tab1 || c.w1 || c.fused_up_rows > 0;
    const float gs0 = __ldg(c.gs0), gs1 = __ldg(c.gs1), gp = gs_pow2(gs0);
    const float f0 = gs0 / gp, f1 = gs1 / gp;  // exact: gp is a power of two
    const int per_tile = gu ? 8 : 16, T = (c.rows + per_tile - 1) / per_tile;  // gate/up: row slots 0-7 gate, 8-15 up
    const int t0 = (int)((long long)blockIdx.x * T / p.parts), t1 = (int)((long long)(blockIdx.x + 1) * T / p.parts);
    const int nch = (bpr + CB - 1) / CB, D = p.depth;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* ring = smem + p.ring_off + (size_t)warp * D * CHUNK;
    const int mytiles = t0 + warp < t1 ? (t1 - t0 - warp + NW - 1) / NW : 0, total = mytiles * nch;
    const PieceCopy copy(lane);
    const uint64_t pol = l2_policy_evict_first();
    const int n1 = c.count1 ? *c.count1 : 0, ngroups = c.w0 ? (c.m + RG - 1) / RG : (c.order ? n1 + *c.count2 : c.m);
    int s = 0, pstage = 0;  // stage read next, stage filled next: they meet again at the end of every group
    for (int grp = blockIdx.y; grp < ngroups; grp += gridDim.y) {
        // the group's rows and matrices: one-row groups, larger groups, or (dense form) RG rows after one another
        int pos = grp * RG, nrows = min(RG, c.m - pos);
        const uint8_t *w0 = (const uint8_t*)c.w0, *w1 = (const uint8_t*)c.w1;
        if (!c.w0) {
            if (c.order)
                pos = grp < n1 ? c.pos1[grp] : c.pos2[grp - n1], nrows = grp < n1 ? 1 : c.rows2[grp - n1];
            else
                pos = grp, nrows = 1;  // the combos as they come
            const int e = c.ids[c.order ? c.order[pos] : pos];
            if (e < 0 || (c.experts > 0 && e >= c.experts)) continue;
            w0 = (const uint8_t*)c.tab0[e];
            w1 = c.tab1 ? (const uint8_t*)c.tab1[e] : (c.fused_up_rows > 0 ? w0 + (size_t)c.fused_up_rows * row_bytes : nullptr);
            if (!w0 || (gu && !w1)) continue;  // this matrix of the expert is not resident
        }
        auto member = [&](int r) { return c.order ? c.order[pos + r] : pos + r; };
        // chunk i of this warp in turn -> the next stage; a group of copies is closed even when there is no chunk left, so that D - 1 younger
        // ones stand behind every chunk that is waited for
        int ptile = t0 + warp, pch = 0, given = 0;
        const uint32_t ring_at = smem_u32(ring);
        auto issue = [&]() {
            if (given++ < total) {
                const uint32_t parts = (uint32_t)min(CB, bpr - pch * CB) * 9u / 4u;
                const uint8_t* lo = w0 + (size_t)ptile * per_tile * row_bytes + (size_t)pch * (CB * 36);
                const uint8_t* hi = gu ? w1 + (lo - w0) : lo + 8 * row_bytes;
                const int left = c.rows - ptile * per_tile;
                copy(ring_at + (uint32_t)(pstage * CHUNK), lo, hi, (uint32_t)row_bytes, (uint32_t)min(left, 8), (uint32_t)(gu ? min(left, 8) : max(left - 8, 0)), parts, pol);
                if (++pch == nch) pch = 0, ptile += NW;
                if (++pstage == D) pstage = 0;
            }
            piece_commit();
        };
        for (int i = 0; i < D; i++) issue();

        // the group's rows: eight lanes per 64-value block; column, block and chunk order as nvfp4_col.cuh reads them
        const int ncol = NPL * nrows;
        for (int r = 0; r < nrows; r++) {
            const int combo = member(r);
            const uint4* xr = (const uint4*)((const char*)c.x + (size_t)(combo / c.x_div) * c.k * XE);
            for (int task = threadIdx.x; task < bpr * 8; task += NW * 32) {  // uniform over eight lanes
                const int b = task >> 3, ch = task & 7;
                uint32_t h[NPL][4];
                float inv;
                if constexpr (NPL == 1)
                    inv = bf16_plane(__ldcg(xr + task), lane, h);
                else
                    inv = f32_planes(__ldcg(xr + 2 * task), __ldcg(xr + 2 * task + 1), lane, h);
#pragma unroll
                for (int pl = 0; pl < NPL; pl++) {
                    const int col = r * NPL + pl;
                    *(uint4*)(smem + p.x_off + ((size_t)(col * bpr + b) * 8 + (ch ^ (4 * (col & 1)))) * 16) = make_uint4(h[pl][0], h[pl][1], h[pl][2], h[pl][3]);
                    if (ch == pl) *(float*)(smem + p.inv_off + ((size_t)b * 8 + col) * 4) = inv * gp;
                }
            }
        }
        __syncthreads();

        const int g = lane >> 2, t = lane & 3;
        const int col = g < ncol ? g : (ncol > 1 ? g & 1 : 0);  // a column beyond the live ones repeats one of them and is not read
        const uint8_t* xa = smem + p.x_off + (size_t)col * bpr * 128 + (col & 1) * 64 + t * 16;
        const int xflip = (col & 1) ? -64 : 64;
        const uint8_t* xi0 = smem + p.inv_off + 8 * t;
        const uint8_t* rbase = ring + g * PITCH + 4 * t;
        for (int tile = t0 + warp; tile < t1; tile += NW) {
            // bf16 rows: a running sum for each block of a chunk, eight in all. With a single one the rounding of k / 64 additions in a row
            // made the results of gate / up less exact than one row's of nvfp4_gemv_m1.cu (relative error against 64 bits, k = 2048 / 4096:
            // 1.5e-7 / 2.1e-7, there 1.3e-7 / 1.4e-7). f32 rows need one: their first plane lies on a grid and its sums hardly round.
            constexpr int NA = NPL == 1 ? CB : 1;
            float acc[NA][4];
#pragma unroll
            for (int i = 0; i < NA; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
            for (int ch = 0; ch < nch; ch++) {
                piece_wait(D - 1);
                __syncwarp();  // the other lanes' copies, too
                const int nb = min(CB, bpr - ch * CB);
                const uint8_t *cbase = rbase + s * CHUNK, *xc = xa + ch * (CB * 128), *xic = xi0 + ch * (CB * 32);
                auto block = [&](int b) {
                    float cc[1][4];
                    block_mma<1>(cc, cbase + 36 * b, cbase + 36 * b + 8 * PITCH, t, [&](int, int hf) { return *(const uint4*)(xc + b * 128 + (hf ? xflip : 0)); });
                    const float2 xi = *(const float2*)(xic + b * 32);
                    float* a = acc[NA > 1 ? b : 0];
                    a[0] = fmaf(cc[0][0], xi.x, a[0]);
                    a[1] = fmaf(cc[0][1], xi.y, a[1]);
                    a[2] = fmaf(cc[0][2], xi.x, a[2]);
                    a[3] = fmaf(cc[0][3], xi.y, a[3]);
                };
                if (nb == CB) {
#pragma unroll
                    for (int b = 0; b < CB; b++) block(b);
                } else if constexpr (NA > 1) {
                    block(0), block(1), block(2), block(3);  // nb is 4: k is a multiple of 256
                } else {
                    for (int b = 0; b < nb; b++) block(b);
                }
                __syncwarp();  // every lane has read the stage
                issue();
                if (++s == D) s = 0;
            }
#pragma unroll
            for (int n = NA / 2; n > 0; n /= 2)
#pragma unroll
                for (int i = 0; i < n; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] += acc[i + n][j];
            // lane (g, t): row slots g and g + 8, columns 2 t and 2 t + 1
            float v[2][2];  // [row slot][activation row of this lane]
            int r0;
            if constexpr (NPL == 1) {
                v[0][0] = acc[0][0], v[0][1] = acc[0][1], v[1][0] = acc[0][2], v[1][1] = acc[0][3];
                r0 = 2 * t;
            } else {
                // columns 0-2 are the planes of row 0, 3-5 those of row 1: lane t = 0 ends up with row 0, lane t = 1 with row 1
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float na = __shfl_down_sync(0xffffffffu, acc[0][2 * i], 1), nb = __shfl_down_sync(0xffffffffu, acc[0][2 * i + 1], 1);
                    v[i][0] = t == 0 ? fmaf(na, 0x1p-22f, fmaf(acc[0][2 * i + 1], 0x1p-11f, acc[0][2 * i])) : fmaf(nb, 0x1p-22f, fmaf(na, 0x1p-11f, acc[0][2 * i + 1]));
                }
                r0 = t;
            }
#pragma unroll
            for (int j = 0; j < (NPL == 1 ? 2 : 1); j++) {
                if (r0 + j >= nrows) continue;
                const int combo = member(r0 + j);
                float* y = c.yptrs ? (float*)c.yptrs[combo] : c.y + (size_t)combo * c.ldy;
                if (gu) {
                    const int idx = tile * 8 + g;
                    if (idx < c.rows) y[idx] = act_gu(v[0][j] * f0, v[1][j] * f1, c.limit);
                } else {
                    const int row = tile * 16 + g;
                    if (row < c.rows) y[row] = v[0][j] * f0;
                    if (row + 8 < c.rows) y[row + 8] = v[1][j] * f0;
                }
            }
        }
        __syncthreads();  // every warp has read this group's rows
    }
}

bool layout(const RowsCall& a, int cps, RowsParams& p, size_t& smem) {
    const int bpr = a.k / 64, cols = 8;
    p.inv_off = 0;
    p.x_off = (p.inv_off + (uint32_t)(bpr * 32) + 127u) & ~127u;
    p.ring_off = p.x_off + (uint32_t)((a.x_f32 ? 6 : cols) * bpr * 128);
    const long long room = (227 * 1024) / cps - 1024 - (long long)p.ring_off;
    long long d = room / (NW * CHUNK);
    if (d > MAX_D) d = MAX_D;
    p.depth = (int)d;
    smem = (size_t)p.ring_off + (size_t)(d > 0 ? d : 0) * NW * CHUNK;
    return d >= 2;
}

}  // namespace

bool cn_rows_fits(const RowsCall& a) {
    RowsParams p = {};
    size_t smem;
    return a.k > 0 && a.k % 256 == 0 && layout(a, 1, p, smem);
}

int cn_rows_launch(const RowsCall& a, cudaStream_t stream, const char* who) {
    RowsParams p = {};
    size_t smem;
    if (a.rows <= 0 || a.k <= 0 || a.k % 256 != 0) CN_FAIL(CN_ERR_SHAPE, "%s: k = %d must be a positive multiple of 256", who, a.k);
    if (((uintptr_t)a.w0 | (uintptr_t)a.w1 | (uintptr_t)a.x) & 15)  // 16-byte asynchronous copies and 128-bit loads
        CN_FAIL(CN_ERR_SHAPE, "%s: weight and activation pointers must be 16-byte aligned", who);
    int cps = 2;
    if (!layout(a, 2, p, smem)) {
        cps = 1;
        if (!layout(a, 1, p, smem)) CN_FAIL(CN_ERR_LIMIT, "%s: k = %d leaves no room for a weight ring beside the activation rows", who, a.k);
    }
    p.c = a;
    if (!p.c.gs1) p.c.gs1 = a.gs0;
    const bool gu = a.tab1 || a.w1 || a.fused_up_rows > 0;
    const int T = (a.rows + (gu ? 8 : 16) - 1) / (gu ? 8 : 16);
    // CTAs per group: four rounds of CTAs if every group were there, but at least two tiles for each warp
    p.parts = (4 * 148 * cps + a.max_groups - 1) / a.max_groups;
    if (p.parts > T / (2 * NW)) p.parts = T / (2 * NW);
    if (p.parts < 1) p.parts = 1;
    // CTAs walk the groups: four rounds of CTAs at most, so that a list much shorter than its bound (the inbox of an
    // expert-parallel rank) costs no more than that
    int gy = (4 * 148 * cps + p.parts - 1) / p.parts;
    if (gy > a.max_groups) gy = a.max_groups;
    const dim3 grid((unsigned)p.parts, (unsigned)gy);
#define CN_ROWS_CASE(NPLV, CPSV)                                                                                   \
    if (a.x_f32 == (NPLV == 3) && cps == CPSV) {                                                                   \
        CN_ALLOW_SMEM((nvfp4_rows_kernel<NPLV, CPSV>), 226 * 1024);                                                \
        CN_CUDA(cn_launch_pdl((nvfp4_rows_kernel<NPLV, CPSV>), grid, dim3(NW * 32), smem, stream, p));             \
        return CN_OK;                                                                                              \
    }
    CN_ROWS_CASE(1, 1) CN_ROWS_CASE(1, 2) CN_ROWS_CASE(3, 1) CN_ROWS_CASE(3, 2)
#undef CN_ROWS_CASE
    return CN_OK;
}
