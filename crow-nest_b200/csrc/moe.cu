// The routed-expert decode step over NVFP4 experts: grouped expert GEMVs after top-k routing, the
// shared expert, and the weighted combine.
//
// Supersedes the routed half of Engine::moe_run (engine/src/gen.rs:4168-4532): gemv_fp4_ptrb over
// the gate|up and down pointer tables (engine/src/kernels.rs:195-233), silu_mul_combo (:1562),
// acc_combo (:1583) and gate_shared (:1593); the operator shape follows GpuMoePlan
// (engine/src/glm5_moe.rs:518-793): a plan owns its scratch, run() only enqueues.
//
// B200 shape of the step: combos (token, rank) are sorted by expert on the device, so the CTAs
// that read one expert's matrices run back to back and every expert's bytes cross HBM once per
// step (repeats are L2 hits); gate, up and the activation are one launch; a null table entry
// skips the combo (the expert lives on another rank).
#include "common.cuh"
#include "moe_step.cuh"
#include "nvfp4_digits.cuh"
#include "nvfp4_gemv.cuh"

namespace {

// order[] = combos sorted by expert id (negative ids last); one CTA of 1024 threads, counting sort in shared memory
__global__ void moe_sort_kernel(const int32_t* __restrict__ ids, int32_t* __restrict__ order, int n, int E) {
    extern __shared__ int cnt[];  // [E + 2] counts, then start offsets; [n] the combos' bins
    int* bin = cnt + E + 2;
    __shared__ int wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i <= E + 1; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    for (int c = tid; c < n; c += blockDim.x) {
        const int e = ids[c];
        const int b = (e < 0 || e >= E) ? E : e;
        bin[c] = b;
        atomicAdd(&cnt[b], 1);
    }
    __syncthreads();
    // exclusive prefix sum over the E + 1 bins: every thread takes a contiguous run, the runs' totals are scanned
    // with warp shuffles
    const int per = (E + 1 + (int)blockDim.x - 1) / (int)blockDim.x;
    const int i0 = tid * per, i1 = min(i0 + per, E + 1);
    int mine = 0;
    for (int i = i0; i < i1; i++) mine += cnt[i];
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int w = wsum[lane], winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += v;
        }
        wsum[lane] = winc - w;  // exclusive
    }
    __syncthreads();
    int run = wsum[wid] + inc - mine;
    for (int i = i0; i < i1; i++) {
        const int c = cnt[i];
        cnt[i] = run;
        run += c;
    }
    __syncthreads();
    // stable within an expert: each combo counts the earlier combos of its expert (n is small)
    for (int c = tid; c < n; c += blockDim.x) {
        const int b = bin[c];
        int before = 0;
        for (int d = 0; d < c; d++) before += bin[d] == b;
        order[cnt[b] + before] = c;
    }
}

__device__ __forceinline__ bool resident(int e, const unsigned long long* __restrict__ tab, int E) { return e >= 0 && e < E && !(tab && tab[e] == 0ull); }

template <bool F32>
__device__ __forceinline__ void one_chunk(const DigitsCall& dc, size_t i, int lane) {
    ChunkValues<F32> v;
    v.load((const char*)dc.x + i * (256 * (F32 ? 4 : 2)), lane);
    put_record<F32>(v, lane, dc.out + i * digit_record(F32));
}
// Records of the chunks of activations, more than there are warps. Rows none of whose combos has a resident expert are left out, since nothing reads them and most inbox slots of an
// expert-parallel rank are such rows: one rank of eight, 512 experts of 2048 x 512, top 10, 64 tokens a rank (637 of 5120 slots in use), routed experts 91.9 -> 80.1 us. A lane looks one of the
// warp's chunks up, the ids and then the entries of four combos at a time. The first chunk of a warp is made without a look, as are all where every warp has one at most: they are made beside
// the grouping on SMs that have nothing else to do, and two more trips to memory in front of them show (160 slots 23.0 -> 23.3 us).
// A chunk is a call here (inlined into the loop the kernel has 56 registers, not 40, and a block of it an SM to itself: seven tokens of 128 experts of 2560 x 768, top 6, 43.0 -> 43.5 us), and inline code where a
// warp has one.
template <bool F32>
__device__ __noinline__ void far_chunk(const DigitsCall& dc, size_t i, int lane) {
    one_chunk<F32>(dc, i, lane);
}
template <bool F32>
__device__ __forceinline__ void put_records(const DigitsCall& dc, const int32_t* __restrict__ ids, const unsigned long long* __restrict__ tab, int n, int E, int w, int warps, int lane) {
    for (int i0 = w; i0 < dc.chunks; i0 += 32 * warps) {
        const int at = i0 + lane * warps;
        bool read = at == w;
        if (!read && at < dc.chunks) {
            const int c0 = at / dc.row_chunks * dc.x_div, c1 = min(c0 + dc.x_div, n);
#pragma unroll 1
            for (int c = c0; c < c1 && !read; c += 4) {
                int e[4];
#pragma unroll
                for (int j = 0; j < 4; j++) e[j] = c + j < c1 ? ids[c + j] : -1;
#pragma unroll
                for (int j = 0; j < 4; j++) read |= resident(e[j], tab, E);
            }
        }
#pragma unroll 1
        for (uint32_t todo = __ballot_sync(0xffffffffu, read); todo; todo &= todo - 1u) far_chunk<F32>(dc, (size_t)(i0 + (__ffs(todo) - 1) * warps), lane);
    }
}

// Sort the combos by expert and cut every expert's run into groups of up to gmax rows, gmax 4 or 8 (one CTA of 1024 threads):
//   order[]           the combos sorted by expert, stable; combos without a resident expert (id outside 0..E-1, or a
//                     null entry of `tab`) last, in any order, and in no group
//   ga[] / counts[0]  positions (in order[]) of the one-row groups: an expert's single row, or the one left over after
//                     its groups of gmax
//   gb[], gbrows[] / counts[1]  first positions and row counts (2..gmax) of the other groups
// Placement: every combo counts the earlier ones among its expert's (the list in shared memory, in the order of the counting atomics), which keeps the sort
// stable; where an expert has more than LONG_RUN rows, or the list does not fit (listed = 0), one warp walks the combos in order instead (match.any finds the lanes of a
// step that share an expert; 20 dependent steps for 640 combos). A step of 64 tokens, top 10 of 512 experts: 203.0 -> 199.9 us, replayed 199.5 -> 198.8.
constexpr int LONG_RUN = 64;
__global__ void __launch_bounds__(1024) moe_group_kernel(const int32_t* __restrict__ ids, const unsigned long long* __restrict__ tab, int n, int E,
                                                         int32_t* __restrict__ order, int* __restrict__ ga, int* __restrict__ gb,
                                                         int* __restrict__ gbrows, int* __restrict__ counts, int gmax, int listed, const DigitsCall dc) {
    extern __shared__ int sm[];  // [E + 1] counts, [E + 1] starts, [E + 1] running, [n] bins, [n] the experts' combos (listed)
    int* cnt = sm;
    int* start = sm + (E + 1);
    int* run = sm + 2 * (E + 1);
    int* bin = sm + 3 * (E + 1);  // expert in the low 14 bits (as many fit beside each other), place among the expert's combos above
    int* list = bin + n;
    __shared__ int wsa[32], wsb[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    // The kernels that take the lists wait before they read them; their launch, barriers and tensor memory go on meanwhile: 64 tokens, top 10 of 512 experts
    // 207.1 -> 197.5 us a step, MUL1 with 16 tokens 266.4 -> 264.3.
    pdl_launch_dependents();
    pdl_wait();
    if (blockIdx.x > 0) {  // not the grouping
        const int w = ((int)blockIdx.x - 1) * 32 + wid, warps = ((int)gridDim.x - 1) * 32;
        if (dc.chunks > warps) {
            if (dc.f32)
                put_records<true>(dc, ids, tab, n, E, w, warps, lane);
            else
                put_records<false>(dc, ids, tab, n, E, w, warps, lane);
        } else if (w < dc.chunks) {
            if (dc.f32)
                one_chunk<true>(dc, w, lane);
            else
                one_chunk<false>(dc, w, lane);
        }
        return;
    }
    for (int i = tid; i <= E; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    for (int c = tid; c < n; c += blockDim.x) {
        const int e = ids[c];
        const int b = resident(e, tab, E) ? e : E;
        bin[c] = b | atomicAdd(&cnt[b], 1) << 14;
    }
    __syncthreads();
    // per expert: one-row groups and larger groups, then three exclusive prefix sums over the experts (rows, a, b)
    const int per = (E + 1 + (int)blockDim.x - 1) / (int)blockDim.x;
    const int i0 = min(tid * per, E + 1), i1 = min(i0 + per, E + 1);
    int rows = 0, na = 0, nb = 0;
    for (int i = i0; i < i1; i++) {
        const int k = cnt[i];
        rows += k;
        if (i < E) na += (k % gmax) == 1, nb += k / gmax + ((k % gmax) >= 2);
    }
    int ir = rows, ia = na, ib = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int vr = __shfl_up_sync(0xffffffffu, ir, o), va = __shfl_up_sync(0xffffffffu, ia, o), vb = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) ir += vr, ia += va, ib += vb;
    }
    __shared__ int wsr[32];
    if (lane == 31) wsr[wid] = ir, wsa[wid] = ia, wsb[wid] = ib;
    __syncthreads();
    if (wid == 0) {
        int r = wsr[lane], a = wsa[lane], b = wsb[lane];
        const int r0 = r, a0 = a, b0 = b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int vr = __shfl_up_sync(0xffffffffu, r, o), va = __shfl_up_sync(0xffffffffu, a, o), vb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) r += vr, a += va, b += vb;
        }
        wsr[lane] = r - r0, wsa[lane] = a - a0, wsb[lane] = b - b0;
        if (lane == 31) counts[0] = a, counts[1] = b;
    }
    __syncthreads();
    int pr = wsr[wid] + ir - rows, pa = wsa[wid] + ia - na, pb = wsb[wid] + ib - nb;
    bool walk = !listed;
    for (int i = i0; i < i1; i++) {
        const int k = cnt[i];
        walk |= k > LONG_RUN && i < E;
        start[i] = pr;
        run[i] = pr;
        if (i < E) {
            for (int q = 0; q < k / gmax; q++) gb[pb] = pr + gmax * q, gbrows[pb] = gmax, pb++;
            const int rem = k % gmax, at = pr + k - rem;
            if (rem == 1) ga[pa++] = at;
            if (rem >= 2) gb[pb] = at, gbrows[pb] = rem, pb++;
        }
        pr += k;
    }
    if (!__syncthreads_or(walk)) {
        for (int c = tid; c < n; c += blockDim.x) list[start[bin[c] & 0x3fff] + (bin[c] >> 14)] = c;
        __syncthreads();
        for (int c = tid; c < n; c += blockDim.x) {
            const int b = bin[c] & 0x3fff, at = start[b], k = b < E ? cnt[b] : 0;
            int before = b < E ? 0 : bin[c] >> 14;  // (nothing reads the order of those without an expert)
            for (int i = 0; i < k; i++) before += list[at + i] < c;
            order[at + before] = c;
        }
        return;
    }
    if (wid == 0) {
        for (int c0 = 0; c0 < n; c0 += 32) {
            const int c = c0 + lane;
            const int b = c < n ? bin[c] & 0x3fff : -1 - lane;  // lanes beyond the end match nobody
            const unsigned same = __match_any_sync(0xffffffffu, b);
            if (c < n) {
                const int base = run[b];
                order[base + __popc(same & ((1u << lane) - 1u))] = c;
            }
            __syncwarp();
            if (c < n && lane == __ffs(same) - 1) run[b] += __popc(same);
            __syncwarp();
        }
    }
}

// y[t][c] = base + sum_j w[t][j] * eo[t*K + j][c], j in pick order; base = shared[t][c]
// (times sigmoid(sgate[t]) when gated), 0 without a shared expert. A combo whose expert has no
// local matrix contributes nothing.
template <int YT>
__global__ void moe_combine_kernel(const float* __restrict__ eo, const float* __restrict__ wts, const int32_t* __restrict__ ids,
                                   const unsigned long long* __restrict__ tab, const float* __restrict__ shared,
                                   const float* __restrict__ sgate, void* __restrict__ y, int H, int K, int E) {
    // the token's K weights and "has a local matrix" flags once per CTA, so that the K loads of a column do not
    // wait on an id -> table -> value chain each
    constexpr int KC = 16;
    __shared__ float s_w[KC];
    __shared__ int s_ok[KC];
    const int c = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    float acc = 0.0f;
    for (int j0 = 0; j0 < K; j0 += KC) {
        const int kc = min(KC, K - j0);
        if (j0 > 0) __syncthreads();
        if ((int)threadIdx.x < kc) {
            const int e = ids[t * K + j0 + threadIdx.x];
            s_ok[threadIdx.x] = !(e < 0 || (E > 0 && e >= E) || (tab && tab[e] == 0ull));
            s_w[threadIdx.x] = wts[t * K + j0 + threadIdx.x];
        }
        __syncthreads();
        if (c < H) {
            float v[KC];
#pragma unroll
            for (int j = 0; j < KC; j++) v[j] = (j < kc && s_ok[j]) ? eo[((size_t)t * K + j0 + j) * H + c] : 0.0f;
#pragma unroll
            for (int j = 0; j < KC; j++)
                if (j < kc && s_ok[j]) acc = __fadd_rn(acc, __fmul_rn(s_w[j], v[j]));
        }
    }
    if (c >= H) return;
    float base = shared ? shared[(size_t)t * H + c] : 0.0f;
    if (shared && sgate) base = __fmul_rn(1.0f / (1.0f + expf(-sgate[t])), base);
    const float v = __fadd_rn(base, acc);
    if (YT == 1)
        ((__nv_bfloat16*)y)[(size_t)t * H + c] = __float2bfloat16_rn(v);
    else
        ((float*)y)[(size_t)t * H + c] = v;
}

// Combos from which the routed step groups the rows of an expert (measured: see routed_experts), and fewer of larger experts: one by one, each combo streams its expert, and f32 rows take CUDA
// cores. The line is where grouping is no slower with or without a shared expert, in combos x hidden x inter. us per step without / with one of 512, one by one / grouped, f32 rows: 31.5 M (30 combos of 2048 x 512, 512
// experts) 29.9 / 30.9 and 30.9 / 34.2, 37.7 M (36) 31.9 / 30.5 and 38.1 / 39.4, 41.9 M (40) 37.4 / 35.7 and 39.3 / 39.1, 41.9 M (32 of 2560 x 512) 35.5 / 34.0 and 39.3 / 39.0, 47.2 M (30 of 2048 x 768) 47.6 / 37.5 and
// 47.3 / 39.5, 52.4 M (40 of 1024 x 1280, 64 experts) 53.6 / 33.9 and 61.1 / 39.2. bf16 rows: 62.9 M (40 of 2048 x 768) 36.9 / 40.9 and 40.0 / 42.3, 70.8 M (36 of 2560 x 768, 128 experts) 39.1 / 41.0 and 47.5 / 48.1, 78.6 M
// (30 of 2048 x 1280, 64 experts) 40.8 / 41.4 and 47.0 / 46.2, 82.6 M (42 of 2560 x 768) 43.7 / 42.9 and 51.6 / 50.0, 98.3 M (30 of 2560 x 1280) 50.1 / 46.5 and 56.6 / 54.0; 16 combos of 4096 x 2048 (134 M) 56.5 / 61.6 and 58.2 / 63.1.
// A rank that holds an eighth of the experts gains more, since dead combos are in no group: 24 combos of 4096 x 2048, three of them live, 44.9 / 31.7, f32 36.1 / 31.6; 16 of f32 29.2 / 28.2.
constexpr int GROUP_COMBOS = 48, GROUP_LEAST = 16;
bool groups_rows(int combos, int hidden, int inter, bool f32) {
    return combos >= GROUP_COMBOS || (combos >= (f32 ? GROUP_LEAST : 24) && (long long)combos * hidden * inter >= (f32 ? 40000000 : 80000000));
}
// Blocks of the grouping kernel that make records at most: one to an SM (1024 threads of 40 registers) beside the one that groups.
constexpr int DIGIT_BLOCKS = 148 - 1;
// Bytes of a plan's store of digits at most.
constexpr size_t DIGITS_MOST = (size_t)64 << 20;

struct MoePlan {
    int hidden, inter, experts, topk, max_tokens, device;
    float* h;        // [max_tokens * topk][inter]
    float* eo;       // [max_tokens * topk][hidden]
    float* hs;       // [max_tokens][shared inter <= inter_s]
    float* ys;       // [max_tokens][hidden]
    int32_t* order;  // [max_tokens * topk]; groups and xd lie behind it
    int* groups;     // [3 * max_tokens * topk + 8]: the group lists of moe_group_kernel and their two counts
    uint8_t* xd;     // records of the digits of x; null where there is no room for them
    size_t xd_bytes;
    int shared_inter;
    // the shared expert does not depend on the routed experts until the combine: it is enqueued on a side stream
    // between two events (fork after the caller's earlier work, join before the combine), also under stream capture
    cudaStream_t side;
    cudaEvent_t fork, join;
    bool shared_pending;  // cn_moe_nvfp4_shared_begin has enqueued the shared expert; the next finish joins it
};

}  // namespace

// the grouping step for other operators of the library (declared in nvfp4_gemv.cuh): lists of `combos` ints each, counts of 2
int cn_moe_group_launch(const int32_t* ids, const unsigned long long* tab, int combos, int experts, int32_t* order, int* ga, int* gb, int* gbrows,
                        int* counts, int gmax, cudaStream_t stream, const DigitsCall& digits) {
    if (gmax != 4 && gmax != 8) CN_FAIL(CN_ERR_SHAPE, "grouping: groups of %d rows (4 or 8)", gmax);
    const size_t smem = (size_t)(3 * (experts + 1) + combos) * sizeof(int);
    if (smem > 160 * 1024) CN_FAIL(CN_ERR_LIMIT, "grouping %d combos over %d experts needs %zu B of shared memory", combos, experts, smem);
    CN_ALLOW_SMEM(moe_group_kernel, 160 * 1024);
    const size_t listed = smem + (size_t)combos * sizeof(int);
    const bool fits = listed <= 160 * 1024;
    const int more = (digits.chunks + 31) / 32, blocks = 1 + (more < DIGIT_BLOCKS ? more : DIGIT_BLOCKS);
    CN_CUDA(cn_launch_pdl(moe_group_kernel, dim3((unsigned)blocks), dim3(1024), fits ? listed : smem, stream, ids, tab, combos, experts, order, ga, gb, gbrows, counts, gmax, (int)fits, digits));
    return CN_OK;
}

extern "C" int cn_moe_sort(const int32_t* ids, int32_t* order, int combos, int experts, cn_stream_t stream) {
    if (combos < 1 || experts < 1 || experts > 8192) CN_FAIL(CN_ERR_SHAPE, "cn_moe_sort: %d combos over %d experts", combos, experts);
    const size_t smem = (size_t)(experts + 2 + combos) * sizeof(int);
    if (smem > 48 * 1024) CN_FAIL(CN_ERR_LIMIT, "cn_moe_sort: %d combos over %d experts need %zu B of shared memory", combos, experts, smem);
    moe_sort_kernel<<<1, 1024, smem, (cudaStream_t)stream>>>(ids, order, combos, experts);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

extern "C" int cn_moe_combine(const float* eo, const float* wts, const int32_t* ids, const unsigned long long* table, const float* shared,
                              const float* sgate, void* y, int tokens, int hidden, int topk, int experts, int dtype, cn_stream_t stream) {
    if (tokens < 1 || hidden < 1 || topk < 1) CN_FAIL(CN_ERR_SHAPE, "cn_moe_combine: tokens %d hidden %d topk %d", tokens, hidden, topk);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_combine: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    dim3 grid((hidden + 255) / 256, tokens);
    if (dtype == CN_BF16)
        moe_combine_kernel<1><<<grid, 256, 0, (cudaStream_t)stream>>>(eo, wts, ids, table, shared, sgate, y, hidden, topk, experts);
    else
        moe_combine_kernel<0><<<grid, 256, 0, (cudaStream_t)stream>>>(eo, wts, ids, table, shared, sgate, y, hidden, topk, experts);
    CN_CUDA(cudaGetLastError());
    return CN_OK;
}

extern "C" int cn_moe_nvfp4_plan_destroy(void* plan);

extern "C" int cn_moe_nvfp4_plan_create(void** plan_out, int hidden, int inter, int shared_inter, int experts, int topk, int max_tokens) {
    if (!plan_out || hidden % 256 || inter % 256 || shared_inter % 256 || experts < 1 || topk < 1 || max_tokens < 1)
        CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_plan_create: hidden %d, inter %d, shared inter %d must be multiples of 256", hidden, inter, shared_inter);
    MoePlan* p = new MoePlan();
    p->hidden = hidden, p->inter = inter, p->experts = experts, p->topk = topk, p->max_tokens = max_tokens, p->shared_inter = shared_inter;
    CN_CUDA(cudaGetDevice(&p->device));
    const size_t combos = (size_t)max_tokens * topk;
    // a failure part-way frees what the earlier steps got (the destroy call takes a half-built plan)
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    step(cudaMalloc(&p->h, combos * inter * sizeof(float)));
    step(cudaMalloc(&p->eo, combos * hidden * sizeof(float)));
    step(cudaMalloc(&p->hs, (size_t)max_tokens * (shared_inter > 0 ? shared_inter : 1) * sizeof(float)));
    step(cudaMalloc(&p->ys, (size_t)max_tokens * hidden * sizeof(float)));
    // lists, and behind them records of the digits of x for the grouped step, bounded; without them (and for more rows than they hold) the digits are made where they are used, which has the same bits
    const size_t order_bytes = (combos * sizeof(int32_t) + 255) / 256 * 256, group_bytes = ((3 * combos + 8) * sizeof(int) + 255) / 256 * 256;
    p->xd_bytes = combos < GROUP_LEAST ? 0 : (size_t)max_tokens * (hidden / 256) * digit_record(true);
    if (p->xd_bytes > DIGITS_MOST) p->xd_bytes = DIGITS_MOST;
    uint8_t* lists = nullptr;
    if (e == cudaSuccess && p->xd_bytes && cudaMalloc(&lists, order_bytes + group_bytes + p->xd_bytes) != cudaSuccess) {
        (void)cudaGetLastError();
        lists = nullptr, p->xd_bytes = 0;
    }
    if (!lists) step(cudaMalloc(&lists, order_bytes + group_bytes));
    if (lists) p->order = (int32_t*)lists, p->groups = (int*)(lists + order_bytes), p->xd = p->xd_bytes ? lists + order_bytes + group_bytes : nullptr;
    step(cudaStreamCreateWithFlags(&p->side, cudaStreamNonBlocking));
    step(cudaEventCreateWithFlags(&p->fork, cudaEventDisableTiming));
    step(cudaEventCreateWithFlags(&p->join, cudaEventDisableTiming));
    if (e != cudaSuccess) {
        cn_moe_nvfp4_plan_destroy(p);
        CN_FAIL(CN_ERR_CUDA, "cn_moe_nvfp4_plan_create: %s", cudaGetErrorString(e));
    }
    *plan_out = p;
    return CN_OK;
}

extern "C" int cn_moe_nvfp4_plan_destroy(void* plan) {
    MoePlan* p = (MoePlan*)plan;
    if (!p) return CN_OK;
    cudaFree(p->h), cudaFree(p->eo), cudaFree(p->hs), cudaFree(p->ys), cudaFree(p->order);
    if (p->side) cudaStreamDestroy(p->side);
    if (p->fork) cudaEventDestroy(p->fork);
    if (p->join) cudaEventDestroy(p->join);
    delete p;
    return CN_OK;
}

namespace {

// a shared expert takes all of its matrices and scales, and a plan that was made for one; checked before anything is enqueued
int check_shared(const MoePlan* p, const void* shared_gate, const void* shared_up, const void* shared_down, const float* shared_gs, const char* who) {
    if (!shared_gate || !shared_up || !shared_down || !shared_gs) CN_FAIL(CN_ERR_SHAPE, "%s: null matrix or scales of the shared expert", who);
    if (p->shared_inter <= 0) CN_FAIL(CN_ERR_SHAPE, "%s: the plan was made without a shared expert", who);
    return CN_OK;
}

constexpr int MAX_ROW = 32768;  // values of a row in the kernel for groups of rows; longer ones are left to the GEMVs, which know their limits

// whether these combos run in groups: by the rule, where the rows and the grouping's shared memory allow it
bool grouped(const MoePlan* p, int combos, bool f32) {
    return groups_rows(combos, p->hidden, p->inter, f32) && p->hidden <= MAX_ROW && p->inter <= MAX_ROW && (size_t)(3 * (p->experts + 1) + combos) * sizeof(int) <= 160 * 1024;
}

}  // namespace

extern "C" int cn_moe_nvfp4_plan_digits(void* plan, void** records, size_t* bytes) {
    const MoePlan* p = (const MoePlan*)plan;
    if (!p || !records || !bytes) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_plan_digits: null argument");
    *records = p->xd, *bytes = p->xd_bytes;
    return CN_OK;
}

namespace {

// the shared expert on every token, up to 8 rows per pass, on the plan's side stream between the fork and join events:
// whatever happens after the fork, the side stream is joined again (a capture of the caller's stream stays valid)
int shared_branch(MoePlan* p, const void* shared_gate, const void* shared_up, const void* shared_down, const float* shared_gs, const void* x,
                  int tokens, float limit, int dtype, cudaStream_t stream) {
    CN_CUDA(cudaEventRecord(p->fork, stream));
    CN_CUDA(cudaStreamWaitEvent(p->side, p->fork, 0));
    const size_t es = dtype == CN_BF16 ? 2 : 4;
    int rc = CN_OK;
    // More rows than a GEMV takes: both projections as one launch each over groups of eight rows (64 tokens, 512 x 2048: 22 and 11 us with the mma.sync kernel that
    // took groups of eight bf16 or two f32 rows; the step 204 -> 199).
    const bool grouped = tokens > CN_MAX_M && p->hidden <= MAX_ROW && p->shared_inter <= MAX_ROW;
    if (grouped) {
        RowsCall u = {}, d = {};
        u.w0 = shared_gate, u.w1 = shared_up, u.m = tokens, u.gs0 = shared_gs, u.gs1 = shared_gs + 1, u.x = x, u.x_div = 1, u.x_f32 = dtype == CN_F32;
        u.y = p->hs, u.ldy = p->shared_inter, u.rows = p->shared_inter, u.k = p->hidden, u.limit = limit, u.max_groups = (tokens + 7) / 8;
        d.w0 = shared_down, d.m = tokens, d.gs0 = shared_gs + 2, d.x = p->hs, d.x_div = 1, d.x_f32 = 1, d.y = p->ys, d.ldy = p->hidden, d.rows = p->hidden;
        d.k = p->shared_inter, d.max_groups = (tokens + 7) / 8;
        rc = cn_rows_launch(u, p->side, "cn_moe_nvfp4_run (shared gate/up)");
        if (rc == CN_OK) rc = cn_rows_launch(d, p->side, "cn_moe_nvfp4_run (shared down)");
    }
    for (int t0 = 0; !grouped && t0 < tokens && rc == CN_OK; t0 += CN_MAX_M) {
        const int m = tokens - t0 < CN_MAX_M ? tokens - t0 : CN_MAX_M;
        GemvCall g = {};
        g.w0 = shared_gate, g.w1 = shared_up, g.gs0 = shared_gs, g.gs1 = shared_gs + 1, g.x = (const char*)x + (size_t)t0 * p->hidden * es;
        g.y = p->hs + (size_t)t0 * p->shared_inter, g.rows = p->shared_inter, g.k = p->hidden, g.m = m, g.ldy = p->shared_inter;
        g.limit = limit, g.dtype = dtype, g.out_f32 = 1;
        rc = cn_gemv_launch(g, p->side, "cn_moe_nvfp4_run (shared gate/up)");
        if (rc != CN_OK) break;
        GemvCall s = {};
        s.w0 = shared_down, s.gs0 = shared_gs + 2, s.x = p->hs + (size_t)t0 * p->shared_inter, s.y = p->ys + (size_t)t0 * p->hidden;
        s.rows = p->hidden, s.k = p->shared_inter, s.m = m, s.ldy = p->hidden, s.dtype = CN_F32, s.out_f32 = 1;
        rc = cn_gemv_launch(s, p->side, "cn_moe_nvfp4_run (shared down)");
    }
    CN_CUDA(cudaEventRecord(p->join, p->side));
    return rc;
}

// ... and from which the ungrouped down projection runs on the tensor cores (measured: see routed_experts).
constexpr int ROWS_COMBOS = 16;
// Units of work (16 result rows of a token x eight 64-value blocks of an expert) up to which a step of that many combos runs in two launches
// (measured: see cn_moe_nvfp4_run).
constexpr long long STEP_UNITS = 8192;

// Routed gate|up of the combos as they come (nearly every CTA of a small step is resident at once and L2 serves an expert's second
// reader).
GemvCall routed_gate_up(const MoePlan* p, const unsigned long long* table_gu, const unsigned long long* table_up, const float* gs_gu, const float* gs_up,
                        const int32_t* ids, const void* x, int combos, int x_div, float limit, int dtype) {
    GemvCall a = {};
    a.gs0 = gs_gu, a.gs1 = gs_up ? gs_up : gs_gu, a.x = x, a.y = p->h, a.rows = p->inter, a.k = p->hidden, a.m = 1, a.ldy = p->inter;
    a.limit = limit, a.dtype = dtype, a.out_f32 = 1, a.ids = ids, a.order = nullptr, a.tab0 = table_gu, a.tab1 = table_up;
    a.fused_up_rows = table_up ? 0 : p->inter, a.x_div = x_div, a.combos = combos, a.experts = p->experts;
    return a;
}

// routed gate|up + activation, then routed down, one launch each over `combos` (token, pick) pairs: combo c reads
// activation row c / x_div and writes eo row c (or to eo_ptrs[c] when given: a row of another buffer, e.g. in a peer's memory)
int routed_experts(MoePlan* p, const unsigned long long* table_gu, const unsigned long long* table_up, const unsigned long long* table_dn,
                   const float* gs_gu, const float* gs_up, const float* gs_dn, const int32_t* ids, const void* x, float* eo,
                   const unsigned long long* eo_ptrs, int combos, int x_div, float limit, int dtype, cudaStream_t stream) {
    const GemvCall a = routed_gate_up(p, table_gu, table_up, gs_gu, gs_up, ids, x, combos, x_div, limit, dtype);
    const bool short_rows = p->hidden <= MAX_ROW && p->inter <= MAX_ROW;
    // From 48 combos on (and fewer of large experts) the combos are sorted by expert and cut into groups of up to eight rows that share one pass over the expert's weights (nvfp4_rows_tc.cu).
    // us per step (64 tokens, 512 experts of 2048 x 512, top 10, unless said otherwise) now / with mma.sync kernels that decoded the weights to f16 for eight bf16
    // or two f32 rows: 163 / 213, 128 tokens 230 / 323, 16 tokens 82 / 109, f32 rows 177 / 234; 64 experts of 1024 x 1280, top 8, 108 tokens 129 / 198;
    // 288 experts of 4096 x 2048, top 8, 10 tokens 175 / 239. Fewer combos: see `groups_rows`.
    if (grouped(p, combos, dtype == CN_F32)) {
        int* ga = p->groups;
        int* gb = ga + combos;
        int* gbrows = gb + combos;
        int* counts = gbrows + combos;
        RowsCall u = {};
        u.ids = ids, u.order = p->order, u.tab0 = table_gu, u.tab1 = table_up, u.fused_up_rows = a.fused_up_rows, u.gs0 = a.gs0, u.gs1 = a.gs1;
        u.x = x, u.x_div = x_div, u.x_f32 = dtype == CN_F32, u.y = p->h, u.ldy = p->inter, u.rows = p->inter, u.k = p->hidden, u.limit = limit;
        u.max_groups = combos < p->experts + combos / 8 ? combos : p->experts + combos / 8;  // an expert ends in one short group
        u.count1 = counts, u.pos1 = ga, u.count2 = counts + 1, u.pos2 = gb, u.rows2 = gbrows;
        RowsCall d = {};
        d.ids = ids, d.order = p->order, d.tab0 = table_dn, d.gs0 = gs_dn, d.x = p->h, d.x_div = 1, d.x_f32 = 1, d.y = eo, d.yptrs = eo_ptrs, d.ldy = p->hidden;
        d.rows = p->hidden, d.k = p->inter, d.max_groups = u.max_groups;
        d.count1 = counts, d.pos1 = ga, d.count2 = counts + 1, d.pos2 = gb, d.rows2 = gbrows;
        const bool f32 = dtype == CN_F32;
        const long long x_chunks = (long long)((combos + x_div - 1) / x_div) * (p->hidden / 256);
        // The digits of x are made once, beside the grouping, and not by every tile of gate / up: us per step without a shared expert, a graph of twelve with other picks, in each tile / so: 64 tokens 153 / 148,
        // 128 tokens 221 / 203, 64 tokens of f32 165 / 158, 288 experts of 4096 x 2048, 32 tokens 517 / 495, 10 tokens 198 / 197, 64 experts of 1024 x 1280, 108 tokens 137 / 126, 16 tokens of 512 experts 67.3 / 67.7; one rank
        // of eight with 64 tokens 91.8 / 79.8. Those of h, a launch of their own in front of the down projection: 64 tokens 167 / 175, 108 tokens 129 / 122, 128 tokens 234 / 232.
        DigitsCall dx = {};
        if (!((uintptr_t)x & 15) && x_chunks * digit_record(f32) <= (long long)p->xd_bytes) {
            dx.x = x, dx.chunks = (int)x_chunks, dx.row_chunks = p->hidden / 256, dx.x_div = x_div, dx.f32 = f32, dx.out = p->xd;
            u.digits = p->xd;
        }
        if (int rc = cn_moe_group_launch(ids, table_gu, combos, p->experts, p->order, ga, gb, gbrows, counts, 8, stream, dx)) return rc;
        if (int rc = cn_rows_launch(u, stream, "cn_moe_nvfp4 (gate/up, grouped)")) return rc;
        return cn_rows_launch(d, stream, "cn_moe_nvfp4 (down, grouped)");
    }
    if (int rc = cn_gemv_launch(a, stream, "cn_moe_nvfp4 (gate/up)")) return rc;
    // The down projection of 16 combos and more: the combos one by one, on the tensor cores instead of FMAs. us per step now / with the mma.sync kernel that kept a warp
    // to a tile: 288 experts of 4096 x 2048, top 8, 5 tokens 136 / 142, 3 tokens 87 / 90; 64 experts of 2048 x 1280, top 8, 4 tokens 51.5 / 53.3. With FMAs (171 for the
    // first) only fewer are faster: 1 token 56 / 62 with that kernel.
    RowsCall one = {};
    one.ids = ids, one.m = combos, one.tab0 = table_dn, one.gs0 = gs_dn, one.x = p->h, one.x_div = 1, one.x_f32 = 1, one.y = eo, one.yptrs = eo_ptrs;
    one.ldy = p->hidden, one.rows = p->hidden, one.k = p->inter, one.max_groups = combos, one.experts = p->experts;
    if (combos >= ROWS_COMBOS && short_rows) return cn_rows_launch(one, stream, "cn_moe_nvfp4 (down)");
    GemvCall d = {};
    d.gs0 = gs_dn, d.x = p->h, d.y = eo, d.yptrs = eo_ptrs, d.rows = p->hidden, d.k = p->inter, d.m = 1, d.ldy = p->hidden, d.dtype = CN_F32, d.out_f32 = 1;
    d.ids = ids, d.order = nullptr, d.tab0 = table_dn, d.x_div = 1, d.combos = combos, d.experts = p->experts;
    return cn_gemv_launch(d, stream, "cn_moe_nvfp4 (down)");
}

}  // namespace

extern "C" int cn_moe_nvfp4_experts(void* plan, const unsigned long long* table_gu, const unsigned long long* table_up,
                                    const unsigned long long* table_dn, const float* gs_gu, const float* gs_up, const float* gs_dn,
                                    const int32_t* ids, const void* x, float* eo, const unsigned long long* eo_ptrs, int combos, int x_div,
                                    float limit, int dtype, cn_stream_t stream) {
    MoePlan* p = (MoePlan*)plan;
    if (!p) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_experts: null plan");
    if (combos < 1 || combos > p->max_tokens * p->topk) CN_FAIL(CN_ERR_LIMIT, "cn_moe_nvfp4_experts: %d combos, the plan holds %d", combos, p->max_tokens * p->topk);
    if (x_div < 1) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_experts: x_div %d", x_div);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_experts: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    if (!eo && !eo_ptrs) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_experts: no output");
    return routed_experts(p, table_gu, table_up, table_dn, gs_gu, gs_up, gs_dn, ids, x, eo, eo_ptrs, combos, x_div, limit, dtype, (cudaStream_t)stream);
}

extern "C" int cn_moe_nvfp4_shared_begin(void* plan, const void* shared_gate, const void* shared_up, const void* shared_down, const float* shared_gs,
                                         const void* x, int tokens, float limit, int dtype, cn_stream_t stream) {
    MoePlan* p = (MoePlan*)plan;
    if (!p) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_shared_begin: null plan");
    if (int rc = check_shared(p, shared_gate, shared_up, shared_down, shared_gs, "cn_moe_nvfp4_shared_begin")) return rc;
    if (tokens < 1 || tokens > p->max_tokens) CN_FAIL(CN_ERR_LIMIT, "cn_moe_nvfp4_shared_begin: %d tokens, the plan holds %d", tokens, p->max_tokens);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_shared_begin: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    const int rc = shared_branch(p, shared_gate, shared_up, shared_down, shared_gs, x, tokens, limit, dtype, (cudaStream_t)stream);
    p->shared_pending = true;  // also after a failure: the side stream was forked and must be joined
    return rc;
}

extern "C" int cn_moe_nvfp4_finish(void* plan, const void* shared_gate, const void* shared_up, const void* shared_down, const float* shared_gs,
                                   const float* sgate, const int32_t* ids, const float* wts, const unsigned long long* table, const void* x,
                                   const float* eo, void* y, int tokens, float limit, int dtype, cn_stream_t stream_) {
    MoePlan* p = (MoePlan*)plan;
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!p) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_finish: null plan");
    if (tokens < 1 || tokens > p->max_tokens) CN_FAIL(CN_ERR_LIMIT, "cn_moe_nvfp4_finish: %d tokens, the plan holds %d", tokens, p->max_tokens);
    if (dtype != CN_F32 && dtype != CN_BF16) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_finish: dtype %d is neither CN_F32 nor CN_BF16", dtype);
    const float* shared = nullptr;
    int rc = CN_OK;
    if (p->shared_pending) {
        p->shared_pending = false;
        CN_CUDA(cudaStreamWaitEvent(stream, p->join, 0));
        shared = p->ys;
    } else if (shared_gate) {
        if ((rc = check_shared(p, shared_gate, shared_up, shared_down, shared_gs, "cn_moe_nvfp4_finish"))) return rc;
        rc = shared_branch(p, shared_gate, shared_up, shared_down, shared_gs, x, tokens, limit, dtype, stream);
        CN_CUDA(cudaStreamWaitEvent(stream, p->join, 0));
        shared = p->ys;
    }
    if (rc != CN_OK) return rc;
    return cn_moe_combine(eo, wts, ids, table, shared, sgate, y, tokens, p->hidden, p->topk, p->experts, dtype, stream_);
}

extern "C" int cn_moe_nvfp4_run(void* plan, const unsigned long long* table_gu, const unsigned long long* table_up,
                                const unsigned long long* table_dn, const float* gs_gu, const float* gs_up, const float* gs_dn,
                                const void* shared_gate, const void* shared_up, const void* shared_down, const float* shared_gs,
                                const float* sgate, const int32_t* ids, const float* wts, const void* x, void* y, int tokens, float limit,
                                int dtype, cn_stream_t stream_) {
    MoePlan* p = (MoePlan*)plan;
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!p) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_run: null plan");
    if (tokens < 1 || tokens > p->max_tokens) CN_FAIL(CN_ERR_LIMIT, "cn_moe_nvfp4_run: %d tokens, the plan holds %d", tokens, p->max_tokens);
    if (dtype != CN_F32 && dtype != CN_BF16 && dtype != CN_BF16_IN_F32_OUT) CN_FAIL(CN_ERR_SHAPE, "cn_moe_nvfp4_run: dtype %d", dtype);
    const int ydtype = dtype == CN_BF16 ? CN_BF16 : CN_F32;  // expert-parallel partial sums leave in f32
    if (dtype == CN_BF16_IN_F32_OUT) dtype = CN_BF16;
    const float* shared = nullptr;
    int rc = CN_OK;
    if (shared_gate && (rc = check_shared(p, shared_gate, shared_up, shared_down, shared_gs, "cn_moe_nvfp4_run"))) return rc;
    if (tokens * p->topk < GROUP_COMBOS && !grouped(p, tokens * p->topk, dtype == CN_F32)) {
        // A small step in two launches: gate / up of the combos and of the shared expert, then their down projections with the combine. A warp
        // of the second waits for each of its units by itself, so from 16 combos on - where the routed kernel below has a warp per tile with two to
        // four chunks in flight - it is only taken for few units of work. us per step in two launches / with the other kernels (a side stream for
        // the shared expert), units: 512 experts of 2048 x 512, top 10, 4 tokens 37 / 43 (5.6 k); 64 of 2048 x 1280, top 10, 2 tokens 41 / 45 (7.9 k), 4 tokens
        // 71 / 65 (15.9 k); 128 of 2560 x 1280, top 6, 3 tokens 49.5 / 48.5 (9.1 k), 4 tokens 64 / 53 (12.2 k); 128 of 1024 x 1280, top 8, 5 tokens 48.9 / 47.1
        // (7.7 k); 288 of 4096 x 2048, top 8, 2 tokens 84 / 71 (18.4 k), 5 tokens 186 / 151; 1 token 48.5, 54.8 with the kernels for fewer than 16 combos.
        MoeDownCall d = {};
        d.ids = ids, d.wts = wts, d.table = table_dn, d.experts = p->experts, d.topk = p->topk, d.h = p->h, d.gs = gs_dn, d.inter = p->inter;
        d.shared = shared_gate ? shared_down : nullptr, d.hs = p->hs, d.shared_gs = shared_gate ? shared_gs + 2 : nullptr, d.sgate = sgate;
        d.shared_inter = p->shared_inter, d.y = y, d.tokens = tokens, d.hidden = p->hidden, d.out_bf16 = ydtype == CN_BF16;
        if (cn_moe_down_combine_fits(d) && (tokens * p->topk < ROWS_COMBOS || cn_moe_down_combine_units(d) <= STEP_UNITS)) {
            GemvCall a = routed_gate_up(p, table_gu, table_up, gs_gu, gs_up, ids, x, tokens * p->topk, p->topk, limit, dtype);
            if (shared_gate)
                a.side_w0 = shared_gate, a.side_w1 = shared_up, a.side_gs = shared_gs, a.side_y = p->hs, a.side_rows = p->shared_inter, a.side_tokens = tokens;
            if ((rc = cn_gemv_launch(a, stream, "cn_moe_nvfp4_run (gate/up)"))) return rc;
            return cn_moe_down_combine_launch(d, stream);
        }
    }
    if (shared_gate) {
        rc = shared_branch(p, shared_gate, shared_up, shared_down, shared_gs, x, tokens, limit, dtype, stream);
        shared = p->ys;
    }
    if (rc == CN_OK)
        rc = routed_experts(p, table_gu, table_up, table_dn, gs_gu, gs_up, gs_dn, ids, x, p->eo, nullptr, tokens * p->topk, p->topk, limit, dtype, stream);
    if (shared) CN_CUDA(cudaStreamWaitEvent(stream, p->join, 0));
    if (rc != CN_OK) return rc;
    return cn_moe_combine(p->eo, wts, ids, table_dn, shared, sgate, y, tokens, p->hidden, p->topk, p->experts, ydtype, stream_);
}
