"""Experts with their rows in groups (48 combos and more): k that ends in a part of a chunk, row counts that end in a part of a tile,
groups of one, two and eight rows and what is left over, f32 and bf16 rows, the shared expert beyond eight rows."""
import ctypes as C

import numpy as np
import pytest
import torch

from crownest_b200 import CrownestError, device_status, moe, ops, synth
from crownest_b200._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,experts,topk,tokens,shared", [(256, 256, 3, 2, 24, 256), (768, 1280, 5, 2, 33, 512), (2048, 512, 64, 4, 40, 0),
                                                                   (1280, 768, 200, 6, 8, 256), (4096, 256, 2, 2, 60, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_grouped_experts_against_64_bits(hidden, inter, experts, topk, tokens, shared, dtype):
    rng = np.random.default_rng(hidden + inter + tokens)

    def matrix(rows, k):
        return torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()

    gu, dn = [matrix(2 * inter, hidden) for _ in range(experts)], [matrix(hidden, inter) for _ in range(experts)]
    sh = [matrix(shared, hidden), matrix(shared, hidden), matrix(hidden, shared)] if shared else None
    gs_gu, gs_dn = 0.03, 0.7
    w = moe.GpuMoeWeights(hidden, inter, experts, gs_gu, gs_dn, gate_up=gu, down=dn, shared=sh, shared_gs=[0.03, 0.03, 0.7], device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, topk, tokens, shared_inter=shared)
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda().to(dtype)
    logits = torch.from_numpy(rng.standard_normal((tokens, experts)).astype(np.float32)).cuda()
    y = torch.empty_like(x)
    plan.run(w, logits, x, y, router="softmax")
    again = torch.empty_like(y)
    plan.run(w, logits, x, again, router="softmax")
    assert torch.equal(y, again)

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m.view(-1), torch.tensor([gs], dtype=torch.float32, device="cuda"), rows, k)).double().view(rows, k)

    def ffn(g, u, d, xs):
        a = xs @ g.t()
        return (a / (1 + torch.exp(-a)) * (xs @ u.t())) @ d.t()

    ids, wts = plan.ids.view(tokens, topk), plan.wts.view(tokens, topk).double()
    x64, want = x.double(), torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for e in range(experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            full = deq(gu[e], 2 * inter, hidden, gs_gu)
            want.index_add_(0, t, wts[t, j, None] * ffn(full[:inter], full[inter:], deq(dn[e], hidden, inter, gs_dn), x64[t]))
    if shared:
        want += ffn(deq(sh[0], shared, hidden, 0.03), deq(sh[1], shared, hidden, 0.03), deq(sh[2], hidden, shared, 0.7), x64)
    # f32 throughout: two long sums of 1.2e-7 each, a dozen f32 roundings; a bf16 result adds its own rounding of at most 2^-9
    bound = 2e-6 if dtype == torch.float32 else 2.0 ** -9 + 2e-6
    assert (y.double() - want).norm() <= bound * want.norm()
    assert device_status() == 0


# large experts are grouped with fewer combos (either side of the rule: 16 and more of f32 rows, 24 and more of bf16 rows)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [7, 8, 11, 12])
def test_fewer_combos_of_large_experts_against_64_bits(tokens, dtype):
    test_grouped_experts_against_64_bits(4096, 2048, 3, 2, tokens, 256, dtype)


# ... and with as many combos x hidden x inter as it takes (40 M of f32 rows: 19 and 20 tokens; 80 M of bf16 rows: 15 and 16)
@pytest.mark.parametrize("hidden,inter,topk,tokens,dtype", [(2048, 512, 2, 19, torch.float32), (2048, 512, 2, 20, torch.float32), (2048, 1280, 2, 15, torch.bfloat16),
                                                            (2048, 1280, 2, 16, torch.bfloat16)])
@pytest.mark.parametrize("shared", [0, 512])
def test_either_side_of_the_grouping_line_against_64_bits(hidden, inter, topk, tokens, dtype, shared):
    test_grouped_experts_against_64_bits(hidden, inter, 5, topk, tokens, shared, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("large", [3, 8])
@pytest.mark.parametrize("size", [1e4, 1e7])
def test_large_values_over_zero_weights_of_grouped_rows(large, size, dtype):
    """As for the GEMV: `large` values of every sixteen are `size` times the others and meet zero weights of gate and up, in steps of 16 (f32) and 24 combos of large experts. What fixed point
    loses of a block, 2^-31 (bf16: 2^-22) of its largest value, goes through the activation and the down projection, whose rows are held the same way."""
    hidden, inter, experts, topk = 4096, 2048, 8, 8
    tokens = 2 if dtype == torch.float32 else 3
    rng = np.random.default_rng(large)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(large)

    def matrix(rows, k, zeros):
        m = torch.randint(0, 256, (rows * k // 64, 36), dtype=torch.uint8, device="cuda", generator=gen)
        m[:, :4] = (torch.randn((rows * k // 64, 4), device="cuda", generator=gen).abs_() * 0.05).to(torch.float8_e4m3fn).view(torch.uint8)
        codes = m[:, 4:].view(-1, 4, 8)
        codes[:, :, :zeros // 2] = 0
        if zeros % 2:
            codes[:, :, zeros // 2] &= 0xF0
        return m.view(-1)

    gu, dn = [matrix(2 * inter, hidden, large) for _ in range(experts)], [matrix(hidden, inter, 0) for _ in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 0.03, 0.7, gate_up=gu, down=dn, device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, topk, tokens)
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda()
    x.view(tokens, hidden // 16, 16)[:, :, :large] *= size
    x = x.to(dtype)
    ids = torch.stack([torch.randperm(experts, device="cuda", generator=gen) for _ in range(tokens)]).int()
    eo = plan.experts_only(w, ids, x, eo=torch.zeros((tokens * topk, hidden), device="cuda"), x_div=topk).double().view(tokens, topk, hidden)

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m, torch.tensor([gs], dtype=torch.float32, device="cuda"), rows, k), rule=True).double().view(rows, k)

    def product(v, m, bits):
        """v times a matrix, and how far off a row in fixed point may be: the last bit of each block's largest value, and f32 sums."""
        blocks = lambda t: t.abs().view(t.shape[0], -1, 16)
        return v @ m.t(), 2.0 ** -bits * (blocks(v).amax(dim=2) @ blocks(m).sum(dim=2).t()) + 2e-6 * (v.abs() @ m.abs().t())

    x64, bits = x.double(), 31 if dtype == torch.float32 else 22
    for e in range(experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        full, down = deq(gu[e], 2 * inter, hidden, 0.03), deq(dn[e], hidden, inter, 0.7)
        a, da = product(x64[t], full[:inter], bits)
        b, db = product(x64[t], full[inter:], bits)
        s = a / (1 + torch.exp(-a))
        h = s * b
        dh = 1.1 * da * (b.abs() + db) + s.abs() * db + 1e-6 * h.abs()  # the slope of SiLU is 1.1 at most
        y, dy = product(h, down, 31)
        assert ((eo[t, j] - y).abs() <= dy + (1 + 1e-6) * (dh @ down.abs().t())).all()
    assert device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [56, 64, 125])
def test_full_groups_repeat_bit_for_bit(tokens, dtype):
    """Every expert has all tokens: groups of eight rows (and of seven or five at the end), one chunk right behind the other. The accumulators of two chunks in flight lie side by side in
    tensor memory; eight f32 rows fill theirs (the down projection's rows are f32 whatever x is). Every run has the same bits and the right ones."""
    hidden, inter, experts = 768, 1280, 4
    rng = np.random.default_rng(tokens)

    def matrix(rows, k):
        return torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()

    gu, dn = [matrix(2 * inter, hidden) for _ in range(experts)], [matrix(hidden, inter) for _ in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 0.03, 0.7, gate_up=gu, down=dn, device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, experts, tokens)
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda().to(dtype)
    logits = torch.from_numpy(rng.standard_normal((tokens, experts)).astype(np.float32)).cuda()
    runs = [torch.empty_like(x) for _ in range(40)]
    for y in runs:
        plan.run(w, logits, x, y, router="softmax")
    assert all(torch.equal(y, runs[0]) for y in runs)

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m.view(-1), torch.tensor([gs], dtype=torch.float32, device="cuda"), rows, k)).double().view(rows, k)

    ids, wts = plan.ids.view(tokens, experts), plan.wts.view(tokens, experts).double()
    x64, want = x.double(), torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for e in range(experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        full = deq(gu[e], 2 * inter, hidden, 0.03)
        a = x64[t] @ full[:inter].t()
        want.index_add_(0, t, wts[t, j, None] * ((a / (1 + torch.exp(-a)) * (x64[t] @ full[inter:].t())) @ deq(dn[e], hidden, inter, 0.7).t()))
    bound = 2e-6 if dtype == torch.float32 else 2.0 ** -9 + 2e-6  # as above
    assert (runs[0].double() - want).norm() <= bound * want.norm()
    assert device_status() == 0



@pytest.mark.parametrize("tokens", [8, 9, 40])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_shared_matrix_off_16_bytes_is_refused(tokens, which):
    """The refusal is the host's, whether the shared expert's rows go one by one or in groups."""
    hidden, inter, experts, topk = 256, 256, 4, 2
    rng = np.random.default_rng(which)

    def matrix(rows, k, off=0):
        b = synth.nvfp4_matrix(rows, k, rng)
        buf = torch.zeros(b.size + 16, dtype=torch.uint8, device="cuda")
        buf[off:off + b.size] = torch.from_numpy(b).cuda()
        return buf[off:off + b.size]

    sh = [matrix(inter, hidden, 4 if which == i else 0) for i in range(3)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 1.0, 1.0, gate_up=[matrix(2 * inter, hidden)] * experts, down=[matrix(hidden, inter)] * experts, shared=sh,
                          shared_gs=[1.0] * 3, device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, topk, tokens, shared_inter=inter)
    x = torch.randn((tokens, hidden), device="cuda").to(torch.bfloat16)
    with pytest.raises(CrownestError, match="16-byte aligned"):
        plan.run(w, torch.randn((tokens, experts), device="cuda"), x)
    torch.cuda.synchronize()
    assert device_status() == 0


@pytest.mark.parametrize("hidden", [2048, 4096])
def test_grouped_gate_up_sums_are_as_exact_as_single_rows(hidden):
    """f32 gate/up results of bf16 rows in groups of eight, read back through a down matrix with a single one in every row."""
    inter, experts, tokens = 512, 4, 64
    rng = np.random.default_rng(hidden)
    gs = 2.0 ** -5
    gu = [torch.from_numpy(synth.nvfp4_matrix(2 * inter, hidden, rng)).cuda() for _ in range(experts)]
    one = np.zeros((hidden, inter // 64, 36), np.uint8)
    one[:, :, :4] = 0x38
    for r in range(hidden):
        c = r % inter
        one[r, c // 64, 4 + c % 64 // 2] = 2 << (4 * (c & 1))
    dn = [torch.from_numpy(one.reshape(-1)).cuda()] * experts
    w = moe.GpuMoeWeights(hidden, inter, experts, gs, 1.0, gate_up=gu, down=dn, device="cuda")
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda().to(torch.bfloat16)
    ids = torch.from_numpy(rng.integers(0, experts, (tokens, 1)).astype(np.int32)).cuda()
    plan = moe.GpuMoePlan(hidden, inter, experts, 1, tokens)
    h = plan.experts_run(w, ids, torch.ones((tokens, 1), device="cuda"), x, partial=True).double()[:, :inter]
    want = torch.empty_like(h)
    for e in range(experts):
        full = ops.dequant(ops.Fp4(gu[e], torch.tensor([gs], device="cuda"), 2 * inter, hidden)).double().view(2 * inter, hidden)
        t = (ids.view(-1) == e).nonzero().view(-1)
        g = x[t].double() @ full.t()
        want[t] = g[:, :inter] / (1 + torch.exp(-g[:, :inter])) * g[:, inter:]
    # An f32 addition rounds by some 2.5e-8 (rms), so a running sum of n terms is off by 2.5e-8 sqrt(n / 2): n = k / 512 <= 8 for each of the
    # eight, 5e-8; joining them 4e-8; the tensor core's cut at 2^-24, 6e-8; gate and up each, 1.25e-7 together; the activation and the
    # way through the down matrix 6e-8. (A single running sum of k / 64 = 64 terms: 1.4e-7, 2e-7 for gate and up.)
    assert (h - want).norm() <= 1.45e-7 * want.norm()
    assert device_status() == 0


@pytest.mark.parametrize("combos,experts", [(20, 12), (47, 6), (60, 100), (200, 6), (64, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_combos_without_a_resident_expert_are_left_out(combos, experts, dtype):
    """Ids below, at and beyond the tables and null table entries among the rows, one by one (fewer than 48 combos) and in groups of up to
    eight: their output rows stay as they were, the others are what 64 bits give."""
    hidden, inter = 512, 768
    rng = np.random.default_rng(combos + experts)
    gs_gu, gs_dn = 2.0 ** -4, 0.5
    gone = {1, experts - 1} if experts > 2 else {1}
    gu = [None if e in gone else torch.from_numpy(synth.nvfp4_matrix(2 * inter, hidden, rng)).cuda() for e in range(experts)]
    dn = [None if e in gone else torch.from_numpy(synth.nvfp4_matrix(hidden, inter, rng)).cuda() for e in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, gs_gu, gs_dn, gate_up=gu, down=dn, device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, 1, combos)
    ids = rng.integers(-2, experts + 2, combos).astype(np.int32)
    ids[:3] = [-1, experts, 0]
    x = torch.from_numpy(rng.standard_normal((combos, hidden)).astype(np.float32)).cuda().to(dtype)
    eo = torch.full((combos, hidden), 7.0, device="cuda")
    plan.experts_only(w, torch.from_numpy(ids).cuda(), x, eo=eo)
    want = torch.full((combos, hidden), 7.0, dtype=torch.float64, device="cuda")

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m, torch.tensor([gs], device="cuda"), rows, k)).double().view(rows, k)

    live = [c for c in range(combos) if 0 <= ids[c] < experts and ids[c] not in gone]
    for c in live:
        g = deq(gu[ids[c]], 2 * inter, hidden, gs_gu) @ x[c].double()
        want[c] = deq(dn[ids[c]], hidden, inter, gs_dn) @ (g[:inter] / (1 + torch.exp(-g[:inter])) * g[inter:])
    out = [c for c in range(combos) if c not in live]
    assert len(out) >= 3 and torch.equal(eo[out], torch.full((len(out), hidden), 7.0, device="cuda"))
    err = (eo.double() - want)[live].norm(dim=1) / want[live].norm(dim=1)
    assert err.max().item() <= 2e-6  # f32 throughout, as above
    assert device_status() == 0


@pytest.mark.parametrize("run", [8, 64, 65, 200])
def test_groups_of_long_runs(run):
    """An expert with up to 64 rows and with more beside others and rows without an expert (placed by two ways of the grouping): every row is that of a step with
    few rows, to f32 sums of another order."""
    hidden, inter, experts = 256, 256, 5
    rng = np.random.default_rng(run)
    gu = [torch.from_numpy(synth.nvfp4_matrix(2 * inter, hidden, rng)).cuda() for _ in range(experts)]
    dn = [torch.from_numpy(synth.nvfp4_matrix(hidden, inter, rng)).cuda() for _ in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 2.0 ** -4, 0.5, gate_up=gu, down=dn, device="cuda")
    ids = rng.permutation(np.concatenate([np.full(run, 3), np.full(70, -1), np.repeat([0, 1, 4], [1, 9, 17])])).astype(np.int32)
    n = len(ids)
    x = torch.from_numpy(rng.standard_normal((n, hidden)).astype(np.float32)).cuda()
    idd, eo = torch.from_numpy(ids).cuda(), torch.full((n, hidden), 7.0, device="cuda")
    moe.GpuMoePlan(hidden, inter, experts, 1, n).experts_only(w, idd, x, eo=eo)
    few, want = moe.GpuMoePlan(hidden, inter, experts, 1, 8), torch.full((n, hidden), 7.0, device="cuda")
    for c in range(0, n, 8):
        few.experts_only(w, idd[c:c + 8], x[c:c + 8], eo=want[c:c + 8])
    assert torch.equal(eo[idd < 0], want[idd < 0])
    assert ((eo - want).norm(dim=1) <= 4e-6 * want.norm(dim=1)).all()  # 2e-6 of either, as above
    assert device_status() == 0


@pytest.mark.parametrize("hidden,inter,tokens,experts", [(256, 256, 50, 2), (512, 256, 100, 3), (768, 1280, 49, 40)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_odd_scales_and_rows_that_are_not_finite(hidden, inter, tokens, experts, dtype):
    """Scale bytes 0x7F and 0xFF, and an infinity and a NaN among the rows of a group: every other row of it is what 64 bits give."""
    rng = np.random.default_rng(hidden + inter)

    def matrix(rows, k):
        m = torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()
        s = m.view(-1, 36)[:, :4]
        s[:] = torch.from_numpy(rng.integers(0x70, 0x7F, tuple(s.shape)).astype(np.uint8)).cuda()  # (all of a size: no sums that cancel)
        pick = torch.from_numpy(rng.integers(0, 50, tuple(s.shape))).cuda()
        s[pick == 0], s[pick == 1] = 0x7F, 0xFF
        return m

    gu, dn = [matrix(2 * inter, hidden) for _ in range(experts)], [matrix(hidden, inter) for _ in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 2.0 ** -13, 2.0 ** -10, gate_up=gu, down=dn, device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, 1, tokens)
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda().to(dtype)
    x[3, 7], x[5, 100] = float("inf"), float("nan")
    ids = torch.from_numpy(rng.integers(0, experts, tokens).astype(np.int32)).cuda()
    eo = torch.empty((tokens, hidden), device="cuda")
    plan.experts_only(w, ids, x, eo=eo)
    assert not eo[5].isfinite().any() and not eo[3].isfinite().all()

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m, torch.tensor([gs], device="cuda"), rows, k), rule=True).double().view(rows, k)

    for c in range(tokens):
        if c in (3, 5):
            continue
        g = deq(gu[ids[c]], 2 * inter, hidden, 2.0 ** -13) @ x[c].double()
        want = deq(dn[ids[c]], hidden, inter, 2.0 ** -10) @ (g[:inter] / (1 + torch.exp(-g[:inter])) * g[inter:])
        assert (eo[c].double() - want).norm() <= 2e-6 * want.norm(), c  # f32 throughout, as above
    assert device_status() == 0


@pytest.mark.parametrize("hidden,inter,rows", [(256, 256, 49), (768, 512, 130), (2048, 256, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_digits_made_once_are_those_made_in_each_tile(hidden, inter, rows, dtype):
    """A plan holds the digits of as many rows as it has tokens; a step over more (one for each pick) makes them in each tile. Same bits, with values that have no digits among them."""
    rng = np.random.default_rng(rows)

    def matrix(n, k):
        return torch.from_numpy(synth.nvfp4_matrix(n, k, rng)).cuda()

    gu, dn = [matrix(2 * inter, hidden) for _ in range(5)], [matrix(hidden, inter) for _ in range(5)]
    w = moe.GpuMoeWeights(hidden, inter, 5, 0.03, 0.7, gate_up=gu, down=dn, device="cuda")
    x = torch.from_numpy((rng.standard_normal((rows, hidden)) * np.where(rng.random((rows, hidden)) < 0.01, 1e4, 1.0)).astype(np.float32)).cuda().to(dtype)
    x[3, 7] = float("inf")
    ids = torch.from_numpy(rng.integers(0, 5, rows).astype(np.int32)).cuda()
    out = []
    for plan in (moe.GpuMoePlan(hidden, inter, 5, 1, rows), moe.GpuMoePlan(hidden, inter, 5, 5, -(-rows // 5))):
        eo = torch.zeros((rows, hidden), device="cuda")
        plan.experts_only(w, ids, x, eo=eo)
        out.append(eo.view(torch.int32).clone())
    assert torch.equal(*out)
    assert device_status() == 0


def _records(plan, rows, hidden, dtype):
    """A plan's records of `rows` rows, as a view of its memory."""
    at, size = C.c_void_p(), C.c_size_t()
    check(lib().cn_moe_nvfp4_plan_digits(plan.handle, C.byref(at), C.byref(size)))
    each = hidden // 256 * (1440 if dtype == torch.float32 else 1056)
    assert rows * each <= size.value

    class View:
        __cuda_array_interface__ = {"shape": (rows, each), "typestr": "|u1", "data": (at.value, False), "version": 3}
    return torch.as_tensor(View(), device="cuda")


@pytest.mark.parametrize("hidden,rows,topk", [(256, 49, 1), (768, 5000, 1), (2048, 3000, 1), (4096, 800, 9), (2560, 600, 17)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_that_no_resident_expert_reads_get_no_digits(hidden, rows, topk, dtype):
    """A rank of an expert-parallel group: ids of -1 (inbox slots that nobody filled), ids beyond the experts, experts that live elsewhere. Rows with a combo of this rank are in the plan's
    store, the others' places beyond a chunk for every warp are as they were; one, two and more rounds of the warps, picks up to eight and beyond. The results are those of a step without a
    store."""
    experts, held, inter = 24, 3, 256
    rng = np.random.default_rng(rows + topk)

    def matrix(n, k):
        return torch.from_numpy(synth.nvfp4_matrix(n, k, rng)).cuda()

    gu, dn = [matrix(2 * inter, hidden) for _ in range(held)], [matrix(hidden, inter) for _ in range(held)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 0.03, 0.7, gate_up=gu + [None] * (experts - held), down=dn + [None] * (experts - held), device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, topk, rows)
    x = torch.from_numpy(rng.standard_normal((rows, hidden)).astype(np.float32)).cuda().to(dtype)
    ids = torch.from_numpy(rng.integers(-6, experts + 4, (rows, topk)).astype(np.int32)).cuda()
    store = _records(plan, rows, hidden, dtype)
    store.fill_(0xA5)
    eo = plan.experts_only(w, ids, x, eo=torch.zeros((rows * topk, hidden), device="cuda"), x_div=topk)
    read = ((ids >= 0) & (ids < held)).any(dim=1)
    written = (store != 0xA5).view(rows * hidden // 256, -1).any(dim=1)
    read = read[:, None].expand(-1, hidden // 256).reshape(-1)
    warps = min(147, -(-read.numel() // 32)) * 32
    assert written[:warps].all() and torch.equal(written[warps:], read[warps:])
    assert read.numel() <= 4704 or (read[4704:].any() and not read[4704:].all())
    few = moe.GpuMoePlan(hidden, inter, experts, rows * topk, 1)  # (a store of one row)
    again = few.experts_only(w, ids, x, eo=torch.zeros_like(eo), x_div=topk)
    assert torch.equal(eo.view(torch.int32), again.view(torch.int32))
    assert device_status() == 0


@pytest.mark.parametrize("size", [1e3, 1e4, 1e7])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_small_values_of_grouped_rows_beside_large_ones(size, dtype):
    """One value in sixteen of a row is large and meets zero weights: gate and up are what the small ones give."""
    hidden, inter, experts, tokens = 512, 512, 3, 60
    rng = np.random.default_rng(int(size))

    def matrix(rows, k):
        m = torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()
        if rows == 2 * inter:
            m.view(-1, 36)[:, 4::8] &= 0xF0  # the low half of a code byte: columns 0, 16, ..
        return m

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m, torch.tensor([gs], device="cuda"), rows, k), rule=True).double().view(rows, k)

    gu, dn = [matrix(2 * inter, hidden) for _ in range(experts)], [matrix(hidden, inter) for _ in range(experts)]
    w = moe.GpuMoeWeights(hidden, inter, experts, 2.0 ** -3, 2.0 ** -3, gate_up=gu, down=dn, device="cuda")
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda()
    x[:, ::16] *= size
    for m in gu:
        assert not deq(m, 2 * inter, hidden, 1.0)[:, ::16].any()
    x = x.to(dtype)
    ids = torch.from_numpy(rng.integers(0, experts, tokens).astype(np.int32)).cuda()
    eo = torch.empty((tokens, hidden), device="cuda")
    moe.GpuMoePlan(hidden, inter, experts, 1, tokens).experts_only(w, ids, x, eo=eo)
    for c in range(tokens):
        g = deq(gu[ids[c]], 2 * inter, hidden, 2.0 ** -3) @ x[c].double()
        want = deq(dn[ids[c]], hidden, inter, 2.0 ** -3) @ (g[:inter] / (1 + torch.exp(-g[:inter])) * g[inter:])
        # f32 throughout, as above; bf16 rows: digits of a block that is not multiplied out end at 2^-22 of its largest value, which is 2^8 of the third largest at most
        assert (eo[c].double() - want).norm() <= (2e-6 if dtype == torch.float32 else 2.0 ** -15) * want.norm(), c
    assert device_status() == 0
