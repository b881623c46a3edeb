"""Steps of fewer than 48 combos: gate / up of the routed and the shared expert in one launch, down projections with the combine in the next.
More units than warps (long k, many picks), k that ends in half a unit, shared experts wider and narrower than the routed ones, ids outside the
tables and experts that are not resident, a gate on the shared expert, f32 results of bf16 rows."""
import numpy as np
import pytest
import torch

from crownest_b200 import CrownestError, device_status, moe, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,topk,tokens,shared", [(256, 256, 1, 1, 0), (512, 768, 11, 4, 256), (256, 512, 1, 47, 1024), (1024, 2048, 8, 5, 2048),
                                                           (768, 1280, 6, 7, 512), (256, 256, 40, 1, 256),
                                                           # long k below 16 combos; 44 combos on both sides of the units that two launches take
                                                           (1024, 2048, 8, 1, 2048), (512, 2048, 4, 11, 1024), (768, 2048, 4, 11, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, "partial"])
def test_small_steps_against_64_bits(hidden, inter, topk, tokens, shared, dtype):
    rng = np.random.default_rng(hidden + inter + tokens)
    experts = 44
    partial, dtype = dtype == "partial", torch.bfloat16 if dtype == "partial" else dtype

    def matrix(rows, k):
        return torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()

    gone = {3, 40}
    gu = [None if e in gone else matrix(2 * inter, hidden) for e in range(experts)]
    dn = [None if e in gone else matrix(hidden, inter) for e in range(experts)]
    sh = [matrix(shared, hidden), matrix(shared, hidden), matrix(hidden, shared)] if shared else None
    gs_gu, gs_dn = 0.03, 0.7
    w = moe.GpuMoeWeights(hidden, inter, experts, gs_gu, gs_dn, gate_up=gu, down=dn, shared=sh, shared_gs=[0.03, 0.02, 0.6], device="cuda")
    plan = moe.GpuMoePlan(hidden, inter, experts, topk, tokens, shared_inter=shared)
    x = torch.from_numpy(rng.standard_normal((tokens, hidden)).astype(np.float32)).cuda().to(dtype)
    ids = np.stack([rng.permutation(experts)[:topk] for _ in range(tokens)]).astype(np.int32)
    if topk > 2:
        ids[0, :3] = [-1, experts, 3]
    wts = torch.from_numpy(rng.uniform(0.1, 1.0, (tokens, topk)).astype(np.float32)).cuda()
    sgate = torch.from_numpy(rng.standard_normal(tokens).astype(np.float32)).cuda() if shared else None
    dev = torch.from_numpy(ids).cuda()
    y = plan.experts_run(w, dev, wts, x, sgate=sgate, partial=partial, limit=6.0)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        out = torch.empty_like(y)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            plan.experts_run(w, dev, wts, x, out, sgate=sgate, partial=partial, limit=6.0)
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, y)

    def deq(m, rows, k, gs):
        return ops.dequant(ops.Fp4(m.view(-1), torch.tensor([gs], dtype=torch.float32, device="cuda"), rows, k)).double().view(rows, k)

    def ffn(g, u, d, xs):
        a, b = (xs @ g.t()).clamp(max=6.0), (xs @ u.t()).clamp(-6.0, 6.0)
        return (a / (1 + torch.exp(-a)) * b) @ d.t()

    x64, want = x.double(), torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for t in range(tokens):
        for j in range(topk):
            e = int(ids[t, j])
            if 0 <= e < experts and e not in gone:
                full = deq(gu[e], 2 * inter, hidden, gs_gu)
                want[t] += wts[t, j].double() * ffn(full[:inter], full[inter:], deq(dn[e], hidden, inter, gs_dn), x64[t:t + 1])[0]
    if shared:
        s = ffn(deq(sh[0], shared, hidden, 0.03), deq(sh[1], shared, hidden, 0.02), deq(sh[2], hidden, shared, 0.6), x64)
        want += s / (1 + torch.exp(-sgate.double()))[:, None]
    # f32 throughout: two long sums of 1.2e-7 each, some dozens of f32 roundings; a bf16 result adds its own rounding of at most 2^-8 of a value
    rms = want.pow(2).mean(dim=1, keepdim=True).sqrt()
    assert ((y.double() - want).abs() <= (2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0) * want.abs() + 1e-5 * rms).all()
    assert (y.double() - want).norm() <= (2e-6 if y.dtype == torch.float32 else 2.0 ** -8) * want.norm()
    assert device_status() == 0


@pytest.mark.parametrize("tokens", [1, 64])
def test_a_shared_expert_that_the_plan_has_no_room_for_is_refused(tokens):
    """Steps of both sizes: a plan made without a shared expert, and a shared expert without its scales or one of its matrices."""
    hidden, inter, experts, topk = 256, 256, 8, 4
    rng = np.random.default_rng(tokens)

    def matrix(rows, k):
        return torch.from_numpy(synth.nvfp4_matrix(rows, k, rng)).cuda()

    w = moe.GpuMoeWeights(hidden, inter, experts, 1.0, 1.0, gate_up=[matrix(2 * inter, hidden) for _ in range(experts)],
                          down=[matrix(hidden, inter) for _ in range(experts)], shared=[matrix(inter, hidden), matrix(inter, hidden), matrix(hidden, inter)],
                          shared_gs=[1.0, 1.0, 1.0], device="cuda")
    x = torch.zeros((tokens, hidden), device="cuda")
    ids = torch.arange(topk, device="cuda", dtype=torch.int32).repeat(tokens, 1)
    wts = torch.ones((tokens, topk), device="cuda")
    eo = torch.zeros((tokens * topk, hidden), device="cuda")
    bare = moe.GpuMoePlan(hidden, inter, experts, topk, tokens)
    for call in (lambda p: p.experts_run(w, ids, wts, x), lambda p: p.shared_begin(w, x), lambda p: p.finish(w, ids, wts, x, eo)):
        with pytest.raises(CrownestError, match="without a shared expert"):
            call(bare)
    whole = moe.GpuMoePlan(hidden, inter, experts, topk, tokens, shared_inter=inter)
    matrices, scales = w.shared, w.shared_gs
    for w.shared, w.shared_gs in ((matrices, None), (matrices[:2] + [None], scales), ([matrices[0], None, matrices[2]], scales)):
        for call in (lambda p: p.experts_run(w, ids, wts, x), lambda p: p.shared_begin(w, x), lambda p: p.finish(w, ids, wts, x, eo)):
            with pytest.raises(CrownestError, match="null matrix or scales"):
                call(whole)
    w.shared, w.shared_gs = matrices, scales
    assert not whole.experts_run(w, ids, wts, x).any()
    assert device_status() == 0
