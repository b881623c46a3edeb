"""Parity of the CUDA MUL1 (EXL3 trellis) path with the CPU checker: bit-exact decoded weights,
GEMV / FFN / MoE outputs within rel L2 <= 1e-3 of the exact-order f32 CPU reference."""
import hashlib
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle
from conftest import GOLDEN
from crownest_b200 import moe, mul1, ops, synth
from oracle import testkit as tk
from test_gpu_nvfp4_gemv import check_close, from_dev_bf16, to_dev_bf16

dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("K,k,n", [(3.0, 256, 128), (2.0, 384, 256), (3.5, 256, 128), (4.0, 128, 128), (8.0, 64, 64), (1.5, 64, 32)])
def test_decoded_weights_are_bit_exact(K, k, n):
    rng = np.random.default_rng(int(K * 10))
    tr = rng.integers(0, 65536, size=oracle.mul1_trellis_bytes(k, n, K) // 2, dtype=np.uint16)
    got = mul1.reconstruct(dev(tr.view(np.int16)), k, n, K).cpu().numpy().view(np.uint16)
    assert np.array_equal(got, oracle.mul1_reconstruct(tr, k, n, K))


def test_quantizer_record_decodes_to_the_exllamav3_digest():
    # the reference's golden: sha256 of exllamav3's own reconstruct output (converter/tests/fixtures)
    for line in open(os.path.join(GOLDEN, "exl3-mul1-decode.tsv")):
        if not line.startswith("q-k3\t"):
            continue
        f = line.rstrip("\n").split("\t")
        hidden, inter = int(f[3]), int(f[4])
        raw = np.fromfile(os.path.join(GOLDEN, f[1]), np.uint8)
        tb = oracle.mul1_trellis_bytes(hidden, inter, 3.0)
        for i, (k, n) in enumerate([(hidden, inter), (hidden, inter), (inter, hidden)]):
            tr = raw[i * tb:(i + 1) * tb].view(np.int16)
            got = mul1.reconstruct(dev(tr), k, n, 3.0).cpu().numpy()
            assert hashlib.sha256(got.tobytes()).hexdigest() == f[5 + i]


def expert_parts(rec, hidden, inter, K):
    tb = oracle.mul1_trellis_bytes(hidden, inter, K)
    at, out = 3 * tb, []
    for nbytes in (2 * hidden, 2 * inter, 2 * hidden, 2 * inter, 2 * inter, 2 * hidden):
        out.append(rec[at:at + nbytes].view(np.uint16))
        at += nbytes
    return tb, out


@pytest.mark.parametrize("K,hidden,inter", [(3.0, 512, 256), (3.0, 4096, 1536), (2.0, 256, 384), (3.5, 256, 128), (4.0, 128, 256)])
@pytest.mark.parametrize("t", [1, 3])
def test_gemv_matches_the_cpu_reference(K, hidden, inter, t):
    rec = tk.mul1_record(7, hidden, inter, K)
    tb, (gs, gv, us, uv, ds, dv) = expert_parts(rec, hidden, inter, K)
    rng = np.random.default_rng(2)
    slots = 2
    d_rec = [dev(rec), dev(rec.copy())]
    ptrs = torch.tensor([r.data_ptr() for r in d_rec], dtype=torch.int64, device="cuda")
    plan = mul1.Mul1Plan(hidden, inter, K, slots=slots, tokens=t)
    for which, (k, n, tro, su, sv) in enumerate([(hidden, inter, 0, gs, gv), (hidden, inter, tb, us, uv), (inter, hidden, 2 * tb, ds, dv)]):
        x = rng.uniform(-2, 2, size=(slots, t, k)).astype(np.float32)
        y = plan.run_slots(which, ptrs, dev(x)).cpu().numpy()
        for s in range(slots):
            ref = oracle.mul1_gemv(rec[tro:tro + tb], su, sv, k, n, K, x[s], threads=8)
            check_close(y[s], ref, f"mul1 gemv K={K} which={which} slot {s}", bf16_out=False)
    plan.free()


@pytest.mark.parametrize("K", [1.0, 1.5, 2.0, 2.5, 3.0, 3.5, 4.0, 5.0, 6.0, 7.0, 8.0])
@pytest.mark.parametrize("t", [1, 2, 4, 7])
@pytest.mark.parametrize("slots", [1, 520])
def test_every_bitrate_at_every_row_count(K, t, slots):
    """Rates whose states come out of one window of the bit stream, of two from the same words or from words of their own, and of three, each with the lane whose window goes round the tile's end; rows
    transformed inside the GEMV (few slots) and staged by a launch of their own (many; the rows of the last slots are looked at). The other records are null."""
    hidden, inter = 768, 512
    rec = tk.mul1_record(int(2 * K) + t, hidden, inter, K)
    tb, (gs, gv, us, uv, ds, dv) = expert_parts(rec, hidden, inter, K)
    d_rec = dev(rec)
    ptrs = torch.zeros(slots, dtype=torch.int64, device="cuda")
    ptrs[-1] = d_rec.data_ptr()
    plan = mul1.Mul1Plan(hidden, inter, K, slots=slots, tokens=t)
    gen = torch.Generator(device="cuda").manual_seed(3)
    for which, (k, n, tro, su, sv) in enumerate([(hidden, inter, 0, gs, gv), (hidden, inter, tb, us, uv), (inter, hidden, 2 * tb, ds, dv)]):
        x = torch.rand((slots, t, k), device="cuda", generator=gen) * 4 - 2
        y = plan.run_slots(which, ptrs, x)[-1].cpu().numpy().astype(np.float64)
        ref = oracle.mul1_gemv(rec[tro:tro + tb], su, sv, k, n, K, x[-1].cpu().numpy(), threads=8).astype(np.float64)
        # two transforms of seven f32 additions and a sum of k products of 22-bit activations, against the same in another order: some 30 roundings of 6e-8
        assert np.linalg.norm(y - ref) <= 4e-6 * np.linalg.norm(ref)
    plan.free()


def test_null_slots_are_skipped_and_rows_are_batch_invariant():
    hidden, inter, K = 512, 256, 3.0
    rec = dev(tk.mul1_record(3, hidden, inter, K))
    plan = mul1.Mul1Plan(hidden, inter, K, slots=3, tokens=4)
    x = torch.randn((3, 4, hidden), device="cuda")
    ptrs = torch.tensor([rec.data_ptr(), 0, rec.data_ptr()], dtype=torch.int64, device="cuda")
    y = torch.full((3, 4, inter), float("nan"), device="cuda")
    plan.run_slots(0, ptrs, x, y)
    assert torch.isnan(y[1]).all() and torch.isfinite(y[0]).all() and torch.isfinite(y[2]).all()
    # one row at a time gives the same bits as four rows at once
    one = mul1.Mul1Plan(hidden, inter, K, slots=1, tokens=1)
    for t in range(4):
        y1 = one.run_slots(0, ptrs[:1], x[0, t:t + 1].contiguous())
        assert torch.equal(y1.view(torch.int32).reshape(-1), y[0, t].view(torch.int32))
    plan.free(), one.free()


@pytest.mark.parametrize("limit", [0.0, 10.0])
def test_expert_ffn_matches_the_cpu_reference(limit):
    hidden, inter, K = 1024, 512, 3.0
    recs = [tk.mul1_record(20 + i, hidden, inter, K) for i in range(3)]
    d = [dev(r) for r in recs]
    ptrs = torch.tensor([r.data_ptr() for r in d], dtype=torch.int64, device="cuda")
    rng = np.random.default_rng(4)
    x = (rng.standard_normal((3, 2, hidden)) * 0.3).astype(np.float32)
    plan = mul1.Mul1Plan(hidden, inter, K, slots=3, tokens=2)
    y = plan.ffn(ptrs, dev(x), limit=limit).cpu().numpy()
    for s in range(3):
        ref = oracle.mul1_expert_ffn(recs[s], hidden, inter, K, x[s], limit=limit, threads=8)
        check_close(y[s], ref, f"mul1 ffn slot {s}", bf16_out=False)
    plan.free()


@pytest.mark.parametrize("tokens", [1, 4, 16])
def test_moe_step_over_mul1_experts_matches_the_cpu_reference(tokens):
    # the benchmark's EXL3 shape: hidden 4096 <-> inter 1536, 64 experts, top-4, K = 3. Only the experts the routing picks
    # get a record (4 / ~15 / ~41 of them); the other table entries are null and nothing may touch them
    hidden, inter, K, experts, topk = 4096, 1536, 3.0, 64, 4
    rng = np.random.default_rng(40 + tokens)
    xb, xf = synth.activations(tokens, hidden, rng)
    xf = (xf * np.float32(0.25)).astype(np.float32)
    xb = synth.bf16_bits(xf)
    xf = synth.bf16_to_f32(xb)
    logits = rng.standard_normal((tokens, experts)).astype(np.float32)
    ids, wts = moe.route_softmax_topk(dev(logits), topk)
    rids, rw = oracle.route_softmax_topk(logits, topk)
    assert np.array_equal(ids.cpu().numpy(), rids)
    picked = sorted(set(int(e) for e in rids.reshape(-1)))
    recs = {e: tk.mul1_record(0x1640 + 9 * e, hidden, inter, K) for e in picked}
    d = {e: dev(r) for e, r in recs.items()}
    table = torch.tensor([d[e].data_ptr() if e in d else 0 for e in range(experts)], dtype=torch.int64, device="cuda")
    plan = mul1.Mul1Plan(hidden, inter, K, slots=tokens * topk, tokens=1)
    y = plan.moe(table, ids, wts, to_dev_bf16(xb), limit=10.0)
    ye = np.zeros((tokens * topk, hidden), np.float32)
    for c in range(tokens * topk):
        ye[c] = oracle.mul1_expert_ffn(recs[rids.reshape(-1)[c]], hidden, inter, K, xf[c // topk: c // topk + 1], limit=10.0, threads=8)[0]
    ref = oracle.moe_combine(ye, rw, None)
    # f32 in / out: the 1e-3 contract proper
    yf = plan.moe(table, ids, wts, dev(xf), limit=10.0)
    check_close(yf.cpu().numpy(), ref, f"mul1 moe f32 tokens={tokens}", bf16_out=False)
    # bf16 in / out (ulp taken no lower than rms / 64: the combine cancels)
    check_close(from_dev_bf16(y), ref, f"mul1 moe tokens={tokens}", ulp_floor=1.0 / 64)
    plan.free()


@pytest.mark.parametrize("tokens,experts,topk", [(32, 6, 3), (40, 5, 4), (10, 6, 3)])
def test_moe_step_with_bundled_rows_matches_the_cpu_reference(tokens, experts, topk):
    """At least two combo slots per expert: the combos are sorted by expert and run as groups of up to four rows that share
    one decode of the expert (one, two, three and four-row groups and unused row slots all occur)."""
    hidden, inter, K = 1024, 512, 3.0
    rng = np.random.default_rng(7 + tokens)
    recs = [tk.mul1_record(0x2000 + 5 * e, hidden, inter, K) for e in range(experts)]
    d = [dev(r) for r in recs]
    table = torch.tensor([r.data_ptr() for r in d], dtype=torch.int64, device="cuda")
    x = (rng.standard_normal((tokens, hidden)) * 0.25).astype(np.float32)
    logits = rng.standard_normal((tokens, experts)).astype(np.float32)
    ids, wts = moe.route_softmax_topk(dev(logits), topk)
    rids, rw = oracle.route_softmax_topk(logits, topk)
    assert np.array_equal(ids.cpu().numpy(), rids)
    plan = mul1.Mul1Plan(hidden, inter, K, slots=tokens * topk, tokens=1)
    y = plan.moe(table, ids, wts, dev(x), limit=10.0)
    ye = np.zeros((tokens * topk, hidden), np.float32)
    for c in range(tokens * topk):
        ye[c] = oracle.mul1_expert_ffn(recs[rids.reshape(-1)[c]], hidden, inter, K, x[c // topk: c // topk + 1], limit=10.0, threads=8)[0]
    ref = oracle.moe_combine(ye, rw, None)
    check_close(y.cpu().numpy(), ref, f"mul1 moe bundled tokens={tokens}", bf16_out=False)
    y2 = plan.moe(table, ids, wts, dev(x), limit=10.0)
    assert torch.equal(y.view(torch.int32), y2.view(torch.int32))
    plan.free()


def records(n, hidden, inter, K, seed):
    """Codes uniform, scales small with random signs; in one allocation, as addresses."""
    rng = np.random.default_rng(seed)
    size = mul1.record_bytes(hidden, inter, K)
    rec = rng.integers(0, 256, (n, size), dtype=np.uint8)
    at = int(3 * (hidden // 16) * (inter // 16) * 32 * K)
    v = (np.abs(rng.standard_normal((n, 3 * (hidden + inter)))) * 0.02 + 1e-3) * rng.choice([-1.0, 1.0], (n, 3 * (hidden + inter)))
    rec[:, at:at + 6 * (hidden + inter)] = v.astype(np.float16).view(np.uint8)
    rec[:, at + 6 * (hidden + inter):] = 0
    d = dev(rec)
    return d, torch.tensor([r.data_ptr() for r in d.unbind(0)], dtype=torch.int64, device="cuda")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("K", [3.0, 3.5])
@pytest.mark.parametrize("t,x_div", [(1, 1), (3, 1), (8, 1), (8, 4)])
def test_rows_transformed_in_a_launch_of_their_own_have_the_same_bits(dtype, K, t, x_div):
    """Many slots take a launch for the input transform, few have it inside the GEMV: slot by slot the same results, also off 16 bytes and beside null records."""
    hidden, inter, slots = 512, 384, 12288 // (4 * 3 * t) // 4 * 4 + 8
    rec, ptrs = records(5, hidden, inter, K, t)
    ptrs = ptrs.repeat(-(-slots // 5))[:slots].clone()
    ptrs[3::7] = 0
    gen = torch.Generator(device="cuda").manual_seed(t)
    whole, one = mul1.Mul1Plan(hidden, inter, K, slots=slots, tokens=t), mul1.Mul1Plan(hidden, inter, K, slots=4, tokens=t)
    for which, k in ((0, hidden), (2, inter)):
        n = slots // x_div * t * k
        x = (torch.randn(n + 1, device="cuda", generator=gen) * 0.25).to(dtype)[1:].view(slots // x_div, t, k)  # off 16 bytes
        y = whole.run_slots(which, ptrs, x, x_div=x_div)
        for s in list(range(0, 16, 4)) + [slots - 4]:
            assert torch.equal(one.run_slots(which, ptrs[s:s + 4], x[s // x_div:(s + 4) // x_div], x_div=x_div), y[s:s + 4]), (which, s)
    x = (torch.randn((slots // x_div, t, hidden), device="cuda", generator=gen) * 0.25).to(dtype)
    y = whole.ffn(ptrs, x, x_div=x_div, limit=5.0)
    assert y.isfinite().all() and y[0].any() and not y[3].any()
    for s in list(range(0, 16, 4)) + [slots - 4]:
        assert torch.equal(one.ffn(ptrs[s:s + 4], x[s // x_div:(s + 4) // x_div], x_div=x_div, limit=5.0), y[s:s + 4]), s


@pytest.mark.parametrize("tokens,experts", [(150, 1500), (150, 40), (40, 40)])
def test_routed_steps_of_many_combos_match_one_token_steps(tokens, experts):
    """Combos that keep a slot each (few of them for the experts there are) and combos in groups of four and eight rows, with their rows transformed in a
    launch of their own: ids outside the table, experts that are not resident; against steps of one token, which have the transform inside the GEMV."""
    hidden, inter, topk, K = 512, 384, 4, 3.0
    rec, ptrs = records(8, hidden, inter, K, 3)
    table = ptrs.repeat(-(-experts // 8))[:experts].clone()
    table[5::11] = 0
    rng = np.random.default_rng(tokens + experts)
    ids = np.stack([rng.permutation(experts)[:topk] for _ in range(tokens)]).astype(np.int32)
    ids[::9, 1], ids[::13, 2] = -1, experts
    d_ids = dev(ids)
    wts = torch.from_numpy(rng.uniform(0.1, 1.0, (tokens, topk)).astype(np.float32)).cuda()
    x = torch.from_numpy((rng.standard_normal((tokens, hidden)) * 0.25).astype(np.float32)).cuda()
    whole, one = mul1.Mul1Plan(hidden, inter, K, slots=tokens * topk), mul1.Mul1Plan(hidden, inter, K, slots=topk)
    y = whole.moe(table, d_ids, wts, x, limit=5.0)
    assert y.isfinite().all()
    for i in range(0, tokens, 7):
        assert torch.equal(one.moe(table, d_ids[i:i + 1], wts[i:i + 1], x[i:i + 1], limit=5.0), y[i:i + 1]), i
