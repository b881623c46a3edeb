"""The CTA-pair GEMM (more than 128 rows) at the edges of its tiles: row counts around 256-row tiles (odd ones take the
one-row stores), token counts around the tile widths it chooses (one and two accumulators, 4 to 8 weight slots), k = 256,
every scale byte in the bf16 decode (subnormal scales ride as subnormal bf16)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle
from crownest_b200 import CrownestError, device_status, ops, synth
from test_gpu_nvfp4_gemv import check_close, from_dev_bf16, to_dev_bf16


@pytest.mark.parametrize("rows,k,m", [(256, 256, 129), (333, 256, 160), (255, 512, 193), (258, 768, 449), (1030, 1280, 225), (2, 2048, 513)])
def test_pair_gemm_matches_the_cpu_reference(rows, k, m):
    rng = np.random.default_rng(rows + m)
    w = synth.nvfp4_matrix(rows, k, rng).copy()
    if k == 256:  # every scale byte, bit 7 and 0x7F included
        w.reshape(-1, 36)[:, :4] = np.arange(rows * (k // 64) * 4, dtype=np.uint32).astype(np.uint8).reshape(-1, 4)
    xb, xf = synth.activations(m, k, rng)
    fw = ops.Fp4.from_host(w, rows, k, np.float32(0.37))
    ref = np.concatenate([oracle.nvfp4_gemv(w, rows, k, np.float32(0.37), xf[t:t + 8], threads=8, path=1) for t in range(0, m, 8)])
    # bf16 rows as they are; the ulp no lower than rms / 64 (f32 accumulation error of either side, as for the other GEMMs)
    check_close(from_dev_bf16(ops.launch_gemm(fw, to_dev_bf16(xb))), ref, f"pair gemm {rows}x{k} m={m}", ulp_floor=1.0 / 64)
    # f32 rows ride as f16 (exact for these bf16 values): the f32 accumulator itself
    yf = ops.launch_gemm(fw, torch.from_numpy(xf).cuda()).cpu().numpy()
    scale = np.sqrt(np.mean(ref.astype(np.float64) ** 2, axis=1, keepdims=True))
    assert np.max(np.abs(yf - ref) / scale) <= 1e-4
    assert device_status() == 0


@pytest.mark.parametrize("m", [129, 513])
def test_rows_of_any_magnitude(m):
    """bf16 rows are not scaled one by one on this path: rows near both ends of what a power of two per row brings into f16 (2^-112 to
    2^113) come out as well as the others, beside ordinary rows."""
    rows, k = 512, 2048
    rng = np.random.default_rng(m)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(1.0))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda()
    for i, scale in enumerate([1e-12, 1e-20, 1e-27, 1e-33, 1e12, 1e27, 1e33]):
        x[5 + 17 * i] *= scale
    x = x.to(torch.bfloat16)
    want = x.double() @ ops.dequant(w).double().view(rows, k).t()
    err = (ops.launch_gemm(w, x).double() - want).norm(dim=1) / want.norm(dim=1)
    # one rounding of the result to bf16 (2^-9 at most) beside f32 sums
    assert err.max().item() <= 2.0 ** -9 + 4e-6
    assert device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,k,at", [(2048, 2048, 4096), (4096, 2048, 1024), (1024, 2048, 7096)])
def test_results_in_the_place_of_the_activations(rows, k, at, dtype):
    """More tiles than CTA pairs, so that late tiles read activations after early ones have written; y starts on, before and inside x."""
    m = 4096
    rng = np.random.default_rng(rows)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(1.0))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(dtype)
    want = ops.launch_gemm(w, x)
    buf = torch.empty(2 * m * max(rows, k) + 8192, dtype=dtype, device="cuda")
    xs, ys = buf[4096:4096 + m * k].view(m, k), buf[at:at + m * rows].view(m, rows)
    xs.copy_(x)
    ops.launch_gemm(w, xs, ys)
    assert torch.equal(ys, want)
    assert device_status() == 0


@pytest.mark.parametrize("relaid", [False, True])
@pytest.mark.parametrize("rows,k,m", [(100, 256, 1), (256, 512, 33), (333, 4096, 9), (600, 4096, 64), (1030, 2048, 65), (5120, 1280, 128), (130, 8192, 129),
                                      (384, 5120, 300), (512, 1024, 513)])
def test_few_rows_split_k_and_relaid_weights(rows, k, m, relaid):
    """Rows at the edges of the f16 path (1, 128, 129 rows), of the split of K (512, 513 rows; one, a few and eight parts) and of the tiles; container
    bytes and stage images (an odd count of 128-row tiles leaves a CTA of the last pair without one)."""
    rng = np.random.default_rng(rows + m)
    w = synth.nvfp4_matrix(rows, k, rng).copy()
    w.reshape(-1, 36)[::7, 1] = 0x7F
    w.reshape(-1, 36)[::5, 2] |= 0x80
    fw = ops.Fp4.from_host(w, rows, k, np.float32(0.37))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda()
    x[m // 2] *= 1e-6
    x = x.to(torch.bfloat16)
    want = x.double() @ ops.dequant(fw, rule=True).double().view(rows, k).t()
    if relaid:
        packed = ops.Fp4Packed(fw)
        run = lambda xs, ys=None: ops.launch_gemm_fp4(packed, xs, ys)
    else:
        run = lambda xs, ys=None: ops.launch_gemm(fw, xs, ys)
    y = run(x)
    # one rounding of the result to bf16 (half a unit of 2^-7: at most 2^-8 of the value) beside f32 sums (1e-6 of the row's scale, see the other GEMM tests)
    rms = want.pow(2).mean(dim=1, keepdim=True).sqrt()
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * rms).all()
    # results over the activations, and in rows further apart than they are long
    buf = torch.zeros(2 * m * max(rows, k) + 64, dtype=torch.bfloat16, device="cuda")
    xs, ys = buf[:m * k].view(m, k), buf[16:16 + m * rows].view(m, rows)
    xs.copy_(x)
    assert torch.equal(run(xs, ys), y)
    wide = torch.zeros((m, rows + 6), dtype=torch.bfloat16, device="cuda")
    run(x, wide[:, :rows])
    assert torch.equal(wide[:, :rows], y) and not wide[:, rows:].any()
    assert device_status() == 0


@pytest.mark.parametrize("relaid", [False, True])
@pytest.mark.parametrize("rows,k,m", [(19200, 256, 33), (300, 768, 65), (520, 1280, 97), (18950, 1024, 128), (256, 2304, 32)])
def test_slots_of_a_whole_weight_stage(rows, k, m, relaid):
    """Up to 128 rows a stage of 256 values of k is one slot of each ring: fewer stages than slots, one more than the A slots, every width of the token tile (32 to 128), and more
    tiles than CTA pairs, whose second round finds the rings wherever the first one left them. Every output."""
    rng = np.random.default_rng(rows + m)
    fw = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(0.37))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    want = x.double() @ ops.dequant(fw, rule=True).double().view(rows, k).t()
    y = ops.launch_gemm_fp4(ops.Fp4Packed(fw), x) if relaid else ops.launch_gemm(fw, x)
    rms = want.pow(2).mean(dim=1, keepdim=True).sqrt()
    # as above: one rounding of the result to bf16 beside f32 sums
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * rms).all()
    assert device_status() == 0


@pytest.mark.parametrize("m", [1, 60, 128])
@pytest.mark.parametrize("form", ["container", "relaid", "f32"])
@pytest.mark.parametrize("rows", [384, 4000])
def test_rows_of_any_magnitude_as_f16(m, form, rows):
    """Rows that are brought into f16 by a power of two each: from subnormal bf16 to the largest finite values, with one part of k and several; an
    infinity or a NaN reaches the results of its own row and leaves the finite terms beside it alone."""
    k = 2048
    rng = np.random.default_rng(m + rows)
    data, unit = synth.nvfp4_matrix(rows, k, rng), np.clip(rng.standard_normal((m, k)), -3.0, 3.0)
    for gs, scales in ((2.0 ** 60, [3e-40, 1e-38, 1e-36, 2e-34, 7e-34, 1e-33, 1e-20, 1.0]), (2.0 ** -60, [1.1e38, 1e38, 2e34, 3e30, 1.0])):
        fw = ops.Fp4.from_host(data, rows, k, np.float32(gs))
        w = ops.Fp4Packed(fw) if form == "relaid" else fw
        x = torch.from_numpy(unit * np.array([scales[i % len(scales)] for i in range(m)])[:, None]).cuda().to(torch.float32)
        x = x if form == "f32" else x.to(torch.bfloat16)
        y = (ops.launch_gemm_fp4 if form == "relaid" else ops.launch_gemm)(w, x)
        want = x.double() @ ops.dequant(fw, rule=True).double().view(rows, k).t()
        err = (y.double() - want).norm(dim=1) / want.norm(dim=1)
        # bf16: one rounding of the result (2^-9 at most) beside f32 sums; f32 rows: one rounding of every value to f16 (2^-12 in the mean square at most),
        # the smallest of them to a subnormal f16 (3e-40 becomes 2^-4, which f16 holds in steps of 2^-24)
        assert err.max().item() <= (2.0 ** -11 if form == "f32" else 2.0 ** -9 + 4e-6)
    fw = ops.Fp4.from_host(data, rows, k, np.float32(1.0))
    w = ops.Fp4Packed(fw) if form == "relaid" else fw
    x = torch.from_numpy(np.abs(unit) * 1e10).cuda().to(torch.float32 if form == "f32" else torch.bfloat16)
    special = x.clone()
    special[0, 7], special[m - 1, 9] = float("inf"), float("inf") if m == 1 else float("nan")
    run = ops.launch_gemm_fp4 if form == "relaid" else ops.launch_gemm
    y, plain = run(w, special), run(w, x)
    col = ops.dequant(fw, rule=True).view(rows, k)
    hit = (torch.where(col[:, 7] != 0, col[:, 7].sign() * float("inf"), float("nan")) if m > 1 else
           torch.where((col[:, 7] != 0) & (col[:, 9] != 0) & (col[:, 7].sign() == col[:, 9].sign()), col[:, 7].sign() * float("inf"), float("nan")))
    assert torch.equal(y[0].float().nan_to_num(nan=-7.0), hit.to(y.dtype).float().nan_to_num(nan=-7.0))
    if m > 1:
        assert y[m - 1].isnan().all()
    if m > 2:
        assert torch.equal(y[1:m - 1], plain[1:m - 1])
    assert device_status() == 0


def rows_as_stored(k, m):
    """Bytes of the activations and their factors, without room for partial sums."""
    return m * k * 2 + (m * 4 + 255) // 256 * 256 + 256


@pytest.mark.parametrize("rows,k,m", [(600, 4096, 64), (1024, 10240, 200), (2048, 8192, 512), (600, 4096, 513), (17408, 512, 300), (40000, 512, 20)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_workspaces_of_every_accepted_size(rows, k, m, dtype):
    """No room for partial sums, room for two or three parts of k, what the matrix takes, what any matrix takes, and more than that: the last three
    give the same bits, all of them the product; below the first the call is refused."""
    rng = np.random.default_rng(rows + m)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(0.37))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(torch.bfloat16).to(dtype)
    want = x.double() @ ops.dequant(w, rule=True).double().view(rows, k).t()
    rms = want.pow(2).mean(dim=1, keepdim=True).sqrt()
    # bf16: one rounding of the result, at most 2^-8 of the value. The sum in tensor memory: each of the k / 16 steps may cut the running sum by 2^-23 of
    # itself, which no output's running sum takes beyond six times the row's scale.
    most = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + k / 16 * 2.0 ** -23 * 6 * rms
    least, own, whole = rows_as_stored(k, m), ops.gemm_workspace_bytes(k, m, rows), ops.gemm_workspace_bytes(k, m)
    assert least <= own <= whole
    ys = {}
    for n in (least, least + 4 * m * rows * 2, least + 4 * m * rows * 3 + 60, own, whole, whole + 4 * m * rows * 4):
        ws = torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda")
        y = ys[n] = ops.launch_gemm(w, x, workspace=ws)
        assert ((y.double() - want).abs() <= most).all()
    assert torch.equal(ys[own], ys[whole]) and torch.equal(ys[whole + 4 * m * rows * 4], ys[whole]) and torch.equal(ops.launch_gemm(w, x), ys[whole])
    with pytest.raises(CrownestError, match="needed"):
        ops.launch_gemm(w, x, workspace=torch.empty(least - 1, dtype=torch.uint8, device="cuda"))
    packed = ops.Fp4Packed(w)
    full = ops.launch_gemm_fp4(packed, x)
    if dtype == torch.bfloat16:
        for n in (least, least + 4 * m * rows * 2):
            y = ops.launch_gemm_fp4(packed, x, workspace=torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda"))
            assert ((y.double() - want).abs() <= most).all()
        assert ((full.double() - want).abs() <= most).all()
    else:  # five cascade levels: the bound of the block-scaled GEMM's own test
        assert ((full.double() - want).abs() <= 1e-4 * rms).all()
    assert device_status() == 0
