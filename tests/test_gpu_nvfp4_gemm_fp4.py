"""The block-scaled FP4 tensor-core GEMM (tcgen05 kind::mxf4nvf4, through the C ABI) and its activation cascade against the
CPU checker: cascade bytes bit-exact with the restatement of the reference's host twin; GEMM outputs within rel L2 <= 1e-3
and 2 bf16 ulp (taken no lower than rms / 64) of the f32-accumulated CPU reference of the exact activations."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle
from crownest_b200 import device_status, ops, synth
from test_gpu_nvfp4_gemv import check_close, from_dev_bf16, to_dev_bf16
from test_gpu_nvfp4_gemm import cpu_rows


@pytest.mark.parametrize("levels", [1, 3, 5])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_cascade_bytes_are_bit_exact(levels, dtype):
    rng = np.random.default_rng(levels)
    k = 640
    x = (rng.standard_normal((9, k)) * np.array([3.0, 0.4, 0.04, 0.004, 1e-4, 300.0, 0.0, 1.0, 1e-30])[:, None]).astype(np.float32)
    x[7, 5] = 1500.0
    if dtype == "bf16":
        xb = synth.bf16_bits(x)
        x = synth.bf16_to_f32(xb)
        got = ops.act_cascade(to_dev_bf16(xb), levels).cpu().numpy()
    else:
        got = ops.act_cascade(torch.from_numpy(x).cuda(), levels).cpu().numpy()
    for r in range(x.shape[0]):
        assert np.array_equal(got[r], oracle.act_cascade(x[r], levels)), f"row {r}"


@pytest.mark.parametrize("rows,k,m", [(128, 256, 32), (256, 512, 64), (200, 1024, 70), (384, 2048, 33), (640, 5120, 96), (1000, 768, 17)])
def test_fp4_gemm_matches_the_cpu_reference(rows, k, m):
    rng = np.random.default_rng(rows + k + m)
    w = synth.nvfp4_matrix(rows, k, rng)
    w.reshape(-1, 36)[::7, 1] = 0x7F  # the NaN code of the tensor core's scale format: must read as 448
    w.reshape(-1, 36)[::5, 2] |= 0x80  # bit 7 is ignored
    gs = np.float32(0.37)
    xb, xf = synth.activations(m, k, rng)
    xf[m // 2] *= np.float32(2.0 ** -20)
    xb = synth.bf16_bits(xf)
    xf = synth.bf16_to_f32(xb)
    fw = ops.Fp4Packed(ops.Fp4.from_host(w, rows, k, gs))
    y = ops.launch_gemm_fp4(fw, to_dev_bf16(xb))
    torch.cuda.synchronize()
    assert device_status() == 0
    ref = cpu_rows(w, rows, k, gs, xf)
    got = from_dev_bf16(y)
    for t in (0, m // 2, m - 1):
        check_close(got[t:t + 1], ref[t:t + 1], f"fp4 gemm {rows}x{k} m={m} row {t}", ulp_floor=1.0 / 64)
    check_close(got, ref, f"fp4 gemm {rows}x{k} m={m}", ulp_floor=1.0 / 64)
    yf = ops.launch_gemm_fp4(fw, torch.from_numpy(xf).cuda()).cpu().numpy()
    scale = np.sqrt(np.mean(ref.astype(np.float64) ** 2, axis=1, keepdims=True))
    assert np.max(np.abs(yf - ref) / scale) <= 1e-4
    y2 = ops.launch_gemm_fp4(fw, to_dev_bf16(xb))
    assert torch.equal(y.view(torch.int16), y2.view(torch.int16))


@pytest.mark.parametrize("rows,k", [(17408, 5120), (5120, 17408)])
@pytest.mark.parametrize("m", [64, 512])
def test_fp4_gemm_on_the_batched_benchmark_matrices(rows, k, m):
    rng = np.random.default_rng(rows + m + 1)
    w = synth.nvfp4_matrix(rows, k, rng)
    gs = np.float32(0.21)
    xb, xf = synth.activations(m, k, rng)
    fw = ops.Fp4Packed(ops.Fp4.from_host(w, rows, k, gs))
    y = ops.launch_gemm_fp4(fw, to_dev_bf16(xb))
    pick = np.unique(np.concatenate([[0, 1, 127, 128, rows - 129, rows - 1], rng.integers(0, rows, size=256)]))
    rb = k // 64 * 36
    sub = np.ascontiguousarray(w.reshape(rows, rb)[pick]).reshape(-1)
    ref = cpu_rows(sub, len(pick), k, gs, xf)
    check_close(from_dev_bf16(y)[:, pick], ref, f"fp4 gemm {rows}x{k} m={m} (sample)", ulp_floor=1.0 / 64)
    assert device_status() == 0


def test_more_rows_than_a_grid_has_in_y():
    rows, k, m = 128, 256, 65600
    rng = np.random.default_rng(8)
    w = synth.nvfp4_matrix(rows, k, rng)
    xb, xf = synth.activations(64, k, rng)
    fw = ops.Fp4Packed(ops.Fp4.from_host(w, rows, k, np.float32(0.37)))
    y = ops.launch_gemm_fp4(fw, to_dev_bf16(xb).repeat(m // 64, 1))
    assert torch.equal(y.view(torch.int16), y[:64].view(torch.int16).repeat(m // 64, 1))
    check_close(from_dev_bf16(y[:64]), cpu_rows(w, rows, k, np.float32(0.37), xf), "first rows", ulp_floor=1.0 / 64)
    assert device_status() == 0


def f32_close(got, x, w, what):
    """f32 rows through five cascade levels: 1.1e-5 of a row in the 2-norm on N(0,1) values of full mantissa (5.5e-6 on bf16 ones), which the host twin of the
    cascade gives for k = 640 .. 17408. An output's scale is the row's norm times that of a mean weight row; twice the figure for the mean
    square, and seven of its standard deviations for the worst of some hundred thousand outputs."""
    x, w = x.double(), w.double()
    scale = x.norm(dim=1, keepdim=True) * w.pow(2).mean().sqrt()
    err = (got.double() - x @ w.t()) / scale
    assert err.pow(2).mean().sqrt() <= 2e-5 and err.abs().max() <= 7e-5, f"{what}: {err.pow(2).mean().sqrt():.1e} {err.abs().max():.1e}"


@pytest.mark.parametrize("rows,k", [(17408, 5120), (5120, 17408)])
@pytest.mark.parametrize("m", [64, 512])
def test_block_scaled_gemm_on_the_batched_benchmark_matrices(rows, k, m):
    """f32 rows, which bf16 values in f32 are not: every value has its full mantissa. One part of k and three."""
    rng = np.random.default_rng(rows + m + 2)
    w = synth.nvfp4_matrix(rows, k, rng)
    x = rng.standard_normal((m, k)).astype(np.float32)
    fw = ops.Fp4Packed(ops.Fp4.from_host(w, rows, k, np.float32(0.21)))
    y = ops.launch_gemm_fp4(fw, torch.from_numpy(x).cuda())
    pick = np.unique(np.concatenate([[0, 1, 127, 128, rows - 129, rows - 1], rng.integers(0, rows, size=128)]))
    sub = torch.from_numpy(np.ascontiguousarray(w.reshape(rows, -1)[pick]).reshape(-1)).cuda()
    part = ops.dequant(ops.Fp4(sub, torch.tensor([0.21], dtype=torch.float32, device="cuda"), len(pick), k), rule=True).view(len(pick), k)
    f32_close(y[:, torch.from_numpy(pick).cuda()], torch.from_numpy(x).cuda(), part, f"{rows}x{k} m={m}")
    assert device_status() == 0


def test_more_f32_rows_than_a_grid_has_in_y():
    rows, k, m = 128, 256, 65600
    rng = np.random.default_rng(9)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(0.37))
    x = torch.from_numpy(rng.standard_normal((64, k)).astype(np.float32)).cuda()
    y = ops.launch_gemm_fp4(ops.Fp4Packed(w), x.repeat(m // 64, 1))
    assert torch.equal(y.view(torch.int32), y[:64].view(torch.int32).repeat(m // 64, 1))
    f32_close(y[:64], x, ops.dequant(w, rule=True).view(rows, k), "first rows")
    assert device_status() == 0


@pytest.mark.parametrize("rows,k,m", [(333, 256, 1), (1, 512, 31), (129, 2048, 32), (640, 17408, 33), (2000, 1280, 65)])
def test_block_scaled_gemm_at_the_edges_of_its_tiles(rows, k, m):
    """One and more 128-row tiles, whole and ragged blocks of 32 tokens, an odd count of them, k in one part and several; rows far apart, results in rows
    further apart than they are long."""
    rng = np.random.default_rng(rows + k + m)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(0.37))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda()
    x[m // 2] *= 2.0 ** -20
    wide = torch.zeros((m, rows + 5), device="cuda")
    ops.launch_gemm_fp4(ops.Fp4Packed(w), x, wide[:, :rows])
    f32_close(wide[:, :rows], x, ops.dequant(w, rule=True).view(rows, k), f"{rows}x{k} m={m}")
    assert not wide[:, rows:].any()
    assert device_status() == 0
