"""f32 rows on the tensor cores (k >= 2048): three f16 planes per row as MMA columns. Sizes at the edges of its tiles (16 rows, 8
indices in the gate/up form), of its parts (72 blocks of 64 values, parts of unequal length) and column groups (2, 5 and 8
rows), the shapes that share a tile between CTAs, and a k at which eight rows become two calls."""
import numpy as np
import pytest
import torch

import oracle
from crownest_b200 import device_status, ops, synth

pytestmark = pytest.mark.gpu


def _make(rows, k, seed, gs=1.7e-3):
    rng = np.random.default_rng(seed)
    w = ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(gs))
    return rng, w, ops.dequant(w).double().view(rows, k)


def _check(y, w64, x):
    """Each product is cut at 2^-24 of its block's largest or better and every partial sum rounds once: a term passes one
    rounding per block of its sum (k / 64 / 8 of them at most per warp, 8 sums, the parts), far fewer than k / 64 + 16."""
    ref, mag = x.double() @ w64.t(), x.double().abs() @ w64.abs().t()
    n = x.shape[1] // 64 + 16
    assert ((y.double() - ref).abs() <= n * 2.0 ** -24 * mag + 1e-30).all()
    assert (y.double() - ref).norm() <= 2.0 ** -23 * ref.norm()  # one f32 ulp in the norm
    assert device_status() == 0


@pytest.mark.parametrize("rows,k", [(1, 2048), (17, 2304), (777, 5120), (4097, 4096), (300, 4864), (2500, 8960), (640, 17408), (5120, 17408), (16, 47616)])
@pytest.mark.parametrize("kind", ["normal", "heavy"])
def test_rows_against_64_bits_and_one_row_calls(rows, k, kind):
    rng, w, w64 = _make(rows, k, rows + k)
    xh = rng.standard_normal((8, k)).astype(np.float32)
    if kind == "heavy":
        xh *= np.exp(2 * rng.standard_normal((8, k))).astype(np.float32)
        xh[3] = 0.0
        xh[2, : k // 2] *= 1e-30  # blocks near the bottom of the exponent range
    x = torch.from_numpy(xh).cuda()
    ones = torch.cat([ops.launch_gemv(w, x[i:i + 1]) for i in range(8)])
    _check(ones, w64, x)
    for m in (2, 3, 5, 6, 8):
        y = ops.launch_gemv(w, x[:m])
        assert torch.equal(y.view(torch.int32), ones[:m].view(torch.int32)), m


@pytest.mark.parametrize("inter,k,m", [(9, 2048, 1), (1111, 2560, 2), (3000, 5120, 4), (2560, 17408, 8)])
def test_gate_up(inter, k, m):
    rng, g, g64 = _make(inter, k, 5, 0.8e-3)
    _, u, u64 = _make(inter, k, 6, 700.0)
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda()
    gg, uu = x.double() @ g64.t(), x.double() @ u64.t()
    want = gg / (1 + torch.exp(-gg)) * uu
    got = ops.launch_gemv_gu(g, u, x)
    # silu(g) * u of two sums within 2^-23 each, and a handful of f32 roundings (expf 2 ulp, divide, two products)
    assert (got.double() - want).norm() <= 8 * 2.0 ** -23 * want.norm()
    assert device_status() == 0


def test_not_finite_values_reach_their_row_only():
    rng, w, w64 = _make(64, 2048, 7)
    xh = rng.standard_normal((3, 2048)).astype(np.float32)
    xh[1, 100], xh[2, 7] = np.inf, np.nan
    y = ops.launch_gemv(w, torch.from_numpy(xh).cuda()).cpu().numpy()
    col = w64[:, 100].cpu().numpy()
    _check(torch.from_numpy(y[:1]).cuda(), w64, torch.from_numpy(xh[:1]).cuda())
    assert np.array_equal(y[1][col != 0], np.inf * np.sign(col[col != 0]).astype(np.float32)) and np.isnan(y[1][col == 0]).all()
    assert np.isnan(y[2]).all()
