"""Several bf16 rows over shapes whose tiles are shared by clusters of two or four CTAs, each over its part of k: few long rows, rows
that end inside a tile, activation rows that fill their slots or not."""
import numpy as np
import pytest
import torch

from crownest_b200 import device_status, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,gu", [(5120, 17408, False), (5111, 17408, False), (2560, 17408, True), (640, 17408, False), (333, 9216, False)])
@pytest.mark.parametrize("m", [2, 3, 4, 5, 8])
def test_rows_of_a_shared_tile(rows, k, gu, m):
    rng = np.random.default_rng(rows + k + m)
    w = [ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(1e-3)) for _ in range(2 if gu else 1)]
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    y64 = [x.double() @ ops.dequant(a).double().view(rows, k).t() for a in w]
    call = (lambda: ops.launch_gemv_gu(w[0], w[1], x)) if gu else (lambda: ops.launch_gemv(w[0], x))
    y = call()
    want = y64[0] / (1 + torch.exp(-y64[0])) * y64[1] if gu else y64[0]
    # one rounding to bf16, 2^-9 at most, beside f32 sums
    assert (y.double() - want).norm() <= (2.0 ** -9 + 4e-6) * want.norm()
    assert torch.equal(y.view(torch.int16), call().view(torch.int16))
    assert device_status() == 0
