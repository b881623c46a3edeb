"""Several bf16 rows over matrices whose rows are summed in one, two or four parts of k, by the CTAs of a cluster or by one CTA after another, with one or
two teams of warps to a CTA: few long rows, a matrix that fills the machine, rows that end inside a tile, activation rows that fill their slots or not. Every row has the
bits of a one-row call."""
import numpy as np
import pytest
import torch

from crownest_b200 import device_status, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,gu", [(5120, 17408, False), (5111, 17408, False), (2560, 17408, True), (640, 17408, False), (1280, 17408, False),
                                       (333, 9216, False), (2048, 8192, False), (2048, 12288, False), (999, 12288, True), (320, 33792, False),
                                       # one part: two teams of a CTA with one tile, with uneven shares, with short rows, with none for the second
                                       (3000, 5120, True), (7161, 5120, False), (700, 1536, False), (40, 4096, False)])
@pytest.mark.parametrize("m", [2, 3, 4, 5, 8])
def test_rows_of_a_shared_tile(rows, k, gu, m):
    rng = np.random.default_rng(rows + k + m)
    w = [ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, rng), rows, k, np.float32(1e-3)) for _ in range(2 if gu else 1)]
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    y64 = [x.double() @ ops.dequant(a).double().view(rows, k).t() for a in w]
    call = (lambda v: ops.launch_gemv_gu(w[0], w[1], v)) if gu else (lambda v: ops.launch_gemv(w[0], v))
    y = call(x)
    want = y64[0] / (1 + torch.exp(-y64[0])) * y64[1] if gu else y64[0]
    # one rounding to bf16, 2^-9 at most, beside f32 sums
    assert (y.double() - want).norm() <= (2.0 ** -9 + 4e-6) * want.norm()
    assert torch.equal(y.view(torch.int16), call(x).view(torch.int16))
    for i in range(m):
        assert torch.equal(call(x[i:i + 1]).view(torch.int16)[0], y.view(torch.int16)[i]), i
    assert device_status() == 0
