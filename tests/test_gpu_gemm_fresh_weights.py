"""Batched GEMM calls whose weights, re-laid weights or tensor scale are written by the kernel directly in front of the call, in the same stream and
without a pause: results are those of the same call after a synchronisation. The kernels in front are one that lets its successor start early
(a GEMV of the library, which writes the values as its results), a device copy and the repack."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from crownest_b200 import device_status, ops, synth


def matrix(rows, k, seed):
    return ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, np.random.default_rng(seed)), rows, k, 0.5)


@pytest.mark.parametrize("m,dtype", [(1, torch.bfloat16), (64, torch.bfloat16), (128, torch.float32), (200, torch.float32), (300, torch.bfloat16)])
@pytest.mark.parametrize("relaid", [False, True])
def test_weights_and_scale_of_the_kernel_in_front(m, dtype, relaid):
    rows, k = 1024, 2048
    x = torch.randn((m, k), device="cuda").to(dtype)
    old, new = matrix(rows, k, 1), matrix(rows, k, 2)
    # a GEMV over many long rows: its launch lets the next one start at once and runs for some twenty microseconds
    busy, bx = matrix(17408, 8192, 3), torch.randn((1, 8192), device="cuda").to(torch.bfloat16)
    w = ops.Fp4(old.w.clone(), torch.ones(1, device="cuda"), rows, k)
    scale_row, sx = matrix(1, 8192, 4), torch.randn((1, 8192), device="cuda")
    y = torch.empty((m, rows), dtype=dtype, device="cuda")

    def call(weights):
        return (ops.launch_gemm_fp4 if relaid else ops.launch_gemm)(weights, x, y)

    def fresh_bytes(pause):
        w.w.copy_(old.w)
        p = ops.Fp4Packed(w) if relaid else w
        torch.cuda.synchronize()
        target = p.packed if relaid else p.w
        # the first 34,816 bytes of the weights are the results of the GEMV in front
        ops.launch_gemv(busy, bx, target[:34816].view(torch.bfloat16).view(1, 17408))
        if pause:
            torch.cuda.synchronize()
        return call(p).clone()

    def copied(pause):
        w.w.copy_(old.w)
        torch.cuda.synchronize()
        w.w.copy_(new.w)
        p = ops.Fp4Packed(w) if relaid else w
        if pause:
            torch.cuda.synchronize()
        return call(p).clone()

    def fresh_scale(pause):
        w.w.copy_(new.w)
        w.gs.fill_(1.0)
        p = ops.Fp4Packed(w) if relaid else w
        torch.cuda.synchronize()
        ops.launch_gemv(scale_row, sx, w.gs.view(1, 1))  # one long f32 row
        if pause:
            torch.cuda.synchronize()
        return call(p).clone()

    for form in (fresh_bytes, copied, fresh_scale):
        want = form(True)
        for _ in range(3):
            got = form(False)
            bits = torch.int16 if dtype == torch.bfloat16 else torch.int32
            assert torch.equal(got.view(bits), want.view(bits)), form.__name__
    assert device_status() == 0
