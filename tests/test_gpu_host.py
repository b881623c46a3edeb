"""The native host side of the small operators: forms of the arguments (one dimension, rows apart, given outputs and leading dimensions), the stream of the
caller, and the errors."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from crownest_b200 import CrownestError, ops, synth


def matrix(rows=320, k=512, seed=1):
    return ops.Fp4.from_host(synth.nvfp4_matrix(rows, k, np.random.default_rng(seed)), rows, k, 0.5)


def test_forms_of_the_arguments():
    w, x = matrix(), torch.randn((3, 512), device="cuda").to(torch.bfloat16)
    y = ops.launch_gemv(w, x)
    assert y.shape == (3, 320) and y.dtype == x.dtype and y.is_contiguous()
    assert torch.equal(ops.launch_gemv(w, x.view(-1)), y)
    apart = torch.zeros((3, 1024), device="cuda", dtype=x.dtype)
    apart[:, ::2] = x
    assert torch.equal(ops.launch_gemv(w, apart[:, ::2]), y)  # not contiguous: copied
    assert torch.equal(ops.launch_gemv(w, x.view(3, 1, 512)), y)
    wide = torch.zeros((3, 400), device="cuda", dtype=x.dtype)
    out = wide[:, :320]
    assert ops.launch_gemv(w, x, out) is out and torch.equal(out, y) and not wide[:, 320:].any()
    flat = torch.zeros(3 * 352, device="cuda", dtype=x.dtype)
    assert ops.launch_gemv(w, x, flat, ldy=352) is flat and torch.equal(flat.view(3, 352)[:, :320], y)
    assert torch.equal(ops.dense_proj(w, x.float()).to(x.dtype).float().isfinite(), torch.ones((3, 320), device="cuda", dtype=torch.bool))
    tokens, logits = ops.lm_head_argmax(w, x.float())
    assert tokens.dtype == torch.int32 and torch.equal(tokens.long(), logits.argmax(1))


def test_the_callers_stream():
    w, x = matrix(2048, 2048), torch.randn((1, 2048), device="cuda").to(torch.bfloat16)
    want = ops.launch_gemv(w, x)
    st, y, src = torch.cuda.Stream(), torch.zeros_like(want), torch.empty_like(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(20_000_000)
        src.copy_(x)  # the call reads what this stream has copied by then
        ops.launch_gemv(w, src, y)
        got = y.clone()
    st.synchronize()
    assert torch.equal(got, want)


def test_errors():
    w = matrix()
    with pytest.raises(CrownestError, match="bf16 or f32, got torch.float16"):
        ops.launch_gemv(w, torch.zeros((1, 512), device="cuda", dtype=torch.float16))
    with pytest.raises(CrownestError, match="activation rows"):
        ops.launch_gemv(w, torch.zeros((9, 512), device="cuda", dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match="invalid for input of size"):
        ops.launch_gemv(w, torch.zeros((1, 500), device="cuda", dtype=torch.bfloat16))
    with pytest.raises(CrownestError, match="scales, the 128x128 grid"):
        ops.fp8_gemv(torch.zeros(128 * 256, device="cuda", dtype=torch.uint8), torch.zeros(1, device="cuda"), torch.zeros((1, 256), device="cuda"), 128, 256)
    with pytest.raises(TypeError):
        ops.launch_gemv(w, None)
