"""The work a decode / prefill host has this library do, as timed cases.

Kinds, and the call behind each (every one through the package's public operators):

  gemv   `ops.launch_gemv`: one quantized projection of a decode (m = 1) or verify (m <= 8) step, launched on its own
  ffn    `ops.dense_ffn_w`: fused gate/up + activation, then down
  head   `ops.lm_head_argmax`: vocabulary projection and token choice
  stack  `dense.DenseStack.decode_step`: a whole decode step of the dense stack, captured once, host row in and host row out
  moe    `moe.GpuMoePlan.run`: router, routed NVFP4 experts, shared expert, combine
  mul1   `moe.route_softmax_topk` + `mul1.Mul1Plan.moe`: the same over MUL1 trellis records
  gemm   `ops.launch_gemm`: batched (prompt) rows on the container layout
  fp4    `ops.launch_gemm_fp4`: batched rows on the re-laid weights
  fp8    `ops.fp8_gemv`: an FP8 projection

Weights have the distribution of `crownest_b200.synth`: uniform E2M1 codes, scale bytes E4M3(|N(0,1)| * 0.05).
"""
import math

import torch

from crownest_b200 import dense, moe, mul1, ops

DEV = "cuda"


def listed():
    return [
        # one square projection on its own: the smallest call a host makes, once per token and matrix
        {"name": "gemv 4096x4096 m1", "kind": "gemv", "rows": 4096, "k": 4096, "m": 1, "dtype": "bf16"},
        # one dense FFN at the engine's own activation type
        {"name": "ffn 5120-17408 f32 m1", "kind": "ffn", "hidden": 5120, "inter": 17408, "m": 1, "dtype": "f32", "limit": 0.0},
        # a token through the 27B-shaped dense stack, and the same stack verifying four drafted rows
        {"name": "stack 64 layers m1", "kind": "stack", "hidden": 5120, "qkv": 7168, "inter": 17408, "layers": 64, "m": 1},
        {"name": "stack 64 layers m4", "kind": "stack", "hidden": 5120, "qkv": 7168, "inter": 17408, "layers": 64, "m": 4},
        # the routed-expert step of one token inside a captured decode step, and of a serving batch launched plainly
        {"name": "moe 512x10 1 token", "kind": "moe", "hidden": 2048, "inter": 512, "experts": 512, "topk": 10, "shared": 512, "router": "softmax",
         "tokens": 1, "dtype": "bf16", "graph": True},
        {"name": "moe 512x10 64 tokens", "kind": "moe", "hidden": 2048, "inter": 512, "experts": 512, "topk": 10, "shared": 512, "router": "softmax",
         "tokens": 64, "dtype": "bf16", "graph": False},
        # the 3-bit trellis experts for one token (plain launches) and for sixteen (captured)
        {"name": "mul1 64x4 1 token", "kind": "mul1", "hidden": 4096, "inter": 1536, "experts": 64, "topk": 4, "K": 3.0, "tokens": 1, "dtype": "bf16",
         "graph": False},
        {"name": "mul1 64x4 16 tokens", "kind": "mul1", "hidden": 4096, "inter": 1536, "experts": 64, "topk": 4, "K": 3.0, "tokens": 16, "dtype": "bf16",
         "graph": True},
        # a batch of 64 rows on the block-scaled path, a short prompt and a prompt chunk on the container layout
        {"name": "fp4 gemm 17408x5120 m64", "kind": "fp4", "rows": 17408, "k": 5120, "m": 64},
        {"name": "gemm 17408x5120 m512", "kind": "gemm", "rows": 17408, "k": 5120, "m": 512},
        {"name": "gemm 5120x17408 m4096", "kind": "gemm", "rows": 5120, "k": 17408, "m": 4096},
        # an FP8 gate/up-sized projection
        {"name": "fp8 34816x5120 m1", "kind": "fp8", "rows": 34816, "k": 5120, "m": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "ffn", "head", "stack", "stack", "moe", "moe", "moe", "mul1", "mul1", "gemm", "gemm", "fp4", "fp8"])
    m = rng.choice([1, 1, 1, 2, 3, 4, 4, 5, 6, 7, 8])
    dtype = rng.choice(["bf16", "bf16", "f32"])
    if kind == "gemv":  # any row count, k in whole 256-value pieces
        return {"kind": kind, "rows": _log(rng, 64, 40000), "k": 256 * _log(rng, 2, 68), "m": m, "dtype": dtype}
    if kind == "ffn":
        return {"kind": kind, "hidden": 256 * _log(rng, 3, 24), "inter": 256 * _log(rng, 4, 68), "m": m, "dtype": dtype, "limit": rng.choice([0.0, 0.0, 10.0])}
    if kind == "head":  # f32 logits: bf16 ones tie
        return {"kind": kind, "rows": rng.randrange(20000, 248321), "k": 256 * rng.randrange(8, 21), "m": m}
    if kind == "stack":
        return {"kind": kind, "hidden": 256 * rng.randrange(8, 21), "qkv": 128 * rng.randrange(24, 65), "inter": 256 * rng.randrange(16, 69),
                "layers": _log(rng, 2, 60), "m": m}
    if kind == "moe":
        tokens = _log(rng, 1, 128)
        graph = rng.random() < 0.5
        if rng.random() < 0.3:  # larger experts, sigmoid router with bias, clamped activation
            return {"kind": kind, "hidden": 4096, "inter": 2048, "experts": 288, "topk": 8, "shared": rng.choice([0, 2048]), "router": "sigmoid",
                    "tokens": min(tokens, 32), "dtype": dtype, "graph": graph}
        return {"kind": kind, "hidden": rng.choice([2048, 2048, 1024, 2560]), "inter": rng.choice([512, 512, 768, 1280]),
                "experts": rng.choice([512, 512, 128, 64]), "topk": rng.choice([10, 10, 8, 6]), "shared": rng.choice([512, 512, 0]), "router": "softmax",
                "tokens": tokens, "dtype": dtype, "graph": graph}
    if kind == "mul1":
        big = rng.random() < 0.6
        return {"kind": kind, "hidden": 4096 if big else 128 * rng.randrange(8, 33), "inter": 1536 if big else 128 * rng.randrange(4, 17),
                "experts": rng.choice([64, 64, 32]), "topk": rng.choice([4, 4, 8]), "K": rng.choice([3.0, 3.0, 3.0, 2.0, 3.5, 4.0]),
                "tokens": _log(rng, 1, 32), "dtype": dtype, "graph": rng.random() < 0.5}
    if kind == "gemm":
        rows, k = rng.choice([(17408, 5120), (5120, 17408), (8192, 5120), (5120, 5120), (rng.randrange(1000, 12000), 256 * rng.randrange(4, 40))])
        return {"kind": kind, "rows": rows, "k": k, "m": _log(rng, 9, 4000)}
    if kind == "fp4":  # the range the block-scaled path is meant for
        rows, k = rng.choice([(17408, 5120), (5120, 17408), (8192, 5120), (rng.randrange(1000, 12000), 256 * rng.randrange(4, 40))])
        return {"kind": kind, "rows": rows, "k": k, "m": _log(rng, 16, 256)}
    return {"kind": "fp8", "rows": _log(rng, 256, 34816), "k": 128 * _log(rng, 8, 136), "m": m}


def _nvfp4(rows, k, gen):
    blocks = rows * k // 64
    w = torch.randint(0, 256, (blocks, 36), dtype=torch.uint8, device=DEV, generator=gen)
    w[:, :4] = (torch.randn((blocks, 4), device=DEV, generator=gen).abs_() * 0.05).to(torch.float8_e4m3fn).view(torch.uint8)
    return w.view(-1)


def _fp4(rows, k, gen):
    return ops.Fp4(_nvfp4(rows, k, gen), torch.ones(1, device=DEV), rows, k)


def _slabs(experts, rows, k, gen):
    """One resident slab per expert, as views of one allocation."""
    return list(_nvfp4(experts * rows, k, gen).view(experts, -1).unbind(0))


def _rows(m, k, gen, dtype="bf16", scale=1.0):
    x = torch.randn((m, k), device=DEV, generator=gen) * scale
    return x.to(torch.bfloat16) if dtype == "bf16" else x


def _records(c, gen):
    """MUL1 records: a uniform code stream for gate | up | down, then six fp16 scale vectors with random signs (the sign
    half of the Hadamard rotation)."""
    h, i, n = c["hidden"], c["inter"], c["experts"]
    size = mul1.record_bytes(h, i, c["K"])
    rec = torch.randint(0, 256, (n, size), dtype=torch.uint8, device=DEV, generator=gen)
    at = int(3 * (h // 16) * (i // 16) * 32 * c["K"])
    vec = 3 * (h + i)
    v = torch.randn((n, vec), device=DEV, generator=gen).abs_() * 0.02 + 1e-3
    v *= torch.randint(0, 2, (n, vec), device=DEV, generator=gen) * 2 - 1
    rec[:, at:at + 2 * vec] = v.to(torch.float16).view(torch.uint8)
    rec[:, at + 2 * vec:] = 0
    return rec


def _captured(step):
    """The step as a host keeps it for a decode loop: recorded once, replayed per token."""
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        step()
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            out = step()
    return g, out


def prepare(case, seed):
    c = case
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    s = {"case": c}
    kind = c["kind"]
    if kind in ("gemv", "head"):
        s["w"] = _fp4(c["rows"], c["k"], gen)
        s["x"] = _rows(c["m"], c["k"], gen, c.get("dtype", "f32"))
    elif kind == "ffn":
        s["w"] = [_fp4(c["inter"], c["hidden"], gen), _fp4(c["inter"], c["hidden"], gen), _fp4(c["hidden"], c["inter"], gen)]
        s["x"] = _rows(c["m"], c["hidden"], gen, c["dtype"])
    elif kind == "stack":
        cfg = {n: c[n] for n in ("hidden", "qkv", "inter", "layers")}
        s["stack"] = dense.DenseStack(cfg, device=DEV, seed=seed, max_m=c["m"])
        s["stack"].capture(c["m"])
        s["x"] = _rows(c["m"], c["hidden"], gen).cpu().pin_memory()
        s["y"] = torch.empty_like(s["x"]).pin_memory()
    elif kind == "moe":
        h, i, n, sh = c["hidden"], c["inter"], c["experts"], c["shared"]
        shared = [_nvfp4(sh, h, gen), _nvfp4(sh, h, gen), _nvfp4(h, sh, gen)] if sh else None
        w = moe.GpuMoeWeights(h, i, n, 1.0, 1.0, gate_up=_slabs(n, 2 * i, h, gen), down=_slabs(n, h, i, gen), shared=shared, shared_gs=[1.0] * 3,
                              device=DEV)
        plan = moe.GpuMoePlan(h, i, n, c["topk"], c["tokens"], shared_inter=sh)
        x = _rows(c["tokens"], h, gen, c["dtype"])
        logits = torch.randn((c["tokens"], n), device=DEV, generator=gen)
        more = {"router": "softmax"}
        if c["router"] == "sigmoid":
            more = {"router": "sigmoid", "bias": torch.randn(n, device=DEV, generator=gen) * 0.1, "scale": 2.5, "limit": 10.0}
        elif sh:
            more["sgate"] = torch.randn(c["tokens"], device=DEV, generator=gen)
        y = torch.empty_like(x)

        def step():
            plan.run(w, logits, x, y, **more)
            return y, plan.ids, plan.wts

        s["step"] = step
    elif kind == "mul1":
        rec = _records(c, gen)
        table = torch.tensor([r.data_ptr() for r in rec.unbind(0)], dtype=torch.int64, device=DEV)
        plan = mul1.Mul1Plan(c["hidden"], c["inter"], c["K"], slots=c["tokens"] * c["topk"], tokens=1)
        x = _rows(c["tokens"], c["hidden"], gen, c["dtype"], 0.25)
        logits = torch.randn((c["tokens"], c["experts"]), device=DEV, generator=gen)
        y = torch.empty_like(x)
        s["records"] = rec

        def step():
            ids, wts = moe.route_softmax_topk(logits, c["topk"])
            plan.moe(table, ids, wts, x, y=y, limit=10.0)
            return y, ids, wts

        s["step"] = step
    elif kind in ("gemm", "fp4"):
        w = _fp4(c["rows"], c["k"], gen)
        s["w"] = w if kind == "gemm" else ops.Fp4Packed(w)
        s["x"] = _rows(c["m"], c["k"], gen)
        s["y"] = torch.empty((c["m"], c["rows"]), dtype=torch.bfloat16, device=DEV)
        s["ws"] = torch.empty(ops.gemm_workspace_bytes(c["k"], c["m"]), dtype=torch.uint8, device=DEV) if kind == "gemm" else None
    else:
        s["w"] = (torch.randn((c["rows"], c["k"]), device=DEV, generator=gen) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
        s["scale"] = torch.rand((-(-c["rows"] // 128), -(-c["k"] // 128)), device=DEV, generator=gen) * 1e-3 + 1e-4
        s["x"] = _rows(c["m"], c["k"], gen)
    if c.get("graph"):
        s["graph"], s["out"] = _captured(s["step"])
    return s


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "gemv":
        return ops.launch_gemv(s["w"], s["x"])
    if kind == "ffn":
        return ops.dense_ffn_w(*s["w"], s["x"], limit=c["limit"])
    if kind == "head":
        return ops.lm_head_argmax(s["w"], s["x"])
    if kind == "stack":
        st = s["stack"]
        return st.decode_step(s["x"], s["y"]), st.q, st.o, st.h
    if kind in ("moe", "mul1"):
        if "graph" in s:
            s["graph"].replay()
            return s["out"]
        return s["step"]()
    if kind == "gemm":
        return ops.launch_gemm(s["w"], s["x"], s["y"], workspace=s["ws"])
    if kind == "fp4":
        return ops.launch_gemm_fp4(s["w"], s["x"], s["y"])
    return ops.fp8_gemv(s["w"], s["scale"], s["x"], c["rows"], c["k"])


def work(case):
    """Weights read once (0.5625 B per NVFP4 value; of routed experts the expected number of distinct ones), activations in
    and results out once, 2 flops per weight and row."""
    c = case
    kind = c["kind"]
    es = 4 if c.get("dtype") == "f32" or kind == "head" else 2
    if kind in ("gemv", "head", "gemm", "fp4", "fp8"):
        rows, k, m = c["rows"], c["k"], c["m"]
        wb = rows * k * (0.5625 if kind != "fp8" else 1.0)
        return {"bytes": wb + m * (rows + k) * es, "flops": 2.0 * m * rows * k}
    if kind == "ffn":
        n = 3 * c["hidden"] * c["inter"]
        return {"bytes": n * 0.5625 + 2 * c["m"] * c["hidden"] * es, "flops": 2.0 * c["m"] * n}
    if kind == "stack":
        n = c["layers"] * (c["hidden"] * (c["qkv"] + c["hidden"]) + 3 * c["hidden"] * c["inter"])
        return {"bytes": n * 0.5625 + 2 * c["m"] * c["hidden"] * es, "flops": 2.0 * c["m"] * n}
    t, n = c["tokens"], 3 * c["hidden"] * c["inter"]
    distinct = c["experts"] * (1 - (1 - c["topk"] / c["experts"]) ** t)
    act = t * (2 * c["hidden"] * es + 4 * c["experts"] + 8 * c["topk"])
    if kind == "moe":
        sh = 3 * c["hidden"] * c["shared"]
        return {"bytes": distinct * n * 0.5625 + sh * 0.5625 + act, "flops": 2.0 * t * (c["topk"] * n + sh)}
    return {"bytes": distinct * (n * c["K"] / 8 + 6 * (c["hidden"] + c["inter"])) + act, "flops": 2.0 * t * c["topk"] * n}


def tolerance(case):
    """f32 results differ by the order of 32-bit sums (and 22-bit activation planes); bf16 results by a rounding of each
    side, the largest by two units in the last place. Expert picks and tokens are whole numbers and stay the same."""
    if case.get("dtype") == "f32" or case["kind"] == "head":
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 5e-3, "max": 2e-2}
