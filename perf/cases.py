"""The calls a user of this framework makes, with the sizes they are made at.

Six public entry points: the compiled MXFP4 scaled-GEMM template (eager, or replayed from a CUDA graph as a decode loop
does), its split-K form that adds into C, `MXFP4Linear` (activations quantised on the fly), the MXFP8 / mixed template,
the routed expert MLP, and the quantiser that turns a trained weight into codes and scales. M runs from one decode row
to a long prefill; N and K over the projections of the configurations in bench.py, the tests and the reference's
benchmark list (K = 16000). Weights are N(0, 0.02), activations N(0, 1), router logits N(0, 1).
"""

import torch

import wave_b200 as wb
from wave_b200 import bf16, f32, ops
from wave_b200.graphs import GraphedScaledGemm

DEV = "cuda"
TORCH = {"f32": torch.float32, "bf16": torch.bfloat16}
WAVE = {"f32": f32, "bf16": bf16}
VARIANT = wb.ScaledMMAType.F32_16x16x128_F8F6F4


def listed():
    return [
        # the smallest call: the parity configuration of the tests, bound by launches and latency
        dict(name="gemm_1k_f32", kind="gemm", M=1024, N=1024, K=1024, out="f32", graph=False),
        # a decode step's projection at batch 16, replayed from a CUDA graph as a decode loop runs it
        dict(name="gemm_decode_m16_graph", kind="gemm", M=16, N=28672, K=8192, out="bf16", graph=True),
        # a prefill chunk of an odd number of tokens through a gate|up projection
        dict(name="gemm_prefill_1111", kind="gemm", M=1111, N=14336, K=4096, out="bf16", graph=False),
        # long prefill: the headline benchmark's shape
        dict(name="gemm_prefill_8k", kind="gemm", M=8192, N=8192, K=8192, out="bf16", graph=False),
        # few output tiles and a long K, adding into a zeroed C: what the split-K templates are for
        dict(name="splitk_512x2048x16000", kind="splitk", M=512, N=2048, K=16000, out="f32"),
        # one decode step of a layer that quantises its own activations, small batch
        dict(name="linear_decode_m8", kind="linear", M=8, N=14336, K=4096, out="bf16"),
        # the same layer type at the other end: a ragged prefill
        dict(name="linear_prefill_3000", kind="linear", M=3000, N=8192, K=8192, out="bf16"),
        # 8-bit operands, prefill
        dict(name="mxfp8_prefill_4k", kind="gemm8", M=4096, N=8192, K=4096, out="bf16", fmt="f8e4m3fn", wbits=8),
        # 8-bit activations against 4-bit weights, decode at batch 64
        dict(name="mixed_decode_m64", kind="gemm8", M=64, N=28672, K=8192, out="bf16", fmt="f8e4m3fn", wbits=4),
        # the expert MLP of the mixture-of-experts configuration, prefill of 4096 tokens
        dict(name="moe_prefill_4096", kind="moe", T=4096, E=8, top_k=2, K=4096, I=7168),
        # the same experts in a decode step of 16 sequences
        dict(name="moe_decode_16", kind="moe", T=16, E=8, top_k=2, K=4096, I=7168),
        # quantising a projection weight when a model is loaded
        dict(name="quantize_28672x8192", kind="quantize", rows=28672, K=8192, src="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _sizes(rng, m_hi, k_step, mnk_max):
    """M, N, K of a projection: log-uniform, N sometimes odd, M cut down where the product would be too large."""
    m = _log(rng, 1, m_hi)
    n = _log(rng, 512, 28672)
    n = n if rng.random() < 0.25 else max(512, n // 64 * 64)
    k = max(512, _log(rng, 512, 16384) // k_step * k_step)
    return max(1, min(m, mnk_max // (n * k))), n, k


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "splitk", "linear", "linear", "gemm8", "moe", "moe", "quantize"])
    out = rng.choice(["bf16", "bf16", "f32"])
    if kind == "gemm":
        m, n, k = _sizes(rng, 8192, 32, 2 ** 38)
        return dict(kind=kind, M=m, N=n, K=k, out=out, graph=m <= 128 and rng.random() < 0.5)
    if kind == "splitk":
        m, n, k = _sizes(rng, 2048, 256, 2 ** 36)
        return dict(kind=kind, M=m, N=n, K=max(1280, k // 640 * 640), out="f32")
    if kind == "linear":
        m, n, k = _sizes(rng, 8192, 32, 2 ** 38)
        return dict(kind=kind, M=m, N=n, K=k, out=out)
    if kind == "gemm8":
        m, n, k = _sizes(rng, 8192, 128, 2 ** 37)
        return dict(kind=kind, M=m, N=n, K=k, out=out, fmt=rng.choice(["f8e4m3fn", "f8e5m2"]), wbits=rng.choice([8, 4]))
    if kind == "moe":
        k, i, e = _log(rng, 1024, 4096) // 128 * 128, _log(rng, 1024, 7168) // 128 * 128, rng.choice([4, 8, 16])
        return dict(kind=kind, T=_log(rng, 1, 4096), E=e, top_k=rng.choice([1, 2, 2]), K=k, I=i)
    k = max(512, _log(rng, 512, 16384) // 32 * 32)
    return dict(kind=kind, rows=_log(rng, 64, min(28672, 2 ** 28 // k)), K=k, src=rng.choice(["bf16", "f32"]))


def _normal(gen, rows, cols, std, dtype=torch.bfloat16):
    return torch.randn(rows, cols, generator=gen, device=DEV, dtype=torch.float32).mul_(std).to(dtype)


def _fp4(gen, rows, cols, std):
    q, s, _ = wb.quantize_mxfp4(_normal(gen, rows, cols, std))
    return q, s


def _fp8(gen, rows, cols, std, fmt):
    dtype = torch.float8_e4m3fn if fmt == "f8e4m3fn" else torch.float8_e5m2
    q, s, _ = ops.quantize_mxfp8(_normal(gen, rows, cols, std), dtype)
    return q, s


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "quantize":
        return dict(kind=kind, x=_normal(gen, case["rows"], case["K"], 0.02, TORCH[case["src"]]))
    if kind == "moe":
        T, E, K, I = case["T"], case["E"], case["K"], case["I"]
        w1 = [_fp4(gen, 2 * I, K, 0.02) for _ in range(E)]
        w2 = [_fp4(gen, K, I, 0.02) for _ in range(E)]
        mlp = wb.MXFP4ExpertMLP([q for q, _ in w1], [s for _, s in w1], [q for q, _ in w2], [s for _, s in w2], top_k=case["top_k"])
        logits = torch.randn(T, E, generator=gen, device=DEV)
        return dict(kind=kind, mlp=mlp, x=_normal(gen, T, K, 1.0), logits=logits)
    M, N, K = case["M"], case["N"], case["K"]
    if kind == "linear":
        layer = wb.MXFP4Linear(*_fp4(gen, N, K, 0.02), output_dtype=TORCH[case["out"]])
        return dict(kind=kind, layer=layer, x=_normal(gen, M, K, 1.0))
    c = torch.empty(M, N, dtype=TORCH[case["out"]], device=DEV)
    if kind == "gemm8":
        a, a_s = _fp8(gen, M, K, 1.0, case["fmt"])
        b, b_s = _fp8(gen, N, K, 0.02, case["fmt"]) if case["wbits"] == 8 else _fp4(gen, N, K, 0.02)
        template, subs = wb.get_scaled_gemm_mxfp8_kernel((M, N, K), VARIANT, case["fmt"], WAVE[case["out"]],
                                                         weight_format="f4e2m1fn" if case["wbits"] == 4 else None)
        options = wb.WaveCompileOptions(subs=subs)
    else:
        a, a_s = _fp4(gen, M, K, 1.0)
        b, b_s = _fp4(gen, N, K, 0.02)
        if kind == "splitk":
            template, options = wb.get_tagged_splitk_mxfp4_gemm((M, N, K), num_splits=5, block_shape=(128, 128, 128), output_type=f32)
        else:
            template, options = wb.get_tagged_mxfp4_gemm((M, N, K), output_dtype=WAVE[case["out"]])
    gemm = wb.wave_compile(wb.set_default_run_config(options), template)
    args = (a, a_s, b, b_s, c)
    graph = GraphedScaledGemm(gemm, *args) if case.get("graph") else None
    return dict(kind=kind, gemm=gemm, args=args, graph=graph)


def run(state):
    kind = state["kind"]
    if kind == "quantize":
        codes, scales, packed = wb.quantize_mxfp4(state["x"])
        return codes, scales, packed.data
    if kind == "moe":
        return state["mlp"](state["x"], state["logits"])
    if kind == "linear":
        return state["layer"](state["x"])
    c = state["args"][4]
    if state["graph"] is not None:
        state["graph"].replay()
        return c
    if kind == "splitk":
        c.zero_()  # the template adds into a C that the caller initialises
    state["gemm"](*state["args"])
    return c


def _mx(rows, cols, bits=4):
    return rows * cols * bits / 8 + rows * cols / 32


def work(case):
    kind = case["kind"]
    if kind == "quantize":
        elem = 4 if case["src"] == "f32" else 2
        n = case["rows"] * case["K"]
        return {"bytes": n * elem + _mx(case["rows"], case["K"]) + n / 32, "flops": 0}
    if kind == "moe":
        T, E, K, I, top = case["T"], case["E"], case["K"], case["I"], case["top_k"]
        used = E * (1 - (1 - top / E) ** T)  # experts that a batch of T tokens reaches, on average
        return {"bytes": T * K * 2 * 2 + T * E * 4 + used * (_mx(2 * I, K) + _mx(K, I)), "flops": 2.0 * T * top * 3 * I * K}
    M, N, K = case["M"], case["N"], case["K"]
    c_bytes = M * N * (4 if case["out"] == "f32" else 2)
    flops = 2.0 * M * N * K
    if kind == "linear":
        return {"bytes": M * K * 2 + _mx(N, K) + c_bytes, "flops": flops}
    if kind == "gemm8":
        return {"bytes": _mx(M, K, 8) + _mx(N, K, case["wbits"]) + c_bytes, "flops": flops}
    return {"bytes": _mx(M, K) + _mx(N, K) + c_bytes, "flops": flops}


def tolerance(case):
    """Relative 2-norm against the same path in 64 bits (dequantised operands, f64 sums), measured on every listed case,
    times about four."""
    if case["kind"] == "quantize":
        return "exact"  # bytes
    if case["kind"] == "moe":
        # 0.030: the hidden activations are quantised to four bits inside the path, and a value next to a rounding
        # boundary goes to the other side when it was rounded to bf16 first and not in the exact path
        return {"rel": 0.1}
    # 0 to 3e-8 for f32 (sums of a few thousand products of 4- or 8-bit values; the order matters little), 1.66e-3 for
    # bf16, which is its rounding
    return {"rel": 1e-5} if case["out"] == "f32" else {"rel": 7e-3}
