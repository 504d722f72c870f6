"""The work whose speed counts: what a program that serves 4-bit weights has this package do, through its public calls.

A case is a dict of plain values. `listed()` gives the standing cases, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a program has in hand before the call (weights laid out once, activations), `run(state)` one
pass and its outputs, `work(case)` the bytes and operations a pass cannot do without, `tolerance(case)` how far another
correct implementation of the same precision may be from the result.

Kinds of work
  linear    one quantised linear layer on activations that are on the GPU: decode batches (1 to 32 rows on slab weights,
            also with the fused SiLU * mul and residual epilogues), batched decode and prefill (up to 4096 rows on
            canonical, interleaved or tiled weights)
  gemv      `gemv_int4`, per-channel quantisation: the drop-in for a script written against the original Python function
  host      a layer whose activations and result live in pinned host memory
  step      one token step through the linears of a decoder stack, captured as a CUDA graph
  token     the same step for a caller on the host: hidden state in, captured step, hidden state out
  unpack    packed codes to one code per byte
  dequant   packed weights to 16-bit weights
  convert   16-bit weights to packed codes, scales and zeros, and these into the layout a kernel reads (loading a model)
"""
import math

import torch

import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4
from quantforge_b200.stack import DecodeLinearStack, linear_bytes

_DT = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
_LAYOUT = {"canonical": qf.QF_LAYOUT_CANONICAL, "interleaved": qf.QF_LAYOUT_INTERLEAVED, "tiled": qf.QF_LAYOUT_TILED}
_EPI = {"none": qf.QF_EPI_NONE, "silu": qf.QF_EPI_SILU_MUL, "residual": qf.QF_EPI_RESIDUAL_ADD}

MAX_WEIGHTS = 8192 * 57344            # codes of the largest single matrix (gate and up of a wide layer together)
MAX_MACS = 2048 * 8192 * 28672        # multiply-adds of the largest linear
MAX_STEP_BYTES = 3_650_000_000        # weights of the largest stack


def listed():
    return [
        # One small decode linear called eagerly, the smallest call there is: latency and host work.
        {"name": "decode-1x4096x4096", "kind": "linear", "M": 1, "K": 4096, "N": 4096, "act": "f16", "out": "f16",
         "zeros": "u4", "group": 128, "layout": "slab", "epilogue": "none"},
        # The largest decode matrix: gate and up of a wide layer as one linear with the activation fused, four requests.
        {"name": "decode-4-gate-up", "kind": "linear", "M": 4, "K": 8192, "N": 57344, "act": "bf16", "out": "bf16",
         "zeros": "u4", "group": 128, "layout": "slab", "epilogue": "silu"},
        # The original script's call on sizes that divide nothing evenly, weights as they came from the file.
        {"name": "gemv-per-channel-ragged", "kind": "gemv", "M": 3, "K": 3968, "N": 5136},
        # Batched decode / speculative verification: 64 rows, long K, prepacked layer object, residual stream added.
        {"name": "batch-64-down", "kind": "linear", "M": 64, "K": 14336, "N": 4096, "act": "bf16", "out": "bf16",
         "zeros": "u4", "group": 128, "layout": "interleaved", "epilogue": "residual"},
        # A prompt of an odd length on a square projection, f16, signed zero points, weights not prepacked.
        {"name": "prefill-777-ragged", "kind": "linear", "M": 777, "K": 4096, "N": 4096, "act": "f16", "out": "f16",
         "zeros": "i8", "group": 256, "layout": "canonical", "epilogue": "none"},
        # A long prompt on the widest projection of a large model, symmetric weights.
        {"name": "prefill-2048-wide", "kind": "linear", "M": 2048, "K": 8192, "N": 28672, "act": "bf16", "out": "bf16",
         "zeros": "const", "group": 128, "layout": "tiled", "epilogue": "none"},
        # A layer called from host code, a few rows at a time: copies in and out belong to the call.
        {"name": "host-2x4096x14336", "kind": "host", "M": 2, "K": 4096, "N": 14336, "act": "f16", "layout": "canonical"},
        # One token through all linears of an 8B-shaped model at batch 1, hidden state from and to the host.
        {"name": "token-8b-batch-1", "kind": "token", "hidden": 4096, "kv": 1024, "ffn": 14336, "layers": 32, "batch": 1,
         "fused": True},
        # The same stack with sixteen requests in flight, hidden state on the GPU.
        {"name": "step-8b-batch-16", "kind": "step", "hidden": 4096, "kv": 1024, "ffn": 14336, "layers": 32, "batch": 16,
         "fused": True},
        # The two materialising operators on whole weight matrices.
        {"name": "unpack-28672x4096", "kind": "unpack", "rows": 28672, "cols": 4096},
        {"name": "dequant-14336x4096", "kind": "dequant", "N": 14336, "K": 4096, "act": "bf16", "zeros": "u4",
         "group": 128},
        # A checkpoint's weight on its way to the decode kernel.
        {"name": "convert-4096x4096", "kind": "convert", "N": 4096, "K": 4096, "act": "bf16", "group": 128,
         "symmetric": False, "layout": "slab"},
    ]


# ------------------------------------------------------------------------------------------------
# drawn cases
# ------------------------------------------------------------------------------------------------
def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _matrix(rng, n_step, most, k_hi=28672, n_hi=57344):
    while True:
        K, N = _log(rng, 512, k_hi, 128), _log(rng, 512, n_hi, n_step)
        if K * N <= most:
            return K, N


def _groups(rng, K):
    return rng.choice([g for g in (128, 128, 128, 256, K) if K % g == 0])


def draw(rng):
    kind = rng.choices(["linear", "gemv", "host", "step", "token", "unpack", "dequant", "convert"],
                       [12, 2, 2, 2, 2, 2, 2, 2])[0]
    act = rng.choice(["f16", "bf16"])
    if kind == "linear":
        layout = rng.choice(["slab", "slab", "canonical", "interleaved", "tiled", "tiled"])
        M = _log(rng, 1, 32 if layout == "slab" else 4096)
        epilogue = rng.choice(["none", "none", "silu", "residual"])
        # weights that were not prepacked may have any multiple of 16 rows in decode batches
        step = 64 if layout == "slab" else 16 if layout == "canonical" and M <= 16 and epilogue == "none" else 128
        K, N = _matrix(rng, step, min(MAX_WEIGHTS, MAX_MACS // M))
        return {"kind": kind, "M": M, "K": K, "N": N, "act": act, "out": rng.choice([act, act, "f32"]),
                "zeros": rng.choice(["u4", "u4", "i8", "const"]), "group": _groups(rng, K), "layout": layout,
                "epilogue": epilogue}
    if kind == "gemv":
        K, N = _matrix(rng, 16, 4096 * 28672)
        return {"kind": kind, "M": _log(rng, 1, 16), "K": K, "N": N}
    if kind == "host":
        layout = rng.choice(["canonical", "tiled"])
        K, N = _matrix(rng, 128, 8192 * 28672)
        return {"kind": kind, "M": _log(rng, 1, 256), "K": K, "N": N, "act": act, "layout": layout}
    if kind in ("step", "token"):
        hidden, kv, ffn = rng.choice([(4096, 1024, 14336), (8192, 1024, 28672),
                                      (_log(rng, 1024, 8192, 256), 512, _log(rng, 2048, 28672, 256))])
        per_layer = (2 * hidden * hidden + 2 * hidden * kv + 3 * hidden * ffn) // 2
        layers = _log(rng, 1, max(1, min(32, MAX_STEP_BYTES * 16 // 17 // per_layer)))
        return {"kind": kind, "hidden": hidden, "kv": kv, "ffn": ffn, "layers": layers, "batch": _log(rng, 1, 64),
                "fused": rng.random() < 0.8}
    if kind == "unpack":
        while True:
            rows, cols = _log(rng, 1, 28672), _log(rng, 64, 14336)
            if 4096 <= rows * cols <= 28672 * 4096:
                return {"kind": kind, "rows": rows, "cols": cols}
    if kind == "dequant":
        K, N = _matrix(rng, 16, 28672 * 8192)
        return {"kind": kind, "N": N, "K": K, "act": act, "zeros": rng.choice(["u4", "i8", "const"]),
                "group": _groups(rng, K)}
    K, N = _matrix(rng, 128, 4096 * 14336)
    return {"kind": kind, "N": N, "K": K, "act": act, "group": rng.choice([128, K]), "symmetric": rng.random() < 0.4,
            "layout": rng.choice(["slab", "tiled"])}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _quantised(gen, N, K, group, act, zeros):
    """Uniform codes and zero points, scales |N(0, 0.02)| / 7: the distributions of the package's benchmark."""
    dev, G = gen.device, K // group
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device=dev, generator=gen)
    sc = (torch.randn(G, N, device=dev, generator=gen).abs() * (0.02 / 7.0)).clamp_min(2.0 ** -14).to(_DT[act])
    if zeros == "const":
        return qw, sc, None
    z = torch.randint(0, 16, (G, N), dtype=torch.int8, device=dev, generator=gen)
    return qw, sc, qf.pack_zeros_u4(z) if zeros == "u4" else z - 8


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "linear":
        M, K, N, g = case["M"], case["K"], case["N"], case["group"]
        qw, sc, zr = _quantised(gen, N, K, g, case["act"], case["zeros"])
        st["x"] = torch.randn(M, K, device=dev, generator=gen).to(_DT[case["act"]])
        st["out_dtype"] = _DT[case["out"]]
        st["epilogue"] = _EPI[case["epilogue"]]
        st["residual"] = (torch.randn(M, N, device=dev, generator=gen).to(st["out_dtype"])
                          if case["epilogue"] == "residual" else None)
        if case["layout"] == "slab":
            st["slab"] = qf.prepack_gemv_slab(qw, sc, zr, group_size=g)
        elif case["layout"] == "canonical":
            st["layer"] = qf.W4A16Linear(qw, sc, zr, group_size=g)
        elif case["layout"] == "tiled":
            st["layer"] = qf.W4A16Linear(qw, sc, zr, group_size=g, prepack=True)
        else:
            st["layer"] = qf.W4A16Linear(qf.prepack_w4(qw), sc, zr, group_size=g, weight_layout=_LAYOUT["interleaved"])
    elif kind == "gemv":
        M, K, N = case["M"], case["K"], case["N"]
        st["w"] = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device=dev, generator=gen)
        st["scale"] = (torch.randn(N, device=dev, generator=gen).abs() * (0.02 / 7.0)).clamp_min(2.0 ** -14).half()
        st["zero"] = torch.randint(0, 16, (N,), dtype=torch.int8, device=dev, generator=gen)
        st["x"] = torch.randn(M, K, device=dev, generator=gen).half()
    elif kind == "host":
        M, K, N = case["M"], case["K"], case["N"]
        qw, sc, zr = _quantised(gen, N, K, 128, case["act"], "u4")
        st["layer"] = qf.W4A16Linear(qw, sc, zr, prepack=case["layout"] == "tiled")
        st["x"] = torch.randn(M, K, device=dev, generator=gen).to(_DT[case["act"]]).cpu().pin_memory()
        st["out"] = torch.empty(M, N, dtype=_DT[case["act"]], pin_memory=True)
    elif kind in ("step", "token"):
        cfg = {"hidden": case["hidden"], "kv": case["kv"], "ffn": case["ffn"], "layers": case["layers"]}
        st["stack"] = DecodeLinearStack(cfg, case["batch"], torch.bfloat16, dev, seed=seed, fuse=case["fused"],
                                        epilogues=case["fused"])
        # There are no norms between these linears and SiLU * mul grows with the square of its input: a small hidden state
        # and a small attention output keep the residual stream of a deep stack finite.
        h = (torch.randn(case["batch"], case["hidden"], device=dev, generator=gen) * 0.015625).to(torch.bfloat16)
        st["stack"].buf["attn"].mul_(0.015625)
        if kind == "step":
            st["h"] = h
            st["graph"] = st["stack"].capture()
            # what the last layer leaves behind: "down" is the hidden state
            st["results"] = (["qkv", "o", "act", "down"] if case["fused"] else ["q", "k", "v", "o", "gate", "up", "down"])
        else:
            st["h"] = h.cpu().pin_memory()
            st["out"] = torch.empty_like(st["h"], pin_memory=True)
            st["stack"].step_host(st["h"], st["out"])  # captures the step
    elif kind == "unpack":
        st["packed"] = torch.randint(-128, 128, (case["rows"], case["cols"]), dtype=torch.int8, device=dev, generator=gen)
    elif kind == "dequant":
        st["qw"], st["sc"], st["zr"] = _quantised(gen, case["N"], case["K"], case["group"], case["act"], case["zeros"])
        st["group"] = case["group"]
    else:
        st["w"] = (torch.randn(case["N"], case["K"], device=dev, generator=gen) * 0.02).to(_DT[case["act"]])
        st["group"], st["symmetric"], st["layout"] = case["group"], case["symmetric"], case["layout"]
    return st


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "linear":
        if "slab" in st:
            return qf.w4a16_linear(st["x"], st["slab"], out_dtype=st["out_dtype"], epilogue=st["epilogue"],
                                   residual=st["residual"])
        layer = st["layer"]
        if st["epilogue"] == qf.QF_EPI_NONE:
            return layer(st["x"], out_dtype=st["out_dtype"])
        return qf.w4a16_linear(st["x"], layer.qweight, layer.scales, layer.zeros, layer.group_size, layer.zero_const,
                               out_dtype=st["out_dtype"], weight_layout=layer.weight_layout, epilogue=st["epilogue"],
                               residual=st["residual"])
    if kind == "gemv":
        return qf.gemv_int4(st["x"], st["w"], st["scale"], st["zero"])
    if kind == "host":
        return st["layer"].forward_host(st["x"], st["out"])
    if kind == "step":
        stack = st["stack"]
        stack.buf["h_in"].copy_(st["h"])
        st["graph"].replay()
        return {name: stack.buf[name] for name in st["results"]}
    if kind == "token":
        return st["stack"].step_host(st["h"], st["out"])
    if kind == "unpack":
        return qf.unpack_int4(st["packed"])
    if kind == "dequant":
        return qf.dequant_w4(st["qw"], st["sc"], st["zr"], group_size=st["group"])
    codes, scales, zeros = quantize_w4(st["w"], st["group"], st["symmetric"])
    qweight = qf.pack_int4(codes)
    qzeros = qf.pack_zeros_u4(zeros) if zeros is not None else None
    if st["layout"] == "slab":
        ready = qf.prepack_gemv_slab(qweight, scales, qzeros, group_size=st["group"]).blob
    else:
        ready = qf.prepack_w4(qweight, layout=_LAYOUT["tiled"])
    return {"qweight": qweight, "scales": scales, "qzeros": qzeros, "ready": ready}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far results may be apart
# ------------------------------------------------------------------------------------------------
def _zero_bytes(zeros, G, N):
    return {"u4": G * N // 2, "i8": G * N, "const": 0}[zeros]


def work(case):
    kind = case["kind"]
    if kind in ("linear", "gemv", "host"):
        M, K, N = case["M"], case["K"], case["N"]
        G = K // case["group"] if kind == "linear" else 1 if kind == "gemv" else K // 128
        zeros = case["zeros"] if kind == "linear" else "i8" if kind == "gemv" else "u4"
        cols = N // 2 if case.get("epilogue") == "silu" else N
        ob = 4 if case.get("out") == "f32" else 2
        nbytes = K * N // 2 + G * N * 2 + _zero_bytes(zeros, G, N) + M * K * 2 + M * cols * ob
        if case.get("epilogue") == "residual":
            nbytes += M * N * ob
        return {"bytes": nbytes, "flops": 2 * M * K * N}
    if kind in ("step", "token"):
        H, KV, F, M = case["hidden"], case["kv"], case["ffn"], case["batch"]
        gate_up = linear_bytes(M, H, 2 * F, out_cols=F) if case["fused"] else 2 * linear_bytes(M, H, F)
        layer = 2 * linear_bytes(M, H, H) + 2 * linear_bytes(M, H, KV) + gate_up + linear_bytes(M, F, H)
        macs = 2 * H * H + 2 * H * KV + 3 * H * F
        return {"bytes": layer * case["layers"], "flops": 2 * M * macs * case["layers"]}
    if kind == "unpack":
        return {"bytes": 3 * case["rows"] * case["cols"], "flops": 0}
    K, N = case["K"], case["N"]
    G = K // case["group"]
    if kind == "dequant":
        return {"bytes": K * N // 2 + G * N * 2 + _zero_bytes(case["zeros"], G, N) + 2 * K * N, "flops": 0}
    zeros = 0 if case["symmetric"] else G * N // 2
    ready = (N // 64) * (K // 128) * 4352 if case["layout"] == "slab" else K * N // 2
    return {"bytes": 2 * K * N + K * N // 2 + G * N * 2 + zeros + ready, "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("unpack", "dequant", "convert"):
        return "exact"  # codes, and one prescribed rounding per weight or scale
    if kind in ("step", "token"):
        return {"rel": 1e-2}  # bf16 hidden states, rounded after every linear
    out = case["out"] if kind == "linear" else "f16" if kind == "gemv" else case["act"]
    # f32: sums of up to 28672 products in another order; f16 and bf16: one rounding of the output
    return {"f32": {"rel": 5e-5}, "f16": {"rel": 1e-3}, "bf16": {"rel": 1e-2}}[out]
