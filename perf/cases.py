"""The work that users of cpu_ops_b200 have it do, as a set of timed cases.

A case is a dict of plain values: the operand formats, the problem size, the layouts and the
epilogue of one GEMM, how many weight matrices one pass goes through, and how the caller
issues the call.  ``listed()`` gives the fixed ones, ``draw(rng)`` further ones of the same
ranges; ``prepare`` / ``run`` / ``work`` / ``tolerance`` say how one is set up, what one
pass is, what it cannot do without, and how far two correct results may be apart.

``call`` is one of
  ``queued``  device tensors, descriptor kept, enqueued on torch's current stream: what a
              serving or training loop does;
  ``plain``   device tensors, the operator called with its Arguments, synchronous: the
              default of the Python API;
  ``host``    numpy arrays, the operator called as a program written for the CPU library
              calls it; copies in and out are part of the call.
"""
from __future__ import annotations

import math

import torch

import cpu_ops_b200 as c

FORMATS = {"e4m3": c.fp8e4m3_t, "e5m2": c.fp8e5m2_t, "e2m1": c.fp4e2m1_t}
# E8M0 exponent from which a format's scales are drawn when nothing else is said: products of
# two operands so scaled sum up to values around one, as activations are before a SiLU or GELU.
UNIT_SCALE = {"e4m3": 114, "e5m2": 108, "e2m1": 120, "u8": 0, "s8": 0}


def _case(name, a, b, m, n, k, **options):
    case = {"a": a, "b": b, "m": m, "n": n, "k": k,
            "a_row_major": True, "b_row_major": a == "u8", "c_row_major": True, "pad": 0,
            "alpha": 1.0, "beta": 0.0, "chain": "", "weights": 1, "call": "queued",
            "scale_a": UNIT_SCALE[a], "scale_b": UNIT_SCALE[b], "scale_span": 6}
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest call: one 256^3 tile set through the default, synchronous operator.
        _case("int8_256", "u8", "s8", 256, 256, 256, beta=1.0, call="plain"),
        # A small projection of a serving batch with its bias and activation fused.
        _case("mxfp8_bias_silu_512", "e4m3", "e4m3", 512, 2048, 1024, chain="bias_silu"),
        # Decode: one token against the up-projections of eight layers (weights cold in L2).
        _case("mxfp4_decode_m1", "e2m1", "e2m1", 1, 14336, 4096, weights=8, scale_a=124, scale_b=124),
        # Decode of a batch of 32 against eight down-projections: few weight rows, long k.
        _case("mxfp8_decode_m32", "e4m3", "e4m3", 32, 4096, 14336, weights=8),
        # The configured int8 GEMM (C is read and added).
        _case("int8_2048", "u8", "s8", 2048, 2048, 2048, beta=1.0),
        # The configured MX fp8 GEMM, the benchmark's default workload.
        _case("mxfp8_4096", "e4m3", "e4m3", 4096, 4096, 4096, beta=0.5, scale_a=122, scale_b=122,
              scale_span=10),
        # MX fp4 at the size of a large prefill.
        _case("mxfp4_8192", "e2m1", "e2m1", 8192, 8192, 8192),
        # The configured int8 GEMM with the fused bias -> ReLU -> clamp chain.
        _case("int8_8192_chain", "u8", "s8", 8192, 8192, 16384, chain="bias_relu_clamp"),
        # The largest configured problem.
        _case("mx_e5m2_16384", "e5m2", "e5m2", 16384, 16384, 16384, scale_a=120, scale_b=120,
              scale_span=14),
        # Odd sizes with leading dimensions of dim + 3, as the reference's own tests pass them.
        _case("int8_ragged", "u8", "s8", 1999, 3001, 1777, beta=1.0, pad=3),
        # A small output with a deep k: the shape split-k exists for.
        _case("int8_deep_k", "u8", "s8", 192, 320, 16384, b_row_major=False),
        # A program of the CPU library, relinked: everything in pageable host memory.
        _case("int8_host_1024", "u8", "s8", 1024, 1024, 1024, beta=1.0, call="host"),
    ]


def _log_int(rng, lo, hi, step=1):
    """Spread over the logarithm; every third value (where `step` allows) stays ragged."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.35:
        grain = step
    else:
        grain = max(step, 16 if x < 256 else 64 if x < 2048 else 256)
    return max(lo, min(hi, int(round(x / grain)) * grain or grain))


def draw(rng):
    family = rng.choice(["decode", "decode", "mx", "mx", "mx", "int8", "int8", "int8", "deep_k", "host"])
    fmt = rng.choice(["e4m3", "e5m2", "e2m1"])
    beta = rng.choice([0.0, 0.0, 1.0])
    if family == "decode":
        return _case(None, fmt, fmt, _log_int(rng, 1, 64), _log_int(rng, 1024, 16384, 8),
                     _log_int(rng, 1024, 14336, 512), weights=8,
                     chain=rng.choice(["", "", "bias"]))
    if family == "mx":
        other = rng.choice([fmt, fmt, fmt, "e2m1"])  # now and then 4-bit weights under 8-bit inputs
        return _case(None, fmt, other, _log_int(rng, 128, 8192), _log_int(rng, 256, 8192, 4),
                     _log_int(rng, 256, 8192, 32), beta=beta,
                     chain=rng.choice(["", "", "bias", "bias_silu", "bias_gelu"]),
                     call=rng.choice(["queued", "queued", "queued", "plain"]))
    if family == "int8":
        return _case(None, "u8", "s8", _log_int(rng, 128, 8192), _log_int(rng, 128, 8192),
                     _log_int(rng, 128, 8192), beta=beta, a_row_major=rng.random() < 0.75,
                     b_row_major=rng.random() < 0.5, c_row_major=rng.random() < 0.75,
                     pad=rng.choice([0, 0, 0, 3]), chain=rng.choice(["", "", "bias", "bias_relu_clamp"]),
                     call=rng.choice(["queued", "queued", "queued", "plain"]))
    if family == "deep_k":
        kind = rng.choice(["u8", "u8", fmt])
        return _case(None, kind, "s8" if kind == "u8" else kind, _log_int(rng, 16, 512),
                     _log_int(rng, 128, 512, 4), _log_int(rng, 4096, 32768, 256), beta=beta,
                     b_row_major=kind == "u8" and rng.random() < 0.5)
    kind = rng.choice(["u8", "u8", fmt])
    return _case(None, kind, "s8" if kind == "u8" else kind, _log_int(rng, 256, 2048),
                 _log_int(rng, 256, 2048, 4), _log_int(rng, 256, 2048, 32), beta=beta, call="host")


# ---- operands ---------------------------------------------------------------------------


def _elements(fmt, rows, ld, g, dev):
    """`rows` rows of `ld` MX elements: every finite code equally likely."""
    per_byte = 2 if fmt == "e2m1" else 1
    x = torch.randint(0, 256, (rows, ld // per_byte), dtype=torch.uint8, device=dev, generator=g)
    if fmt == "e4m3":    # 0x7F and 0xFF are NaN
        x = torch.where((x & 0x7F) == 0x7F, x & 0xFE, x)
    elif fmt == "e5m2":  # an all-ones exponent is Inf or NaN
        x = torch.where((x & 0x7C) == 0x7C, x & 0xFB, x)
    return x


def prepare(case, seed):
    is_int = case["a"] == "u8"
    host = case["call"] == "host"
    dev = torch.device("cpu") if host else torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    as_user = (lambda t: t.numpy()) if host else (lambda t: t)
    options = {} if case["call"] != "queued" else {
        "stream": torch.cuda.current_stream().cuda_stream, "asynchronous": True}
    layout = lambda row_major: c.RowMajor if row_major else c.ColumnMajor  # noqa: E731
    if is_int:
        op = c.GemmU8S8S32(layout(case["a_row_major"]), layout(case["b_row_major"]),
                           layout(case["c_row_major"]), **options)
    else:
        op = c.GemmMx(FORMATS[case["a"]], FORMATS[case["b"]], layout(case["c_row_major"]), **options)

    state = {"op": op, "calls": [], "out": [], "keep": []}
    number = torch.int32 if is_int else torch.float32
    c_rows, c_cols = (m, n) if case["c_row_major"] else (n, m)
    ldc = c_cols + pad
    groups = (k + 31) // 32

    def scales(lowest, rows):
        return torch.randint(lowest, lowest + case["scale_span"] + 1, (rows, groups), dtype=torch.uint8,
                             device=dev, generator=g)

    # one set of activations, `weights` weight matrices
    if is_int:
        a_rows, a_cols = (m, k) if case["a_row_major"] else (k, m)
        A = torch.randint(0, 256, (a_rows, a_cols + pad), dtype=torch.uint8, device=dev, generator=g)
        ref_a = c.TensorRef(as_user(A), a_cols + pad)
    else:
        A = _elements(case["a"], m, k, g, dev)
        SA = scales(case["scale_a"], m)
        ref_a = c.MxTensorRef(as_user(A), as_user(SA), k, groups)
        state["keep"].append(SA)
    state["keep"].append(A)
    for _ in range(case["weights"]):
        if is_int:
            b_rows, b_cols = (k, n) if case["b_row_major"] else (n, k)
            B = torch.randint(-128, 128, (b_rows, b_cols + pad), dtype=torch.int8, device=dev, generator=g)
            ref_b = c.TensorRef(as_user(B), b_cols + pad)
        else:
            B = _elements(case["b"], n, k, g, dev)
            SB = scales(case["scale_b"], n)
            ref_b = c.MxTensorRef(as_user(B), as_user(SB), k, groups)
            state["keep"].append(SB)
        D = torch.zeros((c_rows, ldc), dtype=number, device=dev)
        C = D  # never read when beta == 0, but it has to be there
        if case["beta"] != 0:
            if is_int:
                C = torch.randint(-1000, 1001, (c_rows, ldc), dtype=number, device=dev, generator=g)
            else:
                C = torch.randn((c_rows, ldc), dtype=number, device=dev, generator=g)
        chain = []
        if case["chain"]:
            if is_int:
                bias = torch.randint(-(1 << 15), (1 << 15) + 1, (n,), dtype=number, device=dev, generator=g)
            else:
                bias = torch.randn((n,), dtype=number, device=dev, generator=g)
            state["keep"].append(bias)
            chain.append(c.BiasAdd(as_user(bias)))
            if case["chain"] == "bias_relu_clamp":
                chain += [c.Relu(), c.Clamp(0, 1 << 20)]
            elif case["chain"] == "bias_silu":
                chain.append(c.Silu())
            elif case["chain"] == "bias_gelu":
                chain.append(c.Gelu())
        epilogue = c.LinearCombinationFused(int(case["alpha"]) if is_int else case["alpha"],
                                            int(case["beta"]) if is_int else case["beta"], chain)
        args = op.Arguments(c.GemmCoord(m, n, k), ref_a, ref_b, c.TensorRef(as_user(C), ldc),
                            c.TensorRef(as_user(D), ldc), epilogue)
        state["calls"].append(op.describe(args) if case["call"] == "queued" else args)
        state["keep"] += [B, C, D]
        state["out"].append(as_user(D)[:, :c_cols])
    state["issue"] = op.run if case["call"] == "queued" else op
    return state


def run(state):
    issue = state["issue"]
    for call in state["calls"]:
        if issue(call) != c.Status.kSuccess:
            raise RuntimeError(c._capi.last_error())
    return state["out"]


# ---- what a pass cannot do without, and how far results may be apart ---------------------


def work(case):
    m, n, k, w = case["m"], case["n"], case["k"], case["weights"]
    width = {"e2m1": 0.5}
    activations, weights = m * k * width.get(case["a"], 1.0), n * k * width.get(case["b"], 1.0)
    if case["a"] != "u8":
        activations += m * ((k + 31) // 32)
        weights += n * ((k + 31) // 32)
    outputs = m * n * 4 * (2 if case["beta"] != 0 else 1)
    if case["chain"]:
        outputs += n * 4
    return {"bytes": activations + w * (weights + outputs), "flops": 2.0 * m * n * k * w}


def tolerance(case):
    if case["a"] == "u8":
        return "exact"
    # Sums in f32.  Against a float64 product of the same operands, and between k summed in one
    # piece and in 3 or 8 slices, e4m3 and e5m2 results were seen 2.6e-7 apart at k = 384,
    # 2.4e-6 at 4096 and 7.7e-6 at 14336 and 16384 (growing with k, as a running f32 sum's
    # rounding does), SiLU and GELU adding up to 4e-7.  Products and partial sums of e2m1
    # operands fit f32 whole at these sizes: only the epilogue rounds (2.5e-8 seen).
    if case["a"] == case["b"] == "e2m1":
        return {"rel": 1e-6}
    return {"rel": 2e-6 + 1e-9 * case["k"]}
