"""The performance cases: what a program that uses this library has it do, through the public entry points.

Five kinds of work, each over the range of sizes the library is used at:

  linear     one bf16 linear layer on device buffers through ``lib.matmul_bf16`` (square, decode-shaped, ragged,
             transposed, with and without bias / ReLU, rows that are not a whole number of 16 bytes)
  mlp        a partition of chained linear layers through the oneDNN-graph API: bf16 or f32, device tensors on the
             caller's stream or host buffers through the synchronous call
  int8       a u8 x s8 partition with zero point, per-channel scales and bias, on device tensors
  attention  fused attention (prefill), with and without a causal mask
  block      the decoder MLP block of the reference's tests (RMSNorms, residuals, SiLU-gated MLP), a partition of 25 ops
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("graph-compiler_b200"))

from gc_b200 import api, lib, partitions  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest call: one layer of benchgc's mlp pattern with every argument in host memory, as the reference's C API is called
        {"name": "layer_host", "kind": "mlp", "batch": 128, "hidden": "512x256", "dtype": "bf16", "where": "host", "constant": False, "bound": False},
        # an f32 graph (the type of the reference's own C-API test), one layer on device tensors
        {"name": "layer_f32", "kind": "mlp", "batch": 512, "hidden": "1024x1024", "dtype": "f32", "where": "device", "constant": False, "bound": False},
        # the benchmark's MLP chain, activations and weights resident on the device
        {"name": "chain_device", "kind": "mlp", "batch": 512, "hidden": "4096x16384x4096x16384x4096", "dtype": "bf16", "where": "device", "constant": False, "bound": False},
        # the same chain served to a host program: pinned activations in and out on every call, constant weights
        {"name": "chain_host", "kind": "mlp", "batch": 512, "hidden": "4096x16384x4096x16384x4096", "dtype": "bf16", "where": "host", "constant": True, "bound": True},
        # an ordinary square GEMM of the sweep, and the largest
        {"name": "gemm_2048", "kind": "linear", "M": 2048, "N": 2048, "K": 2048, "ta": False, "tb": False, "bias": False, "relu": False},
        {"name": "gemm_16384", "kind": "linear", "M": 16384, "N": 16384, "K": 16384, "ta": False, "tb": False, "bias": False, "relu": False},
        # decode: a few rows against a large weight matrix
        {"name": "gemm_decode", "kind": "linear", "M": 16, "N": 28672, "K": 8192, "ta": False, "tb": False, "bias": False, "relu": False},
        # a classifier head: an odd number of outputs, so weight rows of 2002 bytes
        {"name": "gemm_ragged", "kind": "linear", "M": 1000, "N": 1001, "K": 2048, "ta": False, "tb": False, "bias": True, "relu": False},
        # the int8 configuration of the benchmark
        {"name": "int8_layer", "kind": "int8", "M": 1024, "N": 4096, "K": 4096, "zp": 128, "bias": True},
        # attention at the benchmark's size
        {"name": "attention_full", "kind": "attention", "batch": 16, "heads": 32, "seq": 2048, "causal": False},
        # prefill of prompts whose length is no multiple of a tile
        {"name": "attention_causal", "kind": "attention", "batch": 2, "heads": 32, "seq": 3001, "causal": True},
        # the decoder MLP block for 32 tokens
        {"name": "decoder_block", "kind": "block", "batch": 1, "seq": 32, "hidden": 4096, "inter": 11008},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _to(v, step):
    return max(step, (v + step // 2) // step * step)


def _draw_linear(rng):
    rows = rng.choice(["decode", "any", "any"])
    m = _log(rng, 1, 64) if rows == "decode" else _log(rng, 65, 8192)
    n, k = _log(rng, 64, 28672), _log(rng, 64, 16384)
    grain = rng.choice(["tile", "tile", "sixteen_bytes", "sixteen_bytes", "odd"])
    if grain == "tile":
        m, n, k = (m if rows == "decode" else _to(m, 128)), _to(n, 128), _to(k, 64)
    elif grain == "sixteen_bytes":
        n, k = _to(n, 8), _to(k, 8)
    ta = rng.random() < 0.15
    if ta and grain != "odd":
        m = _to(m, 8)
    # odd row lengths are slow to fetch: smaller
    most = 2e10 if grain == "odd" else 4e12
    while 2.0 * m * n * k > most:
        n, k = max(65, n // 2 | (n & 1)), max(65, k // 2 | (k & 1))
        if grain != "odd":
            n, k = _to(n, 8), _to(k, 8)
    return {"kind": "linear", "M": m, "N": n, "K": k, "ta": ta, "tb": rng.random() < 0.4, "bias": rng.random() < 0.6, "relu": rng.random() < 0.4}


def _draw_mlp(rng):
    f32 = rng.random() < 0.25
    host = rng.random() < 0.4
    layers = rng.randint(1, 4)
    batch = _log(rng, 1, 512 if f32 else 2048)
    most = 2048 if f32 else 16384
    widths = []
    for _ in range(layers + 1):
        w = _log(rng, 128, most)
        widths.append(_to(w, rng.choice([8, 64, 128])))
    while sum(2.0 * batch * a * b for a, b in zip(widths, widths[1:])) > (6e9 if f32 else 1e12):
        widths = [_to(max(64, w // 2), 8) for w in widths]
    return {"kind": "mlp", "batch": batch, "hidden": "x".join(map(str, widths)), "dtype": "f32" if f32 else "bf16",
            "where": "host" if host else "device", "constant": host and rng.random() < 0.75, "bound": host and rng.random() < 0.5}


def _draw_int8(rng):
    return {"kind": "int8", "M": _log(rng, 1, 4096), "N": _to(_log(rng, 64, 8192), 16), "K": _to(_log(rng, 64, 8192), 16),
            "zp": rng.choice([0, 3, 128, 128]), "bias": rng.random() < 0.7}


def _draw_attention(rng):
    seq = _log(rng, 64, 8192)
    if rng.random() < 0.5:
        seq = _to(seq, 128)
    units = _log(rng, 1, 512)
    while 4.0 * units * seq * seq * 128 > 1.1e12:
        units = max(1, units // 2)
    heads = math.gcd(units, 32)
    return {"kind": "attention", "batch": units // heads, "heads": heads, "seq": seq, "causal": rng.random() < 0.6}


def _draw_block(rng):
    hidden = _to(_log(rng, 512, 4096), 128)
    return {"kind": "block", "batch": rng.choice([1, 1, 2, 4]), "seq": _log(rng, 1, 512), "hidden": hidden, "inter": _to(int(hidden * rng.uniform(2.0, 3.5)), 64)}


def draw(rng):
    kind = rng.choice([_draw_linear, _draw_linear, _draw_linear, _draw_mlp, _draw_mlp, _draw_mlp, _draw_int8, _draw_attention, _draw_attention, _draw_block])
    return kind(rng)


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device=DEV).mul_(2).sub_(1).to(torch.bfloat16)


def _normal(g, std, dtype, *shape):
    return torch.randn(shape, generator=g, device=DEV).mul_(std).to(dtype)


def _prepare_linear(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    A = _uniform(g, *((K, M) if c["ta"] else (M, K)))
    B = _uniform(g, *((N, K) if c["tb"] else (K, N)))
    bias = _uniform(g, N) if c["bias"] else None
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    return {"kind": "linear", "A": A, "B": B, "bias": bias, "relu": c["relu"], "ta": c["ta"], "tb": c["tb"], "out": out}


def _widths(c):
    return [int(w) for w in c["hidden"].split("x")]


def _prepare_mlp(c, g):
    h, dt = _widths(c), torch.float32 if c["dtype"] == "f32" else torch.bfloat16
    layers = len(h) - 1
    js, ids, out_id = partitions.mlp(c["batch"], h, c["dtype"], [True] * layers, "relu", constant_weights=c["constant"])
    ts = [_normal(g, 1.0, dt, c["batch"], h[0])]
    ts += [_normal(g, (2.0 / h[i]) ** 0.5, dt, h[i], h[i + 1]) for i in range(layers)]
    ts += [_normal(g, 0.1, dt, h[i + 1]) for i in range(layers)]
    out = torch.empty(c["batch"], h[-1], dtype=dt, device=DEV)
    if c["where"] == "host":   # a program that binds its buffers once also pins them
        ts = [torch.empty(t.shape, dtype=dt, pin_memory=c["bound"]).copy_(t) for t in ts]
        out = torch.empty(out.shape, dtype=dt, pin_memory=c["bound"])
    compiler = api.GraphCompiler()
    exe = compiler.compile(js)
    ins, outs = dict(zip(ids, ts)), {out_id: out}
    bound = exe.bind(ins, outs) if c["bound"] else None
    return {"kind": "mlp", "where": c["where"], "compiler": compiler, "exe": exe, "bound": bound, "ins": ins, "outs": outs, "out": out}


def _prepare_int8(c, g):
    M, N, K = c["M"], c["N"], c["K"]
    js, ids, out_id = partitions.quantized_matmul(M, N, K, src_zp=c["zp"], bias=c["bias"])
    ts = [torch.randint(0, 256, (M, K), generator=g, device=DEV, dtype=torch.uint8),
          torch.randint(-127, 128, (K, N), generator=g, device=DEV, dtype=torch.int8),
          torch.rand(N, generator=g, device=DEV) * 0.009 + 0.001]
    if c["bias"]:
        ts.append(torch.rand(N, generator=g, device=DEV) * 2 - 1)
    out = torch.empty(M, N, device=DEV)
    compiler = api.GraphCompiler()
    return {"kind": "int8", "compiler": compiler, "exe": compiler.compile(js), "ins": dict(zip(ids, ts)), "outs": {out_id: out}, "out": out}


def _prepare_attention(c, g):
    shape = (c["batch"], c["heads"], c["seq"], 128)
    q, k, v = (_normal(g, 1.0, torch.bfloat16, *shape) for _ in range(3))
    return {"kind": "attention", "q": q, "k": k, "v": v, "causal": c["causal"], "out": torch.empty_like(q)}


def _prepare_block(c, g):
    b, s, h, i = c["batch"], c["seq"], c["hidden"], c["inter"]
    js, ids, outs = partitions.llama2_mlp(b, s, h, i)
    bf = torch.bfloat16
    t = {"x": _normal(g, 1.0, bf, b, s, h), "wo": _normal(g, h ** -0.5, bf, h, h), "resid": _normal(g, 1.0, bf, b, s, h),
         "g1": (1 + _normal(g, 0.1, torch.float32, h)).to(bf), "w_gate": _normal(g, h ** -0.5, bf, i, h),
         "w_up": _normal(g, h ** -0.5, bf, i, h), "w_down": _normal(g, i ** -0.5, bf, h, i),
         "eps": torch.full((1,), 1e-5, device=DEV), "g2": (1 + _normal(g, 0.1, torch.float32, h)).to(bf)}
    out = [torch.empty(b, s, h, dtype=bf, device=DEV) for _ in outs]
    compiler = api.GraphCompiler()
    return {"kind": "block", "compiler": compiler, "exe": compiler.compile(js), "ins": {ids[k]: v for k, v in t.items()}, "outs": dict(zip(outs, out)), "out": out}


def prepare(case, seed):
    make = {"linear": _prepare_linear, "mlp": _prepare_mlp, "int8": _prepare_int8, "attention": _prepare_attention, "block": _prepare_block}
    return make[case["kind"]](case, _rng(seed))


def run(state):
    s = state
    if s["kind"] == "linear":
        return lib.matmul_bf16(s["A"], s["B"], s["bias"], relu=s["relu"], transpose_a=s["ta"], transpose_b=s["tb"], out=s["out"])
    if s["kind"] == "attention":
        return lib.attention_bf16(s["q"], s["k"], s["v"], 1.0 / math.sqrt(128), s["causal"], out=s["out"])
    if s.get("bound") is not None:
        s["bound"].run()
    elif s.get("where") == "host":
        s["exe"].execute(s["ins"], s["outs"])
    else:
        s["exe"].execute_on_stream(s["ins"], s["outs"])
    return s["out"]


def work(case):
    c = case
    if c["kind"] == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2 * (M * K + K * N + M * N + (N if c["bias"] else 0)), "flops": 2 * M * N * K}
    if c["kind"] == "mlp":
        h, e = _widths(c), 4 if c["dtype"] == "f32" else 2
        weights = sum(a * b + b for a, b in zip(h, h[1:]))
        return {"bytes": e * (c["batch"] * (h[0] + h[-1]) + weights), "flops": sum(2 * c["batch"] * a * b for a, b in zip(h, h[1:]))}
    if c["kind"] == "int8":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": M * K + K * N + 4 * M * N + 4 * N * (2 if c["bias"] else 1), "flops": 2 * M * N * K}
    if c["kind"] == "attention":
        units, s = c["batch"] * c["heads"], c["seq"]
        pairs = s * (s + 1) // 2 if c["causal"] else s * s
        return {"bytes": 4 * 2 * units * s * 128, "flops": 4 * units * pairs * 128}
    t, h, i = c["batch"] * c["seq"], c["hidden"], c["inter"]
    return {"bytes": 2 * (h * h + 3 * h * i + 4 * t * h + 2 * h), "flops": 2 * t * (h * h + 3 * h * i)}


def tolerance(case):
    if case["kind"] == "int8":
        return {"rel": 1e-6, "max": 1e-5}   # exact integer sums, then one f32 multiply and one add
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}   # f32 sums in another order
    return {"rel": 1e-2}                    # bf16 results
