"""What a user of this library has it do: the cases its speed is measured on.

Every case is one pass through the public entry points on device-resident tensors, as a model's forward pass calls them:
single projections (`matmul_q4*`, `matmul_q2` / `matmul_q1` and their `_mopa` forms, the `Gemm` builder), the gated MLP
block (`Mlp.accumulate`) and whole transformer layers (`Block.accumulate` on a KV cache).  Weights, caches and output
buffers are what a program holds between calls; inputs and weights are synthetic, made on the GPU from the seed, with the
distributions quantised language-model weights and normalised activations have.
"""
import math

import numpy as np
import torch

import sme_gemm_b200 as sg


def listed():
    return [
        # decode: one token through a 4096-wide projection
        {"name": "q4_decode_1", "kind": "q4", "m": 1, "n": 4096, "k": 4096, "block": 32, "dtype": "f16", "ep": "none", "affine": False},
        # decode of eight sequences at once (a serving batch), bf16 activations, the up projection of a 4096-wide model
        {"name": "q4_decode_8_bf16", "kind": "q4", "m": 8, "n": 14336, "k": 4096, "block": 32, "dtype": "bf16", "ep": "none", "affine": False},
        # prefill: a prompt of 512 tokens, bf16, with the projection's bias, activation and clamp in the store
        {"name": "q4_prefill_512_bf16", "kind": "q4", "m": 512, "n": 14336, "k": 4096, "block": 32, "dtype": "bf16", "ep": "bias_silu_clamp",
         "affine": False},
        # a short prompt through a matrix of no round size: ragged rows, columns and depth
        {"name": "q4_ragged_77", "kind": "q4", "m": 77, "n": 2051, "k": 1500, "block": 32, "dtype": "f16", "ep": "bias_gelu", "affine": False},
        # decode on ternary weights (BitNet b1.58 style), int8 activations
        {"name": "q2_decode_1", "kind": "lowbit", "bits": 2, "m": 1, "n": 11008, "k": 4096, "block": 256, "ep": "none", "mopa": False},
        # decode of eight sequences on 1-bit weights (Q1_0), with a per-column scale and bias
        {"name": "q1_decode_8", "kind": "lowbit", "bits": 1, "m": 8, "n": 14336, "k": 4096, "block": 128, "ep": "scale_bias", "mopa": False},
        # a 512-token prompt on 1-bit weights with int8 activations
        {"name": "q1_prefill_512", "kind": "lowbit", "bits": 1, "m": 512, "n": 14336, "k": 4096, "block": 128, "ep": "none", "mopa": False},
        # the SiLU-gated MLP block 4096 / 14336 at one token and at a 256-token batch
        {"name": "mlp_1", "kind": "mlp", "m": 1, "d": 4096, "f": 14336},
        {"name": "mlp_256", "kind": "mlp", "m": 256, "d": 4096, "f": 14336},
        # one generated character through the six 384-wide layers of a GPT-2 style character model: the smallest calls
        {"name": "char_model_step", "kind": "layers", "layers": 6, "d": 384, "heads": 6, "kv_heads": 6, "hd": 64, "f": 1536, "gated": False,
         "rows": 1, "past": 127},
        # one generated token through a 4096-wide grouped-query layer with 1023 cached positions
        {"name": "layer_decode_1", "kind": "layers", "layers": 1, "d": 4096, "heads": 32, "kv_heads": 8, "hd": 128, "f": 14336, "gated": True,
         "rows": 1, "past": 1023},
        # the second 512-token chunk of a 1024-token prompt through the same layer
        {"name": "layer_prefill_512", "kind": "layers", "layers": 1, "d": 4096, "heads": 32, "kv_heads": 8, "hd": 128, "f": 14336, "gated": True,
         "rows": 512, "past": 512},
    ]


# ------------------------------------------------------------------------------------------------ more of the same ranges

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A matrix dimension: mostly the multiples of 128 that models have, else anything."""
    v = _log(rng, lo, hi)
    return max(lo // 128, round(v / 128)) * 128 if rng.random() < 0.6 else v


def _rows(rng, most=512):
    return min(most, rng.choice([1, 1, _log(rng, 2, 16), _log(rng, 17, 512), _log(rng, 17, 512)]))


def draw(rng):
    kind = rng.choice(["q4", "q4", "q4", "lowbit", "lowbit", "dense", "mlp", "layers", "layers"])
    if kind in ("q4", "lowbit", "dense"):
        m, n, k = _rows(rng), _size(rng, 256, 14336), _size(rng, 256, 8192)
        if n * k > 4096 * 14336:
            k = 4096
        if kind == "q4":
            # Q4_1 files: weights with a minimum per block
            affine = rng.random() < 0.15
            if affine:
                n, k = min(n, 4096), min(k, 2048)
            return {"kind": kind, "m": m, "n": n, "k": k, "block": rng.choice([32, 32, 32, 64, 128]), "dtype": rng.choice(["f16", "f16", "bf16"]),
                    "ep": rng.choice(["none", "none", "bias_gelu", "bias_silu_clamp"]), "affine": affine}
        if kind == "lowbit":
            return {"kind": kind, "bits": rng.choice([1, 2]), "m": m, "n": n, "k": k, "block": rng.choice([64, 128, 128, 256]),
                    "ep": rng.choice(["none", "scale_bias"]), "mopa": rng.random() < 0.3}
        # unquantised weights: the embedding and head projections of small models
        return {"kind": kind, "m": m, "n": min(n, 4096), "k": min(k, 2048), "dtype": rng.choice(["f16", "bf16"]), "ep": rng.choice(["none", "bias_gelu"])}
    if kind == "mlp":
        d = max(2, round(_log(rng, 512, 4096) / 128)) * 128
        return {"kind": kind, "m": _rows(rng, 256), "d": d, "f": min(14336, rng.choice([d * 3, d * 7 // 2, round(d * 8 / 3 / 64) * 64]))}
    if rng.random() < 0.4:      # GPT-2 style: layer norm, plain MLP with GELU, all heads with keys of their own
        hd = rng.choice([32, 64])
        heads = rng.randint(3, 12)
        return {"kind": kind, "layers": rng.randint(2, 6), "d": heads * hd, "heads": heads, "kv_heads": heads, "hd": hd, "f": 4 * heads * hd, "gated": False,
                "rows": rng.choice([1, _log(rng, 2, 256)]), "past": rng.randint(0, 256)}
    hd = rng.choice([64, 128])  # Llama style: RMS norm, gated MLP, grouped queries
    kv_heads = rng.choice([2, 4, 8])
    group = rng.choice([1, 2, 4]) if hd == 128 else rng.choice([2, 3, 4, 8])
    heads = kv_heads * group
    d = heads * hd
    rows = rng.choice([1, _log(rng, 2, 16), _log(rng, 17, 512)])
    past = rng.randint(0, 512) if rows > 16 else _log(rng, 16, 4096)
    return {"kind": kind, "layers": 1, "d": d, "heads": heads, "kv_heads": kv_heads, "hd": hd, "f": d * 7 // 2, "gated": True, "rows": rows, "past": past}


# ------------------------------------------------------------------------------------------------ what a program holds

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _uniform(g, lo, hi, *shape, dtype=torch.float32):
    return (torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo).to(dtype)


def _bits16(t):
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def _pack(codes, bits):
    """Small integers, in order, several to a byte (the first one lowest)."""
    per = 8 // bits
    flat = torch.nn.functional.pad(codes.reshape(-1), (0, -codes.numel() % per)).view(-1, per)
    out = flat[:, 0].clone()
    for i in range(1, per):
        out |= flat[:, i] << (bits * i)
    return out.cpu().numpy()


def _q4(g, n, k, block=32, affine=False):
    """N(0, 0.02) weights in 4 bits per value: an f16 scale (the block's largest value over -8) per column and K-block,
    or a scale and a minimum."""
    nbk = -(-k // block)
    w = _normal(g, k, n, std=0.02)
    pad = torch.nn.functional.pad(w, (0, 0, 0, nbk * block - k)).view(nbk, block, n)
    if affine:
        lo = pad.amin(1)
        scale = ((pad.amax(1) - lo) / 15).half()
        mins = (lo + 8 * scale.float()).half()
    else:
        big = pad.gather(1, pad.abs().argmax(1, keepdim=True))[:, 0]
        scale, mins = (big / -8).half(), torch.zeros_like(big).half()
    s = scale.float()
    inv = torch.where(s == 0, torch.zeros_like(s), 1 / s)
    codes = ((pad - mins.float()[:, None]) * inv[:, None]).round_().clamp_(-8, 7).to(torch.int8).view(nbk * block, n)[:k]
    quants = _pack((codes & 15).view(torch.uint8), 4)
    return sg.Q4Weights.with_params(quants, _bits16(scale.t()).reshape(-1), _bits16(mins.t()).reshape(-1) if affine else None, n, k,
                                    sg.Q4Params(block).affine() if affine else sg.Q4Params(block))


def _lowbit(g, bits, n, k, block):
    nbk = -(-k // block)
    if bits == 2:               # {-1, 0, +1}, equally likely: codes 0, 1, 2 of the ternary codebook
        codes = _pack(torch.randint(0, 3, (k * n,), generator=g, device="cuda", dtype=torch.uint8), 2)
        return sg.Q2Weights.new(codes, _bits16(_uniform(g, 0.01, 0.05, n * nbk, dtype=torch.float16)), n, k, sg.Q2Params(block))
    signs = _pack(torch.randint(0, 2, (k * n,), generator=g, device="cuda", dtype=torch.uint8), 1)
    return sg.Q1Weights.new(signs, _bits16(_uniform(g, 0.005, 0.03, n * nbk, dtype=torch.float16)), sg.WeightLayout.OutIn, n, k, block)


def _layer(g, c):
    d, hd, gated = c["d"], c["hd"], c["gated"]
    qkv = sg.Linear.from_q4(_q4(g, (c["heads"] + 2 * c["kv_heads"]) * hd, d))
    attn = sg.SelfAttention.new(qkv, sg.Linear.from_q4(_q4(g, d, c["heads"] * hd)), c["heads"], c["kv_heads"], hd)
    weight = lambda: _uniform(g, 0.5, 1.5, d).cpu().numpy()  # noqa: E731
    if gated:
        mlp = sg.Mlp.gated(sg.GatedLinear(sg.Linear.from_q4(_q4(g, 2 * c["f"], d)), sg.Gate.Silu), sg.Linear.from_q4(_q4(g, d, c["f"])))
        return sg.Block.new(sg.Norm.rms(weight(), 1e-5), attn, sg.Norm.rms(weight(), 1e-5), mlp)
    mlp = sg.Mlp.new(sg.Linear.from_q4(_q4(g, c["f"], d)), sg.Gate.Gelu, sg.Linear.from_q4(_q4(g, d, c["f"])))
    bias = lambda: _normal(g, d, std=0.1).cpu().numpy()  # noqa: E731
    return sg.Block.new(sg.Norm.layer(weight(), bias(), 1e-5), attn, sg.Norm.layer(weight(), bias(), 1e-5), mlp)


def prepare(case, seed):
    g, c, kind = _gen(seed), case, case["kind"]
    s = {"case": c}
    if kind in ("q4", "lowbit", "dense"):
        dtype = torch.bfloat16 if c.get("dtype") == "bf16" else torch.float16
        m, n, k = c["m"], c["n"], c["k"]
        s["a"] = _normal(g, m, k, dtype=dtype)
        s["c"] = torch.empty((m, n), dtype=dtype, device="cuda")
        s["bias"] = _normal(g, n, std=0.1, dtype=dtype)
        s["scale"] = _uniform(g, 0.5, 1.5, n, dtype=dtype)
        if kind == "q4":
            s["w"] = _q4(g, n, k, c["block"], c["affine"])
        elif kind == "lowbit":
            s["w"] = _lowbit(g, c["bits"], n, k, c["block"])
        else:
            w = _bits16(_normal(g, k, n, std=0.02, dtype=dtype))
            s["w"] = sg.prepack_bf16(w, n, k) if c["dtype"] == "bf16" else sg.prepack_f16(w.view(np.float16), n, k)
    elif kind == "mlp":
        m, d, f = c["m"], c["d"], c["f"]
        s["x"] = _normal(g, m, d, dtype=torch.float16)
        s["y"] = _normal(g, m, d)
        s["mlp"] = sg.Mlp.gated(sg.GatedLinear(sg.Linear.from_q4(_q4(g, 2 * f, d)), sg.Gate.Silu), sg.Linear.from_q4(_q4(g, d, f)))
    else:
        s["x"] = _normal(g, c["rows"], c["d"])
        s["blocks"] = [_layer(g, c) for _ in range(c["layers"])]
        s["caches"] = [b.cache(c["past"] + c["rows"]) for b in s["blocks"]]
        for cache in s["caches"]:
            if c["past"]:
                cache.extend(_normal(g, c["past"], cache.row_len(), dtype=torch.float16), _normal(g, c["past"], cache.row_len(), dtype=torch.float16))
    return s


# ------------------------------------------------------------------------------------------------ one pass

def _graph(s, dtype):
    ep = s["case"]["ep"]
    if ep == "bias_gelu":
        return sg.Epilogue(dtype).add_col(s["bias"]).gelu()
    if ep == "bias_silu_clamp":
        return sg.Epilogue(dtype).add_col(s["bias"]).silu().clamp(-6.0, 6.0)
    if ep == "scale_bias":
        return sg.Epilogue(dtype).mul_col(s["scale"]).add_col(s["bias"])
    return None


def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "q4":
        bf16, ep = c["dtype"] == "bf16", _graph(s, c["dtype"])
        if ep is None:
            (sg.matmul_q4_bf16 if bf16 else sg.matmul_q4)(s["a"], s["w"], s["c"], c["m"])
        else:
            (sg.matmul_q4_bf16_ep if bf16 else sg.matmul_q4_ep)(s["a"], s["w"], s["c"], c["m"], ep)
        return s["c"]
    if kind == "lowbit":
        name = "matmul_q%d%s" % (c["bits"], "_mopa" if c["mopa"] else "")
        ep = _graph(s, "f16")
        if ep is None:
            getattr(sg, name)(s["a"], s["w"], s["c"], c["m"])
        else:
            getattr(sg, name + "_ep")(s["a"], s["w"], s["c"], c["m"], ep)
        return s["c"]
    if kind == "dense":
        gemm = sg.Gemm.new(s["a"], s["w"], c["m"])
        if c["ep"] == "bias_gelu":
            gemm = gemm.add_col(s["bias"]).gelu()
        gemm.run(s["c"])
        return s["c"]
    if kind == "mlp":
        s["mlp"].accumulate(s["x"], s["y"], c["m"])
        return s["y"]
    x = s["x"].clone()                                   # the embedded tokens: the residual stream the layers add to
    for block, cache in zip(s["blocks"], s["caches"]):
        cache.truncate(c["past"])                        # the positions of this pass come after the cached ones
        block.accumulate(x, cache, c["rows"])
    return {"x": x, "keys": [cache.keys() for cache in s["caches"]], "values": [cache.values() for cache in s["caches"]]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def _q4_bytes(n, k, block=32, affine=False):
    return n * k / 2 + (4 if affine else 2) * n * -(-k // block)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("q4", "lowbit", "dense"):
        m, n, k = c["m"], c["n"], c["k"]
        weights = (_q4_bytes(n, k, c["block"], c["affine"]) if kind == "q4" else
                   n * k * c["bits"] / 8 + 2 * n * -(-k // c["block"]) if kind == "lowbit" else 2 * n * k)
        operands = {"none": 0, "scale_bias": 2}.get(c["ep"], 1) * 2 * n
        return {"bytes": weights + 2 * m * (n + k) + operands, "flops": 2 * m * n * k}
    if kind == "mlp":
        m, d, f = c["m"], c["d"], c["f"]
        return {"bytes": _q4_bytes(2 * f, d) + _q4_bytes(d, f) + 2 * m * d + 8 * m * d, "flops": 6 * m * d * f}
    d, f, rows, past, q_len, kv_len = c["d"], c["f"], c["rows"], c["past"], c["heads"] * c["hd"], c["kv_heads"] * c["hd"]
    up = 2 * f if c["gated"] else f
    weights = _q4_bytes(q_len + 2 * kv_len, d) + _q4_bytes(d, q_len) + _q4_bytes(up, d) + _q4_bytes(d, f)
    macs = rows * (d * (q_len + 2 * kv_len) + d * q_len + d * up + d * f) + 2 * q_len * (rows * past + rows * (rows + 1) // 2)
    norms = (8 if c["gated"] else 16) * d
    return {"bytes": c["layers"] * (weights + norms + 4 * kv_len * (past + rows)) + 8 * rows * d, "flops": 2 * c["layers"] * macs}


def tolerance(case):
    if case["kind"] == "lowbit" and not case["mopa"]:
        return "exact"                                   # int8 activations, int32 block sums, folded in the order of the blocks
    # about four times the distance of the listed and some drawn cases from the same chain in 64 bits without roundings:
    # bf16 2.6e-3 (largest 8e-3), f16 projections 6e-4 (2.4e-3), MLP blocks and layers 9e-4 (3.3e-3)
    if case.get("dtype") == "bf16":
        return {"rel": 1e-2, "max": 3e-2}
    return {"rel": 4e-3, "max": 1.4e-2} if case["kind"] in ("mlp", "layers") else {"rel": 2.5e-3, "max": 1e-2}
