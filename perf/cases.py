"""Performance cases of the prefill path, through the public entry points, on one GPU.

A case is a dict of plain values with a ``kind``:

* ``linear``     ``M4QuantizedLinear.forward``: one quantised projection called from torch code (a decode token, a short
                 prompt, a prompt of any length; the module waits for its result, so a pass is a whole call)
* ``gemm``       ``B200Bridge.dispatch_gemm`` / ``dispatch_gemm_ex`` + ``synchronize``: the same projection on buffers the
                 caller owns, which also takes the planar layouts
* ``swiglu``     ``B200Bridge.dispatch_swiglu`` + ``synchronize``: the fused gate/up half of an MLP block
* ``attention``  ``b200_bridge_dispatch_attention_q8kv``: causal attention over a Q8_0 (or fp16) KV cache, enqueued on the
                 library's stream as a link of a chain; ``pos0`` > 0 is a later chunk of a chunked prefill, or a decode token
* ``layer``      ``TransformerLayerCoordinator.forward``: one decoder layer, enqueued on the library's stream
* ``model``      ``TransformerModel.forward`` + ``synchronize``: token ids to logits

Inputs have the value distributions of ``bench.py`` (projections) and of the reference's layer benchmark (layers and
models: weights small enough that a residual stream stays inside fp16), generated on the GPU from the seed alone.
"""
import torch

from __graft_entry__ import load_package

Q4_0, MLX, Q4_K, TERNARY, VAR_RATE, CODEBOOK = 0, 1, 2, 3, 4, 5
PRISM, MLX_G64, TERNARY_ROW = 7, 100, 101
BLOCK = {Q4_0: (32, 18), MLX: (32, 20), Q4_K: (256, 144), TERNARY: (32, 12), VAR_RATE: (256, 160), CODEBOOK: (256, 144), PRISM: (128, 34)}


def listed():
    return [
        # one decode token through a projection of the 8B shape: the smallest call, all latency and launches
        {"name": "linear_decode", "kind": "linear", "fmt": Q4_0, "M": 1, "K": 4096, "N": 4096},
        # a short prompt: the M=33 row of the router sweep, MLX-style 4-bit
        {"name": "linear_short", "kind": "linear", "fmt": MLX, "M": 33, "K": 4096, "N": 4096},
        # one token more than a tile, and a hidden size that is whole blocks of 32 but not whole super-blocks
        {"name": "linear_odd", "kind": "linear", "fmt": Q4_0, "M": 129, "K": 2080, "N": 1100},
        # the ternary up-projection (one scale per row) at its smaller token count
        {"name": "gemm_ternary_m128", "kind": "gemm", "fmt": TERNARY_ROW, "M": 128, "K": 4096, "N": 14336},
        # the projection the headline number is quoted on
        {"name": "gemm_prefill", "kind": "gemm", "fmt": Q4_0, "M": 2048, "K": 4096, "N": 4096},
        # the fused gate/up half of the 8B MLP block
        {"name": "swiglu_prefill", "kind": "swiglu", "fmt": Q4_K, "M": 2048, "K": 4096, "F": 14336},
        # attention of the 8B layer over a Q8_0 cache, whole prompt at once
        {"name": "attention_prefill", "kind": "attention", "Hq": 32, "Hkv": 8, "D": 128, "M": 2048, "pos0": 0, "kv_fp16": False},
        # the reference's other head size: 32 heads of 64, no grouping
        {"name": "attention_d64", "kind": "attention", "Hq": 32, "Hkv": 32, "D": 64, "M": 2048, "pos0": 0, "kv_fp16": False},
        # a late chunk of a chunked prefill: 256 tokens behind 7936 cached ones
        {"name": "attention_chunk", "kind": "attention", "Hq": 32, "Hkv": 8, "D": 128, "M": 256, "pos0": 7936, "kv_fp16": False},
        # a short prompt through one layer of the 8B shape
        {"name": "layer_short", "kind": "layer", "fmt": Q4_0, "M": 33, "K": 4096, "Hq": 32, "Hkv": 8, "D": 128, "F": 14336},
        # the engine's default configuration, a prompt of odd length
        {"name": "model_default", "kind": "model", "layers": 4, "M": 301, "K": 512, "Hq": 8, "Hkv": 2, "D": 64, "F": 1024, "vocab": 1024},
        # the largest: 2048 tokens through the whole 32-layer model of the 8B shape
        {"name": "model_8b", "kind": "model", "layers": 32, "M": 2048, "K": 4096, "Hq": 32, "Hkv": 8, "D": 128, "F": 14336, "vocab": 128256},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["linear", "linear", "gemm", "swiglu", "attention", "attention", "layer", "model"])
    m = 1 if rng.random() < 0.1 else _log(rng, 2, 2048)
    if kind in ("linear", "gemm"):
        fmts = [Q4_0, MLX, Q4_K, TERNARY, VAR_RATE, CODEBOOK] + ([PRISM, MLX_G64, TERNARY_ROW] if kind == "gemm" else [])
        fmt = rng.choice(fmts)
        k = 256 * _log(rng, 2, 56)
        if fmt == PRISM:
            k = 1024 * _log(rng, 1, 14)
        elif fmt in (Q4_0, MLX, TERNARY) and rng.random() < 0.2:
            k = 32 * _log(rng, 16, 130)
        n = 128 * _log(rng, 4, 112) if rng.random() < 0.7 else _log(rng, 512, 8192)
        return {"kind": kind, "fmt": fmt, "M": m, "K": k, "N": n}
    if kind == "swiglu":
        return {"kind": kind, "fmt": rng.choice([Q4_0, MLX, Q4_K, TERNARY, VAR_RATE, CODEBOOK]), "M": m, "K": 256 * _log(rng, 2, 16), "F": 64 * _log(rng, 16, 224)}
    if kind == "attention":
        hkv, g = rng.choice([(32, 1), (8, 4), (8, 1), (4, 8), (2, 4), (16, 2), (8, 3)])
        past = 0 if rng.random() < 0.5 else _log(rng, 64, 8192)
        return {"kind": kind, "Hq": hkv * g, "Hkv": hkv, "D": rng.choice([64, 128]), "M": m, "pos0": past, "kv_fp16": rng.random() < 0.3}
    if kind == "layer":
        k, hq, hkv, d, f = rng.choice([(4096, 32, 8, 128, 14336), (2048, 32, 32, 64, 8192), (512, 8, 2, 64, 1024), (2048, 16, 8, 128, 5632)])
        return {"kind": kind, "fmt": rng.choice([Q4_0, Q4_0, MLX, TERNARY]), "M": m, "K": k, "Hq": hq, "Hkv": hkv, "D": d, "F": f}
    k, hq, hkv, d, f = rng.choice([(4096, 32, 8, 128, 14336), (2048, 32, 8, 64, 8192), (512, 8, 2, 64, 1024)])
    return {"kind": kind, "layers": rng.choice([2, 4, 8]), "M": m, "K": k, "Hq": hq, "Hkv": hkv, "D": d, "F": f, "vocab": rng.choice([1024, 32000])}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=g)


def _f16(g, n, lo, hi):
    return (torch.rand(n, device="cuda", generator=g) * (hi - lo) + lo).to(torch.float16)


def _raw(t):
    return t.contiguous().view(torch.uint8).reshape(t.numel(), 2)


def _ternary_bytes(g, n):
    """n bytes of four 2-bit codes each: 0, 1, 2 with probability 1/4, 1/2, 1/4 (the sum of two fair bits)."""
    a, b = _bytes(g, n), _bytes(g, n)
    return ((a & 0x55) + (b & 0x55))


def _weights(fmt, n, k, g, shrink=1.0):
    """Packed weights [n][k / block].  ``shrink`` scales the fp16 scale fields (layers and models)."""
    if fmt == MLX_G64:
        sc = _f16(g, n * k // 64, 0.005 * shrink, 0.02 * shrink)
        bi = (-8.0 * sc.float() + (torch.rand(sc.numel(), device="cuda", generator=g) - 0.5) * 0.02 * shrink).to(torch.float16)
        return torch.cat([_bytes(g, n * k // 2), _raw(sc).reshape(-1), _raw(bi).reshape(-1)])
    if fmt == TERNARY_ROW:
        return torch.cat([_ternary_bytes(g, n * k // 4), _raw(_f16(g, n, 0.01 * shrink, 0.05 * shrink)).reshape(-1)])
    block, size = BLOCK[fmt]
    nb = n * k // block
    w = _bytes(g, nb, size)
    if fmt == Q4_0:
        w[:, 0:2] = _raw(_f16(g, nb, 0.005 * shrink, 0.02 * shrink))
    elif fmt == MLX:
        sc = _f16(g, nb, 0.005 * shrink, 0.02 * shrink)
        w[:, 0:2] = _raw(sc)
        w[:, 2:4] = _raw((-8.0 * sc.float() + (torch.rand(nb, device="cuda", generator=g) - 0.5) * 0.02 * shrink).to(torch.float16))
    elif fmt == Q4_K:
        w[:, 0:2] = _raw(_f16(g, nb, 2e-4 * shrink, 2e-3 * shrink))
        w[:, 2:4] = _raw(_f16(g, nb, 1e-4 * shrink, 1e-3 * shrink))
    elif fmt == TERNARY:
        w[:, 0:2] = _raw(_f16(g, nb, 0.01 * shrink, 0.05 * shrink))
        w[:, 4:12] = _ternary_bytes(g, nb * 8).reshape(nb, 8)
    elif fmt == VAR_RATE:
        w[:, 0:2] = _raw(_f16(g, nb, 4e-4, 4e-3))
        w[:, 2:4] = _raw(_f16(g, nb, -0.005, 0.01))
        w[:, 20:28] = torch.tensor([(s % 3) << 3 | b for s, b in enumerate((3, 3, 4, 4, 4, 4, 5, 5))], dtype=torch.uint8, device="cuda")
    elif fmt == CODEBOOK:
        w[:, 0:2] = _raw(_f16(g, nb, 3e-4, 3e-3))
        w[:, 2:4] = _raw(_f16(g, nb, -0.004, 0.008))
        w[:, 20:36] = torch.randint(-8, 8, (nb, 16), dtype=torch.int8, device="cuda", generator=g).view(torch.uint8)
    else:
        w[:, 0:2] = _raw(_f16(g, nb, 0.01 * shrink, 0.05 * shrink))
    return w.reshape(-1)


# scale of a layer's weights against a lone projection's at hidden size 4096, so that both residual blocks add about as
# much as the stream already holds and stay inside fp16
LAYER_SHRINK = {Q4_0: 0.16, MLX: 0.16, TERNARY: 1.0}


def _layer_weights(c, g):
    q, kv, s = c["Hq"] * c["D"], c["Hkv"] * c["D"], LAYER_SHRINK[c["fmt"]] * (4096 / c["K"]) ** 0.55
    rows = {"q": (q, c["K"]), "k": (kv, c["K"]), "v": (kv, c["K"]), "o": (c["K"], q), "gate": (c["F"], c["K"]), "up": (c["F"], c["K"]), "down": (c["K"], c["F"])}
    return {name: _weights(c["fmt"], n, k, g, s) for name, (n, k) in rows.items()}


def _kv_cache(bridge, g, c):
    """Keys or values of pos0 + M tokens: fp16 [Hkv][tokens][D], or its Q8_0 records."""
    t = torch.randn(c["Hkv"], c["pos0"] + c["M"], c["D"], device="cuda", generator=g).to(torch.float16)
    if c["kv_fp16"]:
        return t
    packed = torch.empty(t.numel() // 32 * 34, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rc = bridge.lib.b200_bridge_quantize_kv_q8_0(t.data_ptr(), t.numel() * 2, packed.data_ptr(), packed.numel(), t.numel())
    if rc:
        raise RuntimeError(f"quantize failed: {rc}")
    bridge.synchronize()
    return packed


def prepare(case, seed):
    pkg = load_package()
    bridge = pkg.B200Bridge.get_instance()
    if not bridge.init():
        raise RuntimeError("bridge initialisation failed")
    c, g, s = dict(case), _gen(seed), {"case": dict(case), "bridge": bridge}
    kind = c["kind"]
    if kind == "linear":
        from m4_prefill_engine_b200.modules import M4QuantizedLinear
        s["module"] = M4QuantizedLinear(c["K"], c["N"], format=c["fmt"], weight=_weights(c["fmt"], c["N"], c["K"], g))
        s["x"] = torch.randn(c["M"], c["K"], device="cuda", generator=g).to(torch.float16)
    elif kind == "gemm":
        s["w"] = _weights(c["fmt"], c["N"], c["K"], g)
        s["x"] = torch.randn(c["M"], c["K"], device="cuda", generator=g).to(torch.float16)
        s["y"] = torch.empty(c["M"], c["N"], dtype=torch.float16, device="cuda")
    elif kind == "swiglu":
        s["gate"], s["up"] = _weights(c["fmt"], c["F"], c["K"], g, 0.25), _weights(c["fmt"], c["F"], c["K"], g, 0.25)
        s["x"] = (torch.randn(c["M"], c["K"], device="cuda", generator=g) * 0.25).to(torch.float16)
        s["y"] = torch.empty(c["M"], c["F"], dtype=torch.float16, device="cuda")
    elif kind == "attention":
        s["q"] = torch.randn(c["Hq"], c["M"], c["D"], device="cuda", generator=g).to(torch.float16)
        s["k"], s["v"] = _kv_cache(bridge, g, c), _kv_cache(bridge, g, c)
        s["o"] = torch.empty(c["M"], c["Hq"] * c["D"], dtype=torch.float16, device="cuda")
    elif kind == "layer":
        from m4_prefill_engine_b200.layer import TransformerLayerConfig, TransformerLayerCoordinator
        s["w"] = _layer_weights(c, g)
        s["norms"] = [_f16(g, c["K"], 0.5, 1.5) for _ in range(2)]
        s["layer"] = TransformerLayerCoordinator(TransformerLayerConfig(
            M=c["M"], K=c["K"], H=c["Hq"], D=c["D"], N_mlp=c["F"], attn_scale=c["D"] ** -0.5, weight_format=c["fmt"],
            num_kv_heads=c["Hkv"], rms_eps=1e-5, rope_theta=500000.0, kv_q8_0=True))
        s["layer"].set_norm_weights(*s["norms"])
        s["x"] = torch.randn(c["M"], c["K"], device="cuda", generator=g).to(torch.float16)
        s["y"] = torch.empty_like(s["x"])
    else:
        from m4_prefill_engine_b200.model import EngineConfig, TransformerModel
        s["model"] = TransformerModel(EngineConfig(
            num_layers=c["layers"], hidden_dim=c["K"], num_q_heads=c["Hq"], num_kv_heads=c["Hkv"], head_dim=c["D"],
            intermediate_dim=c["F"], vocab_size=c["vocab"]), c["M"])
        s["model"].init_synthetic_weights(seed=int(seed))
        s["tokens"] = torch.randint(0, c["vocab"], (c["M"],), dtype=torch.int32, device="cuda", generator=g)
        s["logits"] = torch.empty(c["M"], c["vocab"], dtype=torch.float16, device="cuda")
    return s


def run(s):
    c, bridge = s["case"], s["bridge"]
    kind = c["kind"]
    if kind == "linear":
        return s["module"](s["x"])
    if kind == "gemm":
        if c["fmt"] in (PRISM, MLX_G64, TERNARY_ROW):
            bridge.dispatch_gemm_ex(s["x"], s["w"], s["y"], c["fmt"], c["M"], c["K"], c["N"])
        else:
            bridge.dispatch_gemm(s["x"], s["w"], s["y"], c["fmt"])
        bridge.synchronize()
        return s["y"]
    if kind == "swiglu":
        bridge.dispatch_swiglu(s["x"], s["gate"], s["up"], s["y"], c["fmt"], c["M"], c["K"], c["F"])
        bridge.synchronize()
        return s["y"]
    if kind == "attention":
        rc = bridge.lib.b200_bridge_dispatch_attention_q8kv(
            s["q"].data_ptr(), s["k"].data_ptr(), s["v"].data_ptr(), s["o"].data_ptr(), c["Hq"], c["Hkv"], c["M"],
            c["pos0"] + c["M"], c["D"], c["D"] ** -0.5, c["pos0"], 1, int(c["kv_fp16"]))
        if rc:
            raise RuntimeError(f"attention failed: {rc}")
        return s["o"]
    if kind == "layer":
        w = s["w"]
        s["layer"].forward(s["x"], w["q"], w["k"], w["v"], w["o"], w["gate"], w["up"], w["down"], s["y"])
        return s["y"]
    s["model"].forward(s["tokens"], s["logits"])
    bridge.synchronize()
    return s["logits"]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _w_bytes(fmt, n, k):
    if fmt == MLX_G64:
        return n * k // 2 + n * k // 16
    if fmt == TERNARY_ROW:
        return n * k // 4 + 2 * n
    return n * (k // BLOCK[fmt][0]) * BLOCK[fmt][1]


def _attention(m, past, hq, hkv, d, kv_bytes_per_value):
    pairs = m * past + m * (m + 1) // 2
    return 4 * hq * m * d + 2 * hkv * (past + m) * d * kv_bytes_per_value, 4 * hq * pairs * d


def _layer(c, fmt):
    m, k, q, kv, f = c["M"], c["K"], c["Hq"] * c["D"], c["Hkv"] * c["D"], c["F"]
    weights = sum(_w_bytes(fmt, n, kk) for n, kk in ((q, k), (kv, k), (kv, k), (k, q), (f, k), (f, k), (k, f)))
    flops = 2 * m * (k * (q + 2 * kv) + q * k + 3 * k * f) + _attention(m, 0, c["Hq"], c["Hkv"], c["D"], 2)[1]
    return weights, flops


def work(case):
    c = case
    kind, m = c["kind"], c["M"]
    if kind in ("linear", "gemm"):
        return {"bytes": _w_bytes(c["fmt"], c["N"], c["K"]) + 2 * m * (c["K"] + c["N"]), "flops": 2 * m * c["N"] * c["K"]}
    if kind == "swiglu":
        return {"bytes": 2 * _w_bytes(c["fmt"], c["F"], c["K"]) + 2 * m * (c["K"] + c["F"]), "flops": 4 * m * c["F"] * c["K"]}
    if kind == "attention":
        b, f = _attention(m, c["pos0"], c["Hq"], c["Hkv"], c["D"], 2 if c["kv_fp16"] else 34 / 32)
        return {"bytes": b, "flops": f}
    if kind == "layer":
        w, f = _layer(c, c["fmt"])
        return {"bytes": w + 4 * m * c["K"], "flops": f}
    w, f = _layer(c, Q4_0)
    return {"bytes": c["layers"] * w + _w_bytes(Q4_0, c["vocab"], c["K"]) + 2 * m * (c["K"] + c["vocab"]),
            "flops": c["layers"] * f + 2 * m * c["K"] * c["vocab"]}


def tolerance(case):
    """Three to four times the largest relative error of the path as first measured against 64-bit arithmetic (``exact``):
    projections 2.1e-4 (ternary) to 3.6e-4, SwiGLU 4.6e-4, attention 4.2e-4, a layer 1.0e-3, models 4.4e-4."""
    kind = case["kind"]
    return {"rel": {"linear": 1.5e-3, "gemm": 1.5e-3, "swiglu": 2e-3, "attention": 1.2e-3, "layer": 3.5e-3, "model": 2e-3}[kind]}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------------------
def _half(b, at):
    """The fp16 field at byte `at` of every block, as float64 [blocks, 1]."""
    return b[:, at:at + 2].contiguous().view(torch.float16).double()


def _bit_fields(b, bits):
    """Little-endian runs of `bits`-bit codes: uint8 [blocks, bytes] -> float64 [blocks, bytes * 8 // bits]."""
    one = (b.unsqueeze(-1) >> torch.arange(8, device=b.device, dtype=torch.uint8)) & 1
    one = one.reshape(b.shape[0], -1)
    n = one.shape[1] // bits
    weight = torch.tensor([1 << i for i in range(bits)], device=b.device, dtype=torch.float64)
    return one[:, :n * bits].reshape(b.shape[0], n, bits).double() @ weight


def _nibbles(b):
    """16 bytes of a block of 32: low nibbles are elements 0 .. 15, high nibbles elements 16 .. 31."""
    return torch.cat([b & 15, b >> 4], dim=1).double()


def _dense(fmt, w, n, k):
    """Packed weights -> float64 [n, k]."""
    if fmt == MLX_G64:
        codes = _bit_fields(w[:n * k // 2].reshape(-1, 32), 4)
        planes = w[n * k // 2:].view(torch.float16).double().reshape(2, -1, 1)
        return (codes * planes[0] + planes[1]).reshape(n, k)
    if fmt == TERNARY_ROW:
        codes = _bit_fields(w[:n * k // 4].reshape(n, k // 4), 2) - 1
        return codes * w[n * k // 4:].view(torch.float16).double().reshape(n, 1)
    b = w.reshape(-1, BLOCK[fmt][1])
    d = _half(b, 0)
    if fmt == Q4_0:
        v = (_nibbles(b[:, 2:]) - 8) * d
    elif fmt == MLX:
        v = _nibbles(b[:, 4:]) * d + _half(b, 2)
    elif fmt == Q4_K:
        lo, hi = b[:, 4:12].long(), b[:, 12:16].long()
        minimum = torch.cat([hi & 15, hi >> 4], dim=1) | ((lo >> 6) << 4)
        codes = _nibbles(b[:, 16:].reshape(-1, 16)).reshape(-1, 8, 32)
        v = codes * (d * (lo & 63).double()).unsqueeze(-1) - (_half(b, 2) * minimum.double()).unsqueeze(-1)
    elif fmt == TERNARY:
        v = (_bit_fields(b[:, 4:], 2) - 1) * d
    elif fmt == VAR_RATE:
        parts, at = [], 32
        for s in range(8):
            bits, order = int(b[0, 20 + s]) & 7, int(b[0, 20 + s]) >> 3        # the same for every block of these inputs
            run = b[:, at:at + 4 * bits]
            q = _nibbles(run) if bits == 4 else _bit_fields(run, bits)
            q = q - 2 ** (bits - 1)
            if order == 1:
                q = torch.cat([q[:, 0::2], q[:, 1::2]], dim=1)
            elif order == 2:
                q = q.flip(1)
            at += 4 * bits
            parts.append(q * (d * b[:, 4 + s:5 + s].double() / 16) + _half(b, 2) + d * (b[:, 12 + s:13 + s].double() - 128) / 16)
        v = torch.cat(parts, dim=1)
    elif fmt == CODEBOOK:
        book = b[:, 20:36].contiguous().view(torch.int8).double()
        codes = _bit_fields(b[:, 48:].reshape(-1, 12), 3).long().reshape(-1, 256)
        scale = (d * b[:, 4:12].double() / 64).repeat_interleave(32, dim=1)
        residual = (d * (b[:, 12:20].double() - 128) / 128).repeat_interleave(32, dim=1)
        v = _half(b, 2) + scale * book[:, :8].gather(1, codes) + residual * book[:, 8:].gather(1, codes)
    else:
        v = (_bit_fields(b[:, 2:], 2) - 1) * d
    return v.reshape(n, k)


def _rows(x, fmt, w, n, k):
    """x @ weights.T, at most 32 million weights at a time (the head of a large model does not fit as float64 otherwise)."""
    step = max(1, (1 << 25) // k)
    if fmt in (MLX_G64, TERNARY_ROW) or step >= n:
        return x @ _dense(fmt, w, n, k).T
    per_row = w.numel() // n
    return torch.cat([x @ _dense(fmt, w[i * per_row:min(n, i + step) * per_row], min(n, i + step) - i, k).T for i in range(0, n, step)], dim=1)


def _q8(t):
    """Values as a Q8_0 cache holds them: 32 codes round(v * 127 / largest) and their scale as fp16."""
    b = t.reshape(-1, 32)
    d = b.abs().amax(dim=1, keepdim=True) / 127
    codes = torch.where(d > 0, b / d, torch.zeros_like(b))
    codes = (codes.sign() * (codes.abs() + 0.5).floor()).clamp(-128, 127)
    return (codes * d.to(torch.float16).double()).reshape(t.shape)


def _exact_attention(q, k, v, pos0):
    """q [Hq, M, D], k and v [Hkv, tokens, D] -> [M, Hq * D], causal behind pos0 cached tokens."""
    hq, m, d = q.shape
    group, tokens = hq // k.shape[0], k.shape[1]
    seen = torch.arange(tokens, device=q.device) <= pos0 + torch.arange(m, device=q.device).unsqueeze(1)
    out = torch.empty(m, hq, d, dtype=torch.float64, device=q.device)
    for h in range(hq):
        s = (q[h] @ k[h // group].T) * d ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(~seen, float("-inf")), dim=1) @ v[h // group]
    return out.reshape(m, hq * d)


def _exact_layer(x, w, norms, c, fmt, eps, theta):
    m, d, k = c["M"], c["D"], c["K"]

    def norm(t, weight):
        return t / (t.square().mean(dim=1, keepdim=True) + eps).sqrt() * weight.double()

    def heads(t, n):
        return t.reshape(m, n, d).transpose(0, 1)

    def rotate(t):
        a = torch.arange(m, device=t.device, dtype=torch.float64).unsqueeze(1) * theta ** (-torch.arange(0, d, 2, device=t.device, dtype=torch.float64) / d)
        lo, hi = t[..., :d // 2], t[..., d // 2:]
        return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], dim=-1)

    h = norm(x, norms[0])
    q = rotate(heads(_rows(h, fmt, w["q"], c["Hq"] * d, k), c["Hq"]))
    kk = _q8(rotate(heads(_rows(h, fmt, w["k"], c["Hkv"] * d, k), c["Hkv"])).contiguous())
    vv = _q8(heads(_rows(h, fmt, w["v"], c["Hkv"] * d, k), c["Hkv"]).contiguous())
    x = x + _rows(_exact_attention(q, kk, vv, 0), fmt, w["o"], k, c["Hq"] * d)
    h = norm(x, norms[1])
    act = torch.nn.functional.silu(_rows(h, fmt, w["gate"], c["F"], k)) * _rows(h, fmt, w["up"], c["F"], k)
    return x + _rows(act, fmt, w["down"], k, c["F"])


def _cached(t, c):
    """Keys or values of the cache as float64 [Hkv, tokens, D]."""
    if c["kv_fp16"]:
        return t.double()
    b = t.reshape(-1, 34)
    return (_half(b, 0) * b[:, 2:].contiguous().view(torch.int8).double()).reshape(c["Hkv"], c["pos0"] + c["M"], c["D"])


def exact(case, seed):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    if kind == "model":
        # the weights of TransformerModel.init_synthetic_weights: the same draws in the same order
        tokens = torch.randint(0, c["vocab"], (c["M"],), dtype=torch.int32, device="cuda", generator=g).long()
        ge, gw = _gen(seed), _gen(int(seed) * 1000)
        x = (torch.randn(c["vocab"], c["K"], device="cuda", generator=ge) * 0.02).to(torch.float16)[tokens].double()

        def q4_0(n, k):
            nb = n * (k // 32)
            blocks = torch.randint(0, 256, (nb, 18), dtype=torch.uint8, device="cuda", generator=gw)
            d = (torch.rand(nb, device="cuda", generator=gw) * (0.0033 - 0.0003) + 0.0003).to(torch.float16)
            blocks[:, 0:2] = d.view(torch.uint8).reshape(nb, 2)
            return blocks.reshape(-1)
        ones = torch.ones(c["K"], device="cuda")
        qd, kvd = c["Hq"] * c["D"], c["Hkv"] * c["D"]
        for _ in range(c["layers"]):
            w = {"q": q4_0(qd, c["K"]), "k": q4_0(kvd, c["K"]), "v": q4_0(kvd, c["K"]), "o": q4_0(c["K"], qd),
                 "gate": q4_0(c["F"], c["K"]), "up": q4_0(c["F"], c["K"]), "down": q4_0(c["K"], c["F"])}
            x = _exact_layer(x, w, (ones, ones), c, Q4_0, 1e-5, 10000.0)
        x = x / (x.square().mean(dim=1, keepdim=True) + 1e-5).sqrt()
        return _rows(x, Q4_0, q4_0(c["vocab"], c["K"]), c["vocab"], c["K"])
    s = prepare(case, seed)
    if kind == "linear":
        return _rows(s["x"].double(), c["fmt"], s["module"].weight, c["N"], c["K"])
    if kind == "gemm":
        return _rows(s["x"].double(), c["fmt"], s["w"], c["N"], c["K"])
    if kind == "swiglu":
        x = s["x"].double()
        return torch.nn.functional.silu(_rows(x, c["fmt"], s["gate"], c["F"], c["K"])) * _rows(x, c["fmt"], s["up"], c["F"], c["K"])
    if kind == "attention":
        return _exact_attention(s["q"].double(), _cached(s["k"], c), _cached(s["v"], c), c["pos0"])
    return _exact_layer(s["x"].double(), s["w"], s["norms"], c, c["fmt"], 1e-5, 500000.0)
