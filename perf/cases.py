"""Performance cases of the quantized-linear path, through ``Backend`` and the step driver.

A case is a dict of plain values; its ``kind`` says which call sequence it runs:

  linear    ``Backend.convrot_linear``: activation prep + int8 / int4 GEMM with fused dequant
  gemv      one decode linear: ``opGemvQuantizeX`` once, then ``opGemvQuantQ8N`` (GGUF formats, m <= 8)
  gemv_f32  ``opGemvQuant``: the single-row decode linear in f32 arithmetic
  layer     the seven linears of one decoder layer (q, k, v, o, gate, up, down) in mixed k-quants
  dit       blocks of the diffusion transformer through ``harness.dit_step_linears``

``listed()`` are the fixed cases, ``draw(rng)`` gives another one of the same ranges.
"""
from __future__ import annotations

import math

import torch

from tensorpencil_b200 import harness, synth
from tensorpencil_b200.backend import Backend

_F16_D = (1e-3, 1e-2)          # range of the f16 block scales, as in the decode benchmark
_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_ESZ = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # One INT8 linear over 256 tokens (a text prompt, or the smallest latent): too few tiles to fill the machine.
        {"name": "linear_i8_m256", "kind": "linear", "m": 256, "n": 3072, "k": 3072, "bits": 8, "x": "f32", "y": "f32"},
        # The MLP projection of a 1024 x 1024 image's transformer block with INT4 weights, f32 activations.
        {"name": "linear_i4_m4608", "kind": "linear", "m": 4608, "n": 12288, "k": 3072, "bits": 4, "x": "f32", "y": "f32"},
        # The down projection over a ragged token count (a small image and its prompt), bf16 activations.
        {"name": "linear_i8_m1111_bf16", "kind": "linear", "m": 1111, "n": 3072, "k": 12288, "bits": 8, "x": "bf16",
         "y": "bf16"},
        # The smallest decode call: a key or value projection of a grouped-query model, one token.
        {"name": "gemv_q8_0_kv_m1", "kind": "gemv", "fmt": "q8_0", "m": 1, "n": 1024, "k": 4096},
        # Decode, one token, up projection of a 27B model.
        {"name": "gemv_q8_0_up_m1", "kind": "gemv", "fmt": "q8_0", "m": 1, "n": 17408, "k": 5120},
        # Decode, eight rows (speculative tokens or eight requests), down projection of the same model.
        {"name": "gemv_q8_0_down_m8", "kind": "gemv", "fmt": "q8_0", "m": 8, "n": 5120, "k": 17408},
        # The single-token linear of steppers that keep f32 activations, up projection of an 8B model.
        {"name": "gemv_f32_m1", "kind": "gemv_f32", "n": 14336, "k": 4096},
        # One decoder layer of a Q4_K_M checkpoint of an 8B model, one token.
        {"name": "layer_q4_k_m_8b_m1", "kind": "layer", "mix": "q4_k_m", "m": 1, "hidden": 4096, "kv": 1024, "mlp": 14336},
        # One decoder layer of a Q5_K_M checkpoint of a 27B model, four speculative tokens.
        {"name": "layer_q5_k_m_27b_m4", "kind": "layer", "mix": "q5_k_m", "m": 4, "hidden": 5120, "kv": 1024, "mlp": 17408},
        # Transformer blocks as a host that keeps the reference's op sequence drives them: every elementwise op its
        # own call, f32, MLP in tiles of 2048 rows; a ragged token count.  (A step is 28 such blocks; one is timed, because
        # a rounding that flips in the quantiser of one linear reaches every token in the next block's attention.)
        {"name": "dit_i8_op_by_op", "kind": "dit", "bits": 8, "tokens": 2345, "latents": 1, "blocks": 1, "hidden": 3072,
         "seq": "unfused", "attn": True, "stream": False},
        # The same block at 1024 x 1024 (4096 image + 512 text tokens) through the fused calls in bf16.
        {"name": "dit_i8_fused_4608", "kind": "dit", "bits": 8, "tokens": 4608, "latents": 1, "blocks": 1, "hidden": 3072,
         "seq": "fused", "attn": True, "stream": False},
        # INT4 blocks streamed from pinned host memory, each used by a batch of latents while the next is on its way.
        {"name": "dit_i4_streamed", "kind": "dit", "bits": 4, "tokens": 4608, "latents": 4, "blocks": 4, "hidden": 3072,
         "seq": "fused", "attn": False, "stream": True},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "gemv", "gemv", "gemv_f32", "layer", "layer", "dit", "dit"])
    if kind == "linear":
        return {"kind": kind, "m": _log_int(rng, 16, 4608), "n": _log_int(rng, 1024, 12288, 16),
                "k": _log_int(rng, 1024, 12288, 256), "bits": rng.choice([8, 4]), "x": rng.choice(["f32", "bf16", "f16"]),
                "y": rng.choice(["f32", "bf16"])}
    if kind == "gemv":
        return {"kind": kind, "fmt": rng.choice(["q8_0", "q8_0", "q4_0", "q4_k", "q5_k", "q6_k", "iq4_nl"]),
                "m": rng.randint(1, 8), "n": _log_int(rng, 1024, 32000), "k": _log_int(rng, 2048, 17408, 256)}
    if kind == "gemv_f32":
        return {"kind": kind, "n": _log_int(rng, 1024, 32000), "k": _log_int(rng, 2048, 17408, 256)}
    if kind == "layer":
        hidden = _log_int(rng, 2048, 5120, 256)
        return {"kind": kind, "mix": rng.choice(["q4_k_m", "q5_k_m", "q8_0", "q4_0"]), "m": rng.randint(1, 8),
                "hidden": hidden, "kv": rng.choice([512, 1024, 2048]), "mlp": _log_int(rng, 2 * hidden, 17408, 256)}
    seq = rng.choice(["unfused", "fused", "fused"])
    stream = seq == "fused" and rng.random() < 0.34
    bits = rng.choice([8, 4])
    return {"kind": kind, "bits": bits, "tokens": _log_int(rng, 512, 4608), "latents": rng.choice([1, 2]),
            "blocks": 3 if stream else 1, "hidden": rng.choice([1536, 2304, 3072]), "seq": seq,
            "attn": bits == 8 and not stream and rng.random() < 0.8, "stream": stream}


# -- state ----------------------------------------------------------------------------------

_be = None


def _backend() -> Backend:
    global _be
    if _be is None:
        _be = Backend(0)
    return _be


def _activations(m, k, g, dtype=torch.float32):
    """N(0,1) with 1 % of the channels scaled x20 (outlier channels)."""
    x = torch.randn((m, k), device=g.device, generator=g)
    ch = torch.randperm(k, device=g.device, generator=g)[: k // 100]
    x[:, ch] *= 20.0
    return x.to(dtype)


def _f16_bytes(shape, lo, hi, g):
    d = torch.rand(shape, device=g.device, generator=g) * (hi - lo) + lo
    return d.to(torch.float16).unsqueeze(-1).view(torch.uint8)


def _gguf_weight(fmt, n, k, g):
    """Rows of GGUF blocks: random quants, finite f16 scales of the size checkpoints have."""
    elems, nbytes = synth.GGUF_BLOCK[fmt]
    shape = (n, k // elems)
    w = torch.randint(0, 256, shape + (nbytes,), dtype=torch.uint8, device=g.device, generator=g)
    if fmt == "q6_k":
        w[..., 208:210] = _f16_bytes(shape, 1e-4, 1e-3, g)
    else:
        w[..., 0:2] = _f16_bytes(shape, *_F16_D, g)
    if fmt in ("q4_k", "q5_k"):
        w[..., 2:4] = _f16_bytes(shape, *_F16_D, g)
    return w.reshape(n, -1)


def _layer_shapes(case):
    """(name, format, rows, columns) of a decoder layer's linears.  The _M mixes keep v and down in q6_k."""
    base, fine = {"q4_k_m": ("q4_k", "q6_k"), "q5_k_m": ("q5_k", "q6_k")}.get(case["mix"], (case["mix"], case["mix"]))
    h, kv, mlp = case["hidden"], case["kv"], case["mlp"]
    return [("q", base, h, h), ("k", base, kv, h), ("v", fine, kv, h), ("o", base, h, h), ("gate", base, mlp, h),
            ("up", base, mlp, h), ("down", fine, h, mlp)]


class _Dit:
    """Weights, modulation vectors and attention tables of a run of blocks, and the latents."""

    def __init__(self, case, seed, g):
        be, h = _backend(), case["hidden"]
        m = case["tokens"] * case["latents"]
        budget = None
        if case["stream"]:     # room for two blocks (their eight weights and scales): one in use, one on its way
            budget = 2 * (17 * h * h * case["bits"] // 8 + 56 * h + 8192)
        self.w = harness.DitWeights(be, case["bits"], blocks=case["blocks"], hidden=h, mlp=4 * h, seed=seed,
                                    stream_budget=budget)
        self.mod = harness.dit_modulation(be, case["blocks"], h, seed=seed + 1)
        self.latents = torch.randn((m, h), device=g.device, generator=g)
        self.x = torch.empty_like(self.latents)
        self.attn = None
        if case["attn"]:
            _, _, _, qn, kn, cos, sin = harness.attention_inputs(case["tokens"], 1, 1, g.device, seed=seed + 2)
            self.attn = {"q_norm": qn, "k_norm": kn, "cos": cos, "sin": sin, "heads": h // 128}

    def __del__(self):
        if getattr(self, "w", None) is not None and self.w.streamer is not None:
            torch.cuda.synchronize()
            self.w.close()


def prepare(case, seed):
    be = _backend()
    g = torch.Generator(device=be.device).manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        s["x"] = _activations(m, k, g, _DTYPES[case["x"]])
        if case["bits"] == 8:
            s["w"] = torch.randint(-127, 128, (n, k), dtype=torch.int8, device=be.device, generator=g)
        else:
            s["w"] = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device=be.device, generator=g)
        s["w_scale"] = torch.rand(n, device=be.device, generator=g) * 9e-3 + 1e-3
    elif kind in ("gemv", "gemv_f32"):
        fmt = case.get("fmt", "q8_0")
        s["x"] = torch.randn((case.get("m", 1), case["k"]), device=be.device, generator=g)
        s["w"] = _gguf_weight(fmt, case["n"], case["k"], g)
    elif kind == "layer":
        s["w"] = {name: _gguf_weight(fmt, n, k, g) for name, fmt, n, k in _layer_shapes(case)}
        h, mlp = case["hidden"], case["mlp"]
        # the inputs of (q, k, v), o, (gate, up) and down: what the norms, the attention and the SiLU gate leave
        s["x"] = {name: torch.randn((case["m"], k), device=be.device, generator=g)
                  for name, k in (("attn_in", h), ("attn_out", h), ("mlp_in", h), ("mlp_act", mlp))}
    else:
        s["dit"] = _Dit(case, seed, g)
    return s


# -- one pass -------------------------------------------------------------------------------


def _decode_linears(be, x, weights):
    """Quantise x [m][k] once, then one grouped GEMV per weight: the decode linear of the steppers."""
    m, k = x.shape
    be.opGemvQuantizeX(x, m * k)
    out = []
    for fmt, w, n in weights:
        y = torch.empty((m, n), dtype=torch.float32, device=be.device)
        be.opGemvQuantQ8N(fmt, y, w, 1.0, n, k, m, 0, m)
        out.append(y)
    return out


def run(state):
    be, case = _backend(), state["case"]
    kind = case["kind"]
    if kind == "linear":
        return be.convrot_linear(state["x"], state["w"], state["w_scale"], case["n"], case["bits"],
                                 out_dtype=_DTYPES[case["y"]])
    if kind == "gemv":
        if case["fmt"] == "q8_0":
            return be.q8_0_linear(state["x"], state["w"], case["n"], case["k"])
        return _decode_linears(be, state["x"], [(case["fmt"], state["w"], case["n"])])[0]
    if kind == "gemv_f32":
        y = torch.empty((1, case["n"]), dtype=torch.float32, device=be.device)
        be.opGemvQuant("q8_0", y, state["x"], state["w"], 1.0, case["n"], case["k"])
        return y
    if kind == "layer":
        w, x = state["w"], state["x"]
        shp = {name: (fmt, w[name], n) for name, fmt, n, _ in _layer_shapes(case)}
        return (_decode_linears(be, x["attn_in"], [shp["q"], shp["k"], shp["v"]])
                + _decode_linears(be, x["attn_out"], [shp["o"]])
                + _decode_linears(be, x["mlp_in"], [shp["gate"], shp["up"]])
                + _decode_linears(be, x["mlp_act"], [shp["down"]]))
    d = state["dit"]
    d.x.copy_(d.latents)     # the step updates the residual stream in place
    fused = case["seq"] == "fused"
    return harness.dit_step_linears(be, d.w, d.x, torch.bfloat16 if fused else torch.float32,
                                    mlp_tile=d.x.shape[0] if fused else harness.MLP_TILE, mode=case["seq"], mod=d.mod,
                                    attn=d.attn, latents=case["latents"], mlp_pair=fused, qkvg_group=fused)


# -- what a pass cannot do without, and how far two correct results can be apart ------------


def _gguf_bytes(fmt, n, k):
    elems, nbytes = synth.GGUF_BLOCK[fmt]
    return n * (k // elems) * nbytes


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": m * k * _ESZ[case["x"]] + n * k * case["bits"] // 8 + 4 * n + m * n * _ESZ[case["y"]],
                "flops": 2.0 * m * n * k}
    if kind in ("gemv", "gemv_f32"):
        m, n, k = case.get("m", 1), case["n"], case["k"]
        return {"bytes": _gguf_bytes(case.get("fmt", "q8_0"), n, k) + 4 * m * (n + k), "flops": 2.0 * m * n * k}
    if kind == "layer":
        m = case["m"]
        shapes = _layer_shapes(case)
        return {"bytes": sum(_gguf_bytes(f, n, k) + 4 * m * n for _, f, n, k in shapes)
                + 4 * m * (3 * case["hidden"] + case["mlp"]),
                "flops": sum(2.0 * m * n * k for _, _, n, k in shapes)}
    h, m = case["hidden"], case["tokens"] * case["latents"]
    flops = harness.dit_linear_ops(m, case["blocks"], h, 4 * h)
    if case["attn"]:
        flops += case["blocks"] * case["latents"] * 4.0 * case["tokens"] ** 2 * h
    return {"bytes": case["blocks"] * 17 * h * h * case["bits"] // 8 + 8 * m * h, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        # exact integers, then two f32 products (and one rounding to bf16)
        return {"rel": 1e-5} if case["y"] == "f32" else {"rel": 4e-3}
    if kind in ("gemv", "gemv_f32", "layer"):
        return {"rel": 1e-5}     # f32 sums in another order
    # Between linears a value is quantised to 8 or 4 bits: a last-bit difference (bf16 rounding, softmax) that flips a
    # rounding moves it by a whole quantisation step, which the following linear spreads over its row.  Measured: a block
    # with its attention in 64 bits differs by 0.021 (largest value 0.24), the streamed blocks with 1 ulp of noise on
    # their modulation vectors by 0.025 (1.2) -- the difference of two equally good quantisations, so it saturates there.
    return {"rel": 3e-2, "max": 0.99}


# -- the same results in 64 bits --------------------------------------------------------------


def _f16(b):
    return b.contiguous().view(torch.float16).double()          # [..., 2] bytes -> [..., 1]


def _dequant(fmt, w, k):
    """[n][row bytes] of GGUF blocks -> [n][k] in f64."""
    if fmt in ("q8_0", "q4_0", "iq4_nl"):
        b = w.reshape(w.shape[0], k // 32, -1)
        d = _f16(b[..., :2])
        if fmt == "q8_0":
            v = b[..., 2:].contiguous().view(torch.int8).double()
        else:
            q = torch.cat([b[..., 2:] & 15, b[..., 2:] >> 4], dim=-1)
            if fmt == "q4_0":
                v = q.double() - 8
            else:
                table = torch.tensor([-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113],
                                     dtype=torch.float64, device=w.device)
                v = table[q.long()]
        return (d * v).reshape(-1, k)
    b = w.reshape(w.shape[0], k // 256, -1)
    if fmt == "q6_k":
        ql, qh = b[..., :128].unflatten(-1, (2, 2, 32)), b[..., 128:192].unflatten(-1, (2, 1, 32))
        low = torch.cat([ql & 15, ql >> 4], dim=-2)                                      # [.., half, 4, 32]
        high = torch.cat([(qh >> (2 * p)) & 3 for p in range(4)], dim=-2)
        sc = b[..., 192:208].contiguous().view(torch.int8).double().unsqueeze(-1)
        q = ((low | (high << 4)).double() - 32).flatten(-3).unflatten(-1, (16, 16))
        return (_f16(b[..., 208:210]).unsqueeze(-1) * sc * q).reshape(-1, k)
    d, dmin, s = _f16(b[..., 0:2]), _f16(b[..., 2:4]), b[..., 4:16]
    sc = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | (s[..., :4] >> 6 << 4)], dim=-1)
    mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | (s[..., 4:8] >> 6 << 4)], dim=-1)
    qs = b[..., -128:].unflatten(-1, (4, 1, 32))
    q = torch.cat([qs & 15, qs >> 4], dim=-2).flatten(-3, -2)                              # [.., 8, 32]
    if fmt == "q5_k":
        q = q | torch.stack([(b[..., 16:48] >> i & 1) << 4 for i in range(8)], dim=-2)
    return ((d * sc.double()).unsqueeze(-1) * q.double() - (dmin * mn.double()).unsqueeze(-1)).reshape(-1, k)


def _q8_1(x):
    """The values that the activation quantiser of the decode linears leaves: 32 of them share one scale."""
    b = x.unflatten(-1, (-1, 32))
    amax = b.abs().amax(-1, keepdim=True)
    q = torch.where(amax > 0, torch.round(b * (127.0 / amax)), torch.zeros_like(b))       # f32: the same ties
    return ((amax / 127.0).double() * q.double()).flatten(-2)


def _gguf_linear(fmt, w, x, k):
    rows = max(1, (1 << 27) // k)
    return torch.cat([x @ _dequant(fmt, w[r:r + rows], k).T for r in range(0, w.shape[0], rows)], dim=1)


def _rotate(x):
    """Every 256 columns times the orthonormal Hadamard matrix that is the Kronecker power of the 4 x 4 one."""
    h4 = torch.tensor([[1, 1, 1, -1], [1, 1, -1, 1], [1, -1, 1, 1], [-1, 1, 1, 1]], dtype=torch.float64, device=x.device)
    h = torch.kron(torch.kron(h4, h4), torch.kron(h4, h4)) / 16
    return (x.double().unflatten(-1, (-1, 256)) @ h.T).flatten(-2)


def exact(case, seed):
    """The quantised operands as they are, everything after them in 64 bits.  None for the transformer blocks: their
    linears quantise what the one before computed, so their results have no value that every correct rounding is near."""
    kind = case["kind"]
    if kind == "dit":
        return None
    s = prepare(case, seed)
    if kind == "linear":
        maxq = 127 if case["bits"] == 8 else 7
        r = _rotate(s["x"])
        a = (r.abs().amax(1, keepdim=True) / maxq).clamp_min(1e-12)
        q = torch.sign(r) * torch.floor((r / a).abs() + 0.5)
        w = s["w"]
        if case["bits"] == 4:
            n = torch.stack([w & 15, w >> 4], dim=-1).flatten(-2)
            w = n.to(torch.int8) - 16 * (n > 7).to(torch.int8)
        return (q @ w.double().T) * a * s["w_scale"].double()
    if kind == "gemv_f32":
        return _gguf_linear("q8_0", s["w"], s["x"].double(), case["k"])
    if kind == "gemv":
        return _gguf_linear(case["fmt"], s["w"], _q8_1(s["x"]), case["k"])
    of = {"q": "attn_in", "k": "attn_in", "v": "attn_in", "o": "attn_out", "gate": "mlp_in", "up": "mlp_in", "down": "mlp_act"}
    return [_gguf_linear(fmt, s["w"][name], _q8_1(s["x"][of[name]]), k) for name, fmt, _, k in _layer_shapes(case)]
