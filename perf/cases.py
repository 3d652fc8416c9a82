"""The work that users of llmp_b200 have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points as a serving program calls them:
a decode step is queued once, captured in a CUDA graph and replayed (the library's calls only
queue work, so they can be captured); a prefill call and a single small call are queued as they
come.  Weights and activations are synthetic values in the reference's block formats, drawn on
the device from the seed; the shapes are the benchmark's (`bench.py`) and the tests'.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, weights and what else a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    tolerance(case)     how far another correct implementation may be from this one
    exact(case, seed)   what a pass returns, evaluated in 64 bits by plain torch
"""
from __future__ import annotations

import torch

import llmp_b200 as ops

HIDDEN, INTER, LAYERS = 2560, 10240, 34          # the benchmark's decode step
EXPERTS, USED, MOE_HIDDEN, MOE_INTER = 128, 8, 2048, 768
MOE_PREFILL = 97                                 # from here a routed block is a prefill's


def listed() -> list[dict]:
    return [
        # One F32 column through one small Q8_0 matrix: what a single call costs.
        {"name": "call_q8_0_2560x256", "kind": "mmvq", "k": 2560, "n": 256, "cols": 1},
        # A decode step's feed-forward blocks (quantize, gate|up GeGLU, quantize, down; every
        # layer its own weights): one sequence, a few, a small batch.
        {"name": "ffn_q4k_b1", "kind": "ffn", "hidden": HIDDEN, "inter": INTER, "layers": LAYERS,
         "tokens": 1, "glu": "geglu"},
        {"name": "ffn_q4k_b3", "kind": "ffn", "hidden": HIDDEN, "inter": INTER, "layers": LAYERS,
         "tokens": 3, "glu": "geglu"},
        {"name": "ffn_q4k_b8", "kind": "ffn", "hidden": HIDDEN, "inter": INTER, "layers": LAYERS,
         "tokens": 8, "glu": "geglu"},
        # The square Q8_0 projections of a decode step, one sequence.
        {"name": "proj_q8_0_b1", "kind": "proj", "k": 4096, "n": 4096, "layers": 16, "tokens": 1},
        # The same matrices through the decode module's product over F32 activations.
        {"name": "decode_vector_b1", "kind": "decode_vector", "decoder": "q8_0", "k": 4096, "n": 4096,
         "layers": 16, "tokens": 1},
        # Prefill of a short prompt of odd length straight from the Q4_K blocks, and of a long
        # one from the weights as a program relays them at load time.
        {"name": "mmq_203_blocks", "kind": "mmq", "tokens": 203, "k": HIDDEN, "n": INTER, "slab": False,
         "bf16": True},
        {"name": "mmq_4096_slab", "kind": "mmq", "tokens": 4096, "k": 4096, "n": 14336, "slab": True,
         "bf16": True},
        # An MXFP8 linear layer: activations quantized, then the block-scaled GEMM.
        {"name": "mxfp8_linear_2048", "kind": "mxfp8", "tokens": 2048, "k": 4096, "n": 12288},
        # Routed-expert blocks: one sequence, a batch of sequences, a prefill.
        {"name": "moe_t1", "kind": "moe", "tokens": 1, "experts": EXPERTS, "used": USED,
         "hidden": MOE_HIDDEN, "inter": MOE_INTER, "layers": 8},
        {"name": "moe_t64", "kind": "moe", "tokens": 64, "experts": EXPERTS, "used": USED,
         "hidden": MOE_HIDDEN, "inter": MOE_INTER, "layers": 2},
        {"name": "moe_t4096", "kind": "moe", "tokens": 4096, "experts": EXPERTS, "used": USED,
         "hidden": MOE_HIDDEN, "inter": MOE_INTER, "layers": 1},
    ]


def _log(rng, lo: int, hi: int) -> int:
    """An integer of [lo, hi], even over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng) -> dict:
    kind = rng.choice(["mmvq", "ffn", "ffn", "proj", "decode_vector", "mmq", "mmq", "mxfp8", "moe", "moe"])
    if kind == "mmvq":
        return {"kind": kind, "k": 32 * _log(rng, 16, 128), "n": _log(rng, 64, 2048), "cols": rng.randint(1, 8)}
    if kind == "ffn":
        hidden, inter = 256 * _log(rng, 4, 20), 256 * _log(rng, 8, 56)
        layers = max(1, min(LAYERS, LAYERS * HIDDEN * INTER // (hidden * inter)))
        return {"kind": kind, "hidden": hidden, "inter": inter, "layers": rng.randint(max(1, layers // 2), layers),
                "tokens": rng.randint(1, 8), "glu": rng.choice(["geglu", "swiglu"])}
    if kind in ("proj", "decode_vector"):
        k, n = 128 * _log(rng, 8, 64), _log(rng, 256, 8192)
        c = {"kind": kind, "k": k, "n": n, "layers": max(1, min(48, (1 << 28) // (k * n))), "tokens": rng.randint(1, 4)}
        if kind == "decode_vector":
            c["decoder"] = rng.choice(["q8_0", "mxfp8", "bf16"])
        return c
    if kind == "mmq":
        k, n = 256 * _log(rng, 4, 32), _log(rng, 512, 14336)
        most = min(4096, 4096 * 4096 * 14336 // (k * n))
        return {"kind": kind, "tokens": _log(rng, 17, most), "k": k, "n": n, "slab": rng.random() < 0.5,
                "bf16": rng.random() < 0.5}
    if kind == "mxfp8":
        return {"kind": kind, "tokens": _log(rng, 17, 4096), "k": 128 * _log(rng, 8, 40), "n": _log(rng, 1024, 12288)}
    experts = rng.choice([16, 32, 64, 128])
    return {"kind": "moe", "tokens": _log(rng, 1, 4096), "experts": experts, "used": rng.choice([2, 4, 8]),
            "hidden": rng.choice([1024, 2048]), "inter": 256 * rng.randint(2, 6), "layers": 1}


# ------------------------------------------------------------------ operands
def _halves(gen, shape, scale: float) -> torch.Tensor:
    """FP16 |N(0, 0.02)| / scale, as bytes."""
    v = torch.randn(shape, device="cuda", generator=gen).abs_() * (0.02 / scale)
    return v.half().view(torch.uint8).view(*shape, 2)


def _q4_k(gen, rows: int, k: int) -> torch.Tensor:
    """uint8 [rows, k / 256 * 144]: uniform codes and 6-bit scales, FP16 d and dmin."""
    w = torch.randint(0, 256, (rows, k // 256, 144), dtype=torch.uint8, device="cuda", generator=gen)
    w[:, :, 0:2] = _halves(gen, (rows, k // 256), 15.0 * 32.0)
    w[:, :, 2:4] = _halves(gen, (rows, k // 256), 32.0)
    return w.view(rows, -1)


def _q8_0(gen, rows: int, k: int) -> torch.Tensor:
    """uint8 [rows, k / 32 * 34]: codes of [-127, 127], FP16 scales."""
    w = torch.randint(-127, 128, (rows, k // 32, 34), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
    w[:, :, 0:2] = _halves(gen, (rows, k // 32), 127.0)
    return w.view(rows, -1)


def _normal(gen, *shape) -> torch.Tensor:
    return torch.randn(shape, device="cuda", generator=gen)


def _captured(body):
    """`body` queued twice on a side stream, then captured there: the graph a serving loop replays."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        body()
        body()
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = body()
    torch.cuda.current_stream().wait_stream(side)
    return {"graph": graph, "out": out}


# ------------------------------------------------------------------ states
def _prepare_mmvq(c, gen):
    return {"w": _q8_0(gen, c["n"], c["k"]), "x": _normal(gen, c["cols"], c["k"])}


def _run_mmvq(c, s):
    return ops.mmvq(s["w"], ops.TYPE_Q8_0, c["k"], c["n"], s["x"])


def _inputs_ffn(c, gen):
    hidden, inter = c["hidden"], c["inter"]
    weights = [(_q4_k(gen, inter, hidden), _q4_k(gen, inter, hidden), _q4_k(gen, hidden, inter))
               for _ in range(c["layers"])]
    return weights, _normal(gen, c["layers"], c["tokens"], hidden)


def _prepare_ffn(c, gen):
    hidden, inter, tokens = c["hidden"], c["inter"], c["tokens"]
    glu = ops.GLU_GEGLU if c["glu"] == "geglu" else ops.GLU_SWIGLU
    weights, x = _inputs_ffn(c, gen)
    y = torch.empty_like(x)
    h = torch.empty((tokens, inter), device="cuda")
    q8x, q8h = ops.quantize_q8(x[0]), ops.quantize_q8(h.zero_())

    def step():
        for i, (gate, up, down) in enumerate(weights):
            ops.quantize_q8(x[i], out=q8x)
            ops.vecq(up, ops.TYPE_Q4_K, hidden, inter, q8x, tokens, gate=gate, glu=glu, out=h)
            ops.quantize_q8(h, out=q8h)
            ops.vecq(down, ops.TYPE_Q4_K, inter, hidden, q8h, tokens, out=y[i])
        return y

    return {"weights": weights, "x": x, **_captured(step)}


def _inputs_proj(c, gen):
    weights = [_q8_0(gen, c["n"], c["k"]) for _ in range(c["layers"])]
    return weights, _normal(gen, c["layers"], c["tokens"], c["k"])


def _prepare_proj(c, gen):
    k, n, tokens = c["k"], c["n"], c["tokens"]
    weights, x = _inputs_proj(c, gen)
    y = torch.empty((c["layers"], tokens, n), device="cuda")
    q8 = ops.quantize_q8(x[0])

    def step():
        for i, w in enumerate(weights):
            ops.quantize_q8(x[i], out=q8)
            ops.vecq(w, ops.TYPE_Q8_0, k, n, q8, tokens, out=y[i])
        return y

    return {"weights": weights, "x": x, **_captured(step)}


def _inputs_decode_vector(c, gen):
    k, n = c["k"], c["n"]
    x = _normal(gen, c["layers"], c["tokens"], k)
    weights = []
    for _ in range(c["layers"]):
        if c["decoder"] == "q8_0":
            weights.append((ops.DECODER_Q8_0, _q8_0(gen, n, k), None))
        elif c["decoder"] == "mxfp8":
            codes, atoms = ops.mxfp8_quantize(_normal(gen, n, k) * 0.02)
            weights.append((ops.DECODER_MXFP8_ATOMS, codes, atoms))
        else:
            weights.append((ops.DECODER_BF16, (_normal(gen, n, k) * 0.02).bfloat16().view(torch.uint8), None))
    return weights, x


def _prepare_decode_vector(c, gen):
    k, n, tokens = c["k"], c["n"], c["tokens"]
    weights, x = _inputs_decode_vector(c, gen)
    y = torch.empty((c["layers"], tokens, n), device="cuda")

    def step():
        for i, (decoder, data, scales) in enumerate(weights):
            ops.decode_vector(decoder, data, x[i], k, n, scales=scales, out=y[i])
        return y

    return {"weights": weights, "x": x, **_captured(step)}


def _inputs_mmq(c, gen):
    x = _normal(gen, c["tokens"], c["k"])
    return _q4_k(gen, c["n"], c["k"]), x.bfloat16() if c["bf16"] else x


def _prepare_mmq(c, gen):
    w, x = _inputs_mmq(c, gen)
    s = {"x": x, "w": w, "slab": None}
    if c["slab"]:
        s["slab"], s["w"] = ops.q4k_relayout(w, c["k"], c["n"]), None
    return s


def _run_mmq(c, s):
    return ops.mmq(s["w"], ops.mmq_quantize(s["x"]), c["k"], c["n"], slab=s["slab"])


def _prepare_mxfp8(c, gen):
    w, w_scales = ops.mxfp8_quantize(_normal(gen, c["n"], c["k"]) * 0.02)
    return {"x": _normal(gen, c["tokens"], c["k"]).bfloat16(), "w": w, "w_scales": w_scales}


def _run_mxfp8(c, s):
    a, a_scales = ops.mxfp8_quantize(s["x"])
    return ops.mxfp8_gemm(a, a_scales, s["w"], s["w_scales"], bf16=True)


def _inputs_moe(c, gen):
    """Per layer: activations, the experts' weights, and the router's choice for every token."""
    tokens, experts, used, hidden, inter = (c[n] for n in ("tokens", "experts", "used", "hidden", "inter"))
    for _ in range(c["layers"]):
        gate_up = _q4_k(gen, experts * 2 * inter, hidden).view(experts, 2 * inter, -1)
        down = _q4_k(gen, experts * hidden, inter).view(experts, hidden, -1)
        p, ids = torch.topk(torch.softmax(_normal(gen, tokens, experts), 1), used, dim=1)
        yield gate_up, down, ids.int(), (p / p.sum(1, keepdim=True)).contiguous(), _normal(gen, tokens, hidden)


def _prepare_moe(c, gen):
    tokens, hidden, inter = c["tokens"], c["hidden"], c["inter"]
    layers = []
    for gate_up, down, ids, weights, x in _inputs_moe(c, gen):
        # a prefill's experts as a program relays them at load time
        slabs = None
        if tokens >= MOE_PREFILL:
            slabs = (ops.q4k_relayout(gate_up, hidden, 2 * inter, glu=True),
                     ops.q4k_relayout(down, inter, hidden), True)
        layers.append((x, ids, weights, gate_up, down, slabs))

    def step():
        return [ops.moe_ffn(x, ids, w, gate_up, down, hidden, inter, slabs=slabs)
                for x, ids, w, gate_up, down, slabs in layers]

    if tokens >= MOE_PREFILL:
        return {"step": step}
    return {"layers": layers, **_captured(step)}


_PREPARE = {"mmvq": _prepare_mmvq, "ffn": _prepare_ffn, "proj": _prepare_proj,
            "decode_vector": _prepare_decode_vector, "mmq": _prepare_mmq, "mxfp8": _prepare_mxfp8,
            "moe": _prepare_moe}
_RUN = {"mmvq": _run_mmvq, "mmq": _run_mmq, "mxfp8": _run_mxfp8}


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return {"case": case, **_PREPARE[case["kind"]](case, gen)}


def run(state: dict):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if "step" in state:
        return state["step"]()
    return _RUN[state["case"]["kind"]](state["case"], state)


# ------------------------------------------------------------------ what a pass is
def work(case: dict) -> dict:
    """Weights in their block format once, F32 (or BF16) activations in, results out."""
    c, kind = case, case["kind"]
    if kind == "mmvq":
        k, n, t = c["k"], c["n"], c["cols"]
        return {"bytes": n * k * 34 / 32 + 4 * t * (k + n), "flops": 2.0 * k * n * t}
    if kind == "ffn":
        one = 3 * c["hidden"] * c["inter"]
        return {"bytes": c["layers"] * (one * 0.5625 + 8 * c["tokens"] * c["hidden"]),
                "flops": 2.0 * c["layers"] * one * c["tokens"]}
    if kind in ("proj", "decode_vector"):
        k, n, t = c["k"], c["n"], c["tokens"]
        byte = {"q8_0": 34 / 32, "mxfp8": 33 / 32, "bf16": 2.0}[c.get("decoder", "q8_0")]
        return {"bytes": c["layers"] * (n * k * byte + 4 * t * (k + n)), "flops": 2.0 * c["layers"] * k * n * t}
    if kind == "mmq":
        k, n, t = c["k"], c["n"], c["tokens"]
        return {"bytes": n * k * 0.5625 + t * (k * (2 if c["bf16"] else 4) + 4 * n), "flops": 2.0 * k * n * t}
    if kind == "mxfp8":
        k, n, t = c["k"], c["n"], c["tokens"]
        return {"bytes": n * k * 33 / 32 + t * (2 * k + 2 * n), "flops": 2.0 * k * n * t}
    pairs, one = c["tokens"] * c["used"], 3 * c["hidden"] * c["inter"]
    # experts that at least one token names, when the tokens choose evenly
    named = c["experts"] * (1.0 - (1.0 - c["used"] / c["experts"]) ** c["tokens"])
    return {"bytes": c["layers"] * (named * one * 0.5625 + 8 * c["tokens"] * c["hidden"]),
            "flops": 2.0 * c["layers"] * one * pairs}


def tolerance(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("mmvq", "proj", "decode_vector"):
        return {"rel": 2e-6}            # F32 sums in another order
    if kind == "mmq":
        return {"rel": 5e-6}
    if kind == "mxfp8":
        return {"rel": 5e-3}            # results rounded to BF16
    # the intermediate is quantized to 8 bits: a sum in another order moves some of its codes
    return {"rel": 1e-3, "max": 0.05}


# ------------------------------------------------------------------ the same in 64 bits
# The block formats' own roundings (8-bit codes, FP16 scales and sums) are part of what a pass
# returns and are restated; every product and sum is taken in 64 bits.
def _f16(raw: torch.Tensor) -> torch.Tensor:
    return raw.contiguous().view(torch.float16).squeeze(-1)


def _blocks_of_32(x: torch.Tensor, reciprocal: bool):
    """x F32 [rows, k] as 8-bit blocks: codes [rows, k / 32, 32], scales and sums [rows, k / 32]."""
    v = x.float().view(x.shape[0], -1, 32)
    amax = v.abs().amax(2, keepdim=True)
    live = torch.where(amax > 0, amax, torch.ones_like(amax))
    if reciprocal:
        # (one rounding: a number over a tensor would be the reciprocal times the number)
        inverse = torch.full_like(live, 127.0) / live
        codes, d = (v * inverse).double(), torch.ones_like(live) / inverse
    else:
        d = live / torch.full_like(live, 127.0)
        codes = (v / d).double()
    codes = torch.trunc(codes + torch.where(codes < 0, -0.5, 0.5))
    d = torch.where(amax > 0, d, torch.zeros_like(d))
    q = v.view(x.shape[0], v.shape[1], 8, 4)
    p = ((q[..., 0] + q[..., 1]) + q[..., 2]) + q[..., 3]
    s = ((p[..., 0] + p[..., 4]) + (p[..., 2] + p[..., 6])) + ((p[..., 1] + p[..., 5]) + (p[..., 3] + p[..., 7]))
    return codes, d.squeeze(2).half().double(), s.half().double()


def _q4_k_parts(w: torch.Tensor):
    """Codes [rows, k / 32, 32], FP16 d and dmin [rows, k / 256, 1], scales and minima [rows, k / 256, 8]."""
    b = w.reshape(w.shape[0], -1, 144)
    d, dmin, s = _f16(b[:, :, 0:2])[..., None], _f16(b[:, :, 2:4])[..., None], b[:, :, 4:16].int()
    sc = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], 2)
    mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], 2)
    c = b[:, :, 16:].view(b.shape[0], b.shape[1], 4, 32)
    return torch.stack([c & 15, c >> 4], 3).view(b.shape[0], -1, 32), d, dmin, sc, mn


def _dot_q4_k(w: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """The decode products' x [rows, k] by Q4_K rows: the minima multiply the codes' sums."""
    codes, d, dmin, sc, mn = _q4_k_parts(w)
    scale = (d.double() * sc).view(w.shape[0], -1, 1)
    minimum = (dmin.double() * mn).view(w.shape[0], -1, 1)
    dense = (codes.double() * scale - minimum).view(w.shape[0], -1)
    q, d8, _ = _blocks_of_32(x, False)
    return (q * d8[..., None]).view(x.shape[0], -1) @ dense.T


def _matmul_q4_k(w: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """The prefill products': FP16 products of the scales, the minima multiply the inputs' sums."""
    codes, d, dmin, sc, mn = _q4_k_parts(w)
    scale = (d * sc.half()).double().view(w.shape[0], -1, 1)
    minimum = (dmin * mn.half()).double().view(w.shape[0], -1)
    dense = (codes.double() * scale).view(w.shape[0], -1)
    q, d8, s8 = _blocks_of_32(x, True)
    return (q * d8[..., None]).view(x.shape[0], -1) @ dense.T - s8 @ minimum.T


def _dot_q8_0(w: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    q, d8, _ = _blocks_of_32(x, False)
    return (q * d8[..., None]).view(x.shape[0], -1) @ _dense_q8_0(w).T


def _dense_q8_0(w: torch.Tensor) -> torch.Tensor:
    b = w.view(w.shape[0], -1, 34)
    return (_f16(b[:, :, 0:2]).double()[..., None] * b[:, :, 2:].contiguous().view(torch.int8)).view(w.shape[0], -1)


def _glu(kind: str, gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    f = torch.nn.functional
    return (f.gelu(gate, approximate="tanh") if kind == "geglu" else f.silu(gate)) * up


def exact(case: dict, seed: int):
    c, kind = case, case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "mmvq":
        s = _prepare_mmvq(c, gen)
        return _dot_q8_0(s["w"], s["x"])
    if kind == "ffn":
        weights, x = _inputs_ffn(c, gen)
        return torch.stack([_dot_q4_k(down, _glu(c["glu"], _dot_q4_k(gate, x[i]), _dot_q4_k(up, x[i])))
                            for i, (gate, up, down) in enumerate(weights)])
    if kind == "proj":
        weights, x = _inputs_proj(c, gen)
        return torch.stack([_dot_q8_0(w, x[i]) for i, w in enumerate(weights)])
    if kind == "decode_vector" and c["decoder"] != "mxfp8":
        weights, x = _inputs_decode_vector(c, gen)
        return torch.stack([x[i].double() @ (_dense_q8_0(w) if c["decoder"] == "q8_0" else
                                             w.view(torch.bfloat16).double()).T
                            for i, (_, w, _) in enumerate(weights)])
    if kind == "mmq":
        return _matmul_q4_k(*_inputs_mmq(c, gen))
    if kind == "moe":
        outs = []
        for gate_up, down, ids, weights, x in _inputs_moe(c, gen):
            dot = _matmul_q4_k if c["tokens"] >= MOE_PREFILL else _dot_q4_k
            y = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
            for e in ids.unique().tolist():
                rows, slots = (ids == e).nonzero(as_tuple=True)
                gu = dot(gate_up[e], x[rows])
                h = _glu("swiglu", gu[:, :c["inter"]], gu[:, c["inter"]:])
                y.index_add_(0, rows, dot(down[e], h) * weights[rows, slots, None].double())
            outs.append(y)
        return outs
    return None  # MXFP8: the weights in hand are this package's own quantization of them
