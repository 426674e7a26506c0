"""The work that users of this library have it do, as measurable cases.

Every case goes through the public host mirror (``zllm_b200.backend``), eagerly, on tensors and weights that a runtime
holds anyway.  Kinds:

  linear  one projection (``Backend::linear`` / ``linear_add``)
  pair    up- and down-projection of one feed-forward block, as two calls (the prefill stack of the benchmark)
  mlp     ``gated_mlp_add_residual``: gate, up, SiLU, down, residual
  step    the linear work of a decoder step: embedding rows, then per layer RMSNorm + q/k/v, RoPE, output projection with
          residual and the gated MLP with residual, at the end RMSNorm + LM head.  Attention is outside this library, so
          a layer starts from the embedded row instead of the previous layer's attention output
  batch   independent projections of the decode sweep in one ``linear_batch`` call, or, with ``host``, in one
          ``linear_host_batch`` bracket on page-locked host buffers (activations come from the host and results go back)
  moe     router, routed experts and the shared expert of a mixture-of-experts layer
  requant Q8_0 -> f32 -> Q4_K (``requantize_q4_k``: what a loader does to a tensor it wants smaller)

Weights are N(0, 0.02) through this library's encoders (Q5_K and Q6_K have none: random codes under scales that give the
same spread), activations N(0, 1); everything is made from the seed.
"""
import math

import torch

from zllm_b200 import ffi
from zllm_b200.backend import B200Context, MoeExperts, moe_forward, moe_route

_TYPES = {"q4_0": ffi.Q4_0, "q8_0": ffi.Q8_0, "q4_k": ffi.Q4_K, "q5_k": ffi.Q5_K, "q6_k": ffi.Q6_K, "iq4_nl": ffi.IQ4_NL}
_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_SIZE = {"f32": 4, "f16": 2, "bf16": 2}
_SWEEP = "3840x3840,3840x15360,15360x3840,5120x17408,17408x5120"  # columns x rows of the decode sweep
_context = None


def _ctx():
    """One context per process and device, as a runtime keeps it."""
    global _context
    if _context is None:
        _context = B200Context(0)
    return _context


def listed():
    return [
        # the smallest call of the path: the key projection of a 1B-class decoder, one token; latency and launches
        {"name": "row_q4k_1536x512", "kind": "linear", "type": "q4_k", "cols": 1536, "rows": 512, "m": 1, "dtype": "f32", "residual": False},
        # single-stream decoding of a 1B-class Q4_K_M decoder (Q6_K for v and down in half of the layers, Q8_0 embedding and head)
        {"name": "step_1b_q4km", "kind": "step", "hidden": 1536, "kv": 512, "ffn": 3840, "head_dim": 64, "layers": 12, "vocab": 32768, "attn": "q4_k", "mlp": "q4_k", "more": "q6_k", "m": 1, "dtype": "f32"},
        # single-stream decoding of a mid-size decoder with Q8_0 attention and IQ4_NL feed-forward weights
        {"name": "step_mixed_q8_iq4nl", "kind": "step", "hidden": 3840, "kv": 3840, "ffn": 15360, "head_dim": 128, "layers": 4, "vocab": 32768, "attn": "q8_0", "mlp": "iq4_nl", "more": "iq4_nl", "m": 1, "dtype": "f16"},
        # the decode sweep at one row: the projections that are ready together, one call
        {"name": "sweep_q4k_m1", "kind": "batch", "type": "q4_k", "shapes": _SWEEP, "m": 1, "dtype": "f32", "host": False},
        # the same sweep for 16 sequences, activations on the host
        {"name": "sweep_q4_0_m16_host", "kind": "batch", "type": "q4_0", "shapes": _SWEEP, "m": 16, "dtype": "f32", "host": True},
        # 48 sequences decoding together (or a short prompt): more rows than the decode kernels take
        {"name": "pair_q4k_m48", "kind": "pair", "type": "q4_k", "hidden": 5120, "ffn": 17408, "m": 48, "dtype": "bf16"},
        # prefill of a 512-token chunk
        {"name": "pair_q4k_m512", "kind": "pair", "type": "q4_k", "hidden": 5120, "ffn": 17408, "m": 512, "dtype": "bf16"},
        # prefill of long prompts: the largest dense batch
        {"name": "pair_q4k_m16384", "kind": "pair", "type": "q4_k", "hidden": 5120, "ffn": 17408, "m": 16384, "dtype": "bf16"},
        # feed-forward block of a ragged prompt, block-32 weights
        {"name": "mlp_iq4nl_m3001", "kind": "mlp", "up": "iq4_nl", "down": "iq4_nl", "hidden": 3840, "ffn": 15360, "m": 3001, "dtype": "f16"},
        # mixture-of-experts decode: 64 sequences
        {"name": "moe_q4k_m64", "kind": "moe", "type": "q4_k", "experts": 256, "top_k": 8, "hidden": 7168, "inter": 2048, "m": 64, "dtype": "bf16", "shared": True},
        # mixture-of-experts prefill
        {"name": "moe_q4k_m8192", "kind": "moe", "type": "q4_k", "experts": 256, "top_k": 8, "hidden": 7168, "inter": 2048, "m": 8192, "dtype": "bf16", "shared": True},
        # requantising one large tensor at load time
        {"name": "requant_17408x5120", "kind": "requant", "rows": 17408, "cols": 5120},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _step_of(v, step):
    return max(step, v // step * step)


def draw(rng):
    kind = rng.choice(["linear", "linear", "step", "batch", "pair", "mlp", "moe", "requant"])
    types = ["q4_k", "q4_k", "q4_k", "q4_0", "q8_0", "iq4_nl", "q5_k", "q6_k"]
    dtype = rng.choice(["f32", "f16", "bf16"])
    if kind == "linear":
        t = rng.choice(types)
        return {"kind": kind, "type": t, "cols": _step_of(_log(rng, 512, 17408), 256 if t.endswith("_k") else 32), "rows": _log(rng, 256, 32768), "m": _log(rng, 1, 4096), "dtype": dtype, "residual": rng.random() < 0.5}
    if kind == "pair":
        hidden = _step_of(_log(rng, 1024, 5120), 256)
        return {"kind": kind, "type": rng.choice(types), "hidden": hidden, "ffn": _step_of(hidden * rng.randint(20, 40) // 10, 256), "m": _log(rng, 17, 8192), "dtype": rng.choice(["f16", "bf16"])}
    if kind == "mlp":
        hidden = _step_of(_log(rng, 1024, 5120), 256)
        return {"kind": kind, "up": rng.choice(types), "down": rng.choice(types), "hidden": hidden, "ffn": _step_of(hidden * rng.randint(20, 40) // 10, 256), "m": _log(rng, 1, 8192), "dtype": dtype}
    if kind == "step":
        hidden = _step_of(_log(rng, 1024, 5120), 256)
        return {"kind": kind, "hidden": hidden, "kv": rng.choice([hidden, hidden // 2, hidden // 4]) // 128 * 128, "ffn": _step_of(hidden * rng.randint(20, 40) // 10, 256), "head_dim": rng.choice([64, 128]), "layers": rng.randint(2, 6),
                "vocab": _log(rng, 16384, 65536) // 64 * 64, "attn": rng.choice(types), "mlp": rng.choice(types), "more": rng.choice(types), "m": _log(rng, 1, 256) if rng.random() < 0.5 else 1, "dtype": dtype}
    if kind == "batch":
        shapes = [f"{_step_of(_log(rng, 1024, 17408), 256)}x{_log(rng, 512, 17408)}" for _ in range(rng.randint(2, 8))]
        host = rng.random() < 0.3
        return {"kind": kind, "type": rng.choice(types), "shapes": ",".join(shapes), "m": rng.randint(1, 16) if rng.random() < 0.5 else 1, "dtype": rng.choice(["f32", "f16"]) if host else dtype, "host": host}
    if kind == "moe":
        experts = rng.choice([16, 32, 64, 128])
        return {"kind": kind, "type": rng.choice(types), "experts": experts, "top_k": rng.choice([2, 4, 6, 8]), "hidden": _step_of(_log(rng, 1024, 5120), 256), "inter": _step_of(_log(rng, 512, 2048), 256), "m": _log(rng, 1, 4096),
                "dtype": dtype, "shared": rng.random() < 0.5}
    return {"kind": kind, "rows": _log(rng, 512, 17408), "cols": _step_of(_log(rng, 512, 17408), 256)}


# ---- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rows(gen, m, cols, dtype="f32"):
    return torch.randn((m, cols), generator=gen, device="cuda", dtype=torch.float32).to(_DTYPES[dtype])


def _half_bytes(values):
    return values.to(torch.float16).reshape(-1, 1).view(torch.uint8)


def _weight(ctx, gen, kind, rows, cols):
    t = _TYPES[kind]
    if kind not in ("q5_k", "q6_k"):
        return ctx.prepare_weight(t, ctx.quantize(t, _rows(gen, rows, cols) * 0.02), rows, cols)
    elems, size = ffi.BLOCK[t]
    blocks = rows * cols // elems
    packed = torch.randint(0, 256, (blocks, size), generator=gen, device="cuda", dtype=torch.uint8)
    spread = torch.rand(blocks, generator=gen, device="cuda") * 0.4 + 0.8
    if kind == "q5_k":  # d, dmin: codes 0..31 under 6-bit scales, less a minimum that centres them
        packed[:, 0:2] = _half_bytes(spread * 6e-5)
        packed[:, 2:4] = _half_bytes(spread * 9e-4)
    else:               # d: codes -32..31 under signed 8-bit scales
        packed[:, 208:210] = _half_bytes(spread * 1.5e-5)
    return ctx.prepare_weight(t, packed.reshape(-1), rows, cols)


def _shapes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype).pin_memory()


def prepare(case, seed):
    ctx, gen, kind = _ctx(), _gen(seed), case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind == "linear":
        s["w"] = _weight(ctx, gen, case["type"], case["rows"], case["cols"])
        s["x"] = _rows(gen, case["m"], case["cols"], case["dtype"])
        s["residual"] = _rows(gen, case["m"], case["rows"], case["dtype"]) if case["residual"] else None
    elif kind == "pair":
        s["up"] = _weight(ctx, gen, case["type"], case["ffn"], case["hidden"])
        s["down"] = _weight(ctx, gen, case["type"], case["hidden"], case["ffn"])
        s["x"] = _rows(gen, case["m"], case["hidden"], case["dtype"])
        s["h"] = _rows(gen, case["m"], case["ffn"], case["dtype"])
    elif kind == "mlp":
        s["w"] = [_weight(ctx, gen, case["up"], case["ffn"], case["hidden"]), _weight(ctx, gen, case["up"], case["ffn"], case["hidden"]), _weight(ctx, gen, case["down"], case["hidden"], case["ffn"])]
        s["x"] = _rows(gen, case["m"], case["hidden"], case["dtype"])
        s["residual"] = _rows(gen, case["m"], case["hidden"], case["dtype"])
    elif kind == "step":
        hidden, kv, ffn = case["hidden"], case["kv"], case["ffn"]
        s["embedding"] = _weight(ctx, gen, "q8_0", case["vocab"], hidden)
        s["head"] = _weight(ctx, gen, "q8_0", case["vocab"], hidden)
        s["tokens"] = torch.randint(0, case["vocab"], (case["m"],), generator=gen, device="cuda", dtype=torch.int32)
        s["layers"] = []
        for i in range(case["layers"]):
            more = case["more"] if i % 2 else None  # the mixes of GGUF files give some layers' v and down another type
            s["layers"].append({
                "q": _weight(ctx, gen, case["attn"], hidden, hidden), "k": _weight(ctx, gen, case["attn"], kv, hidden), "v": _weight(ctx, gen, (case["attn"] if case["attn"] == "q8_0" else more) or case["attn"], kv, hidden),
                "o": _weight(ctx, gen, case["attn"], hidden, hidden), "gate": _weight(ctx, gen, case["mlp"], ffn, hidden), "up": _weight(ctx, gen, case["mlp"], ffn, hidden),
                "down": _weight(ctx, gen, more or case["mlp"], hidden, ffn), "norm": torch.rand(hidden, generator=gen, device="cuda") + 0.5})
        s["norm"] = torch.rand(hidden, generator=gen, device="cuda") + 0.5
        half = case["head_dim"] // 2
        angle = torch.arange(4096, device="cuda").unsqueeze(1) * torch.pow(10000.0, -torch.arange(half, device="cuda") / half)
        s["cos"], s["sin"] = torch.cos(angle).contiguous(), torch.sin(angle).contiguous()
        s["position"] = int(torch.randint(0, 2048, (1,), generator=gen, device="cuda"))
    elif kind == "batch":
        s["w"] = [_weight(ctx, gen, case["type"], rows, cols) for cols, rows in _shapes(case)]
        if case["host"]:
            s["jobs"], s["keep"] = [], []
            shared = {}  # projections of one width read the same activations
            for (cols, rows), w in zip(_shapes(case), s["w"]):
                if cols not in shared:
                    shared[cols] = _pinned((case["m"], cols), _DTYPES[case["dtype"]])
                    shared[cols].copy_(_rows(gen, case["m"], cols, case["dtype"]))
                y = _pinned((case["m"], rows), _DTYPES[case["dtype"]])
                s["keep"] += [shared[cols], y]
                s["jobs"].append((shared[cols].numpy(), w, y.numpy()))
        else:
            shared = {cols: _rows(gen, case["m"], cols, case["dtype"]) for cols, _ in _shapes(case)}
            s["jobs"] = [(shared[cols], w) for (cols, _), w in zip(_shapes(case), s["w"])]
    elif kind == "moe":
        experts, hidden, inter = case["experts"], case["hidden"], case["inter"]
        gate, up, down = [], [], []
        for _ in range(experts):
            gate.append(_weight(ctx, gen, case["type"], inter, hidden))
            up.append(_weight(ctx, gen, case["type"], inter, hidden))
            down.append(_weight(ctx, gen, case["type"], hidden, inter))
        s["table"] = MoeExperts(ctx, gate, up, down)
        s["shared"] = (_weight(ctx, gen, case["type"], inter, hidden), _weight(ctx, gen, case["type"], inter, hidden), _weight(ctx, gen, case["type"], hidden, inter)) if case["shared"] else None
        s["router"] = _rows(gen, experts, hidden) / math.sqrt(hidden)  # logits N(0, 1)
        s["x"] = _rows(gen, case["m"], hidden, case["dtype"])
    else:
        s["w"] = _weight(ctx, gen, "q8_0", case["rows"], case["cols"])
    return s


def _run_step(s):
    ctx, case = s["ctx"], s["case"]
    dtype, heads, kv_heads = _DTYPES[case["dtype"]], case["hidden"] // case["head_dim"], case["kv"] // case["head_dim"]
    x = ctx.gather_rows(s["embedding"], s["tokens"], dtype=dtype)
    out = {}
    for i, w in enumerate(s["layers"]):
        q, k, v = ctx.rmsnorm_linear_multi(x, w["norm"], 1e-6, [w["q"], w["k"], w["v"]])
        ctx.rope_prefix_qk(q, k, heads, kv_heads, case["head_dim"], s["position"], s["cos"], s["sin"])
        h = ctx.linear_add(q, w["o"], x)
        y = ctx.gated_mlp_add_residual(h, w["gate"], w["up"], w["down"], h)
        out[f"k{i}"], out[f"v{i}"], out[f"y{i}"] = k, v, y
    out["logits"] = ctx.rmsnorm_linear(y, s["norm"], 1e-6, s["head"], out_dtype=torch.float32)
    return out


def run(state):
    s, ctx, case = state, state["ctx"], state["case"]
    kind = case["kind"]
    if kind == "linear":
        return ctx.linear(s["x"], s["w"], residual=s["residual"])
    if kind == "pair":
        return ctx.linear(s["x"], s["up"]), ctx.linear(s["h"], s["down"])
    if kind == "mlp":
        return ctx.gated_mlp_add_residual(s["x"], *s["w"], s["residual"])
    if kind == "step":
        return _run_step(s)
    if kind == "batch":
        if case["host"]:
            ctx.linear_host_batch(s["jobs"])
            return [y for _, _, y in s["jobs"]]
        return ctx.linear_batch(s["jobs"])
    if kind == "moe":
        ids, weights = moe_route(ctx, s["x"], s["router"], case["top_k"])
        y = moe_forward(ctx, s["table"], s["x"], ids, weights, shared=s["shared"])
        return {"y": y, "ids": ids, "weights": weights}
    values = ctx.dequantize(s["w"])
    return {"values": values, "packed": ctx.quantize(ffi.Q4_K, values)}


# ---- what a pass cannot do without
def _packed(kind, rows, cols):
    elems, size = ffi.BLOCK[_TYPES[kind]]
    return rows * cols // elems * size


def work(case):
    kind, m = case["kind"], case.get("m", 1)
    b = _SIZE[case.get("dtype", "f32")]
    if kind == "linear":
        n, k = case["rows"], case["cols"]
        return {"bytes": _packed(case["type"], n, k) + m * (k + n * (2 if case["residual"] else 1)) * b, "flops": 2.0 * m * n * k}
    if kind == "pair":
        n, k = case["ffn"], case["hidden"]
        return {"bytes": 2 * _packed(case["type"], n, k) + 2 * m * (n + k) * b, "flops": 4.0 * m * n * k}
    if kind == "mlp":
        n, k = case["ffn"], case["hidden"]
        return {"bytes": 2 * _packed(case["up"], n, k) + _packed(case["down"], k, n) + 3 * m * k * b, "flops": 6.0 * m * n * k}
    if kind == "step":
        h, kv, f, layers = case["hidden"], case["kv"], case["ffn"], case["layers"]
        total = _packed("q8_0", case["vocab"], h) + m * (_packed("q8_0", 1, h) + case["vocab"] * 4)
        for i in range(layers):
            more = case["more"] if i % 2 else None
            total += 2 * _packed(case["attn"], h, h) + _packed(case["attn"], kv, h) + _packed((case["attn"] if case["attn"] == "q8_0" else more) or case["attn"], kv, h)
            total += 2 * _packed(case["mlp"], f, h) + _packed(more or case["mlp"], h, f) + m * (2 * kv + h) * b
        return {"bytes": total, "flops": 2.0 * m * (layers * (2 * h * h + 2 * kv * h + 3 * f * h) + case["vocab"] * h)}
    if kind == "batch":
        shapes = _shapes(case)
        return {"bytes": sum(_packed(case["type"], n, k) + m * n * b for k, n in shapes) + sum(m * k * b for k in {k for k, _ in shapes}), "flops": sum(2.0 * m * n * k for k, n in shapes)}
    if kind == "moe":
        e, top, h, i = case["experts"], case["top_k"], case["hidden"], case["inter"]
        hit = e * (1.0 - (1.0 - top / e) ** m)  # experts that some token routes to
        per = 2 * _packed(case["type"], i, h) + _packed(case["type"], h, i)
        own = 1 if case["shared"] else 0
        return {"bytes": (hit + own) * per + e * h * 4 + m * (2 * h * b + top * 8), "flops": 6.0 * m * (top + own) * h * i + 2.0 * m * e * h}
    n = case["rows"] * case["cols"]
    return {"bytes": n * (1.0625 + 4 + 0.5625), "flops": 2.0 * n}


def tolerance(case):
    if case["kind"] == "requant":
        return "exact"  # dequantised values and packed bytes are defined bit for bit
    dtype, m = case["dtype"], case["m"]
    if dtype == "bf16":
        rel = 1e-2
    elif dtype == "f16":
        rel = 2e-3
    else:  # f32 rows: decode takes activations as 16-bit integers of a slice, prefill takes f16 operands
        rel = 2e-4 if m <= 16 and case["kind"] != "moe" else 2e-3
    if case["kind"] == "moe":
        return {"rel": rel, "max": 0.2, "differ": 0.005}  # a near-tie in the router moves a token to another expert
    return {"rel": rel}
