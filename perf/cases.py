"""Measured cases of the routed-MoE path: what a host program runs through the
public entry points, from one decoded token to a 16384-token prefill.

Every case is a dict of plain values; ``kind`` names the entry point:

* ``layer``   ``MoELayer.forward``: the whole layer (router, experts, shared expert).
* ``block``   ``k3_moe_block_forward``: the layer between its RMSNorm and the residual add.
* ``latent``  ``k3_moe_latent_layer_forward``: the reference's real shape, experts on
  a latent vector of width 3584.
* ``store``   ``PartialStore.token``: experts in pinned host memory, a bounded number
  of device slots, one token after the other.
* ``ops_token`` / ``ops_expert`` / ``ops_static``  the reference's operator interface
  (``k3_rocm_*``), called as its engine calls it: one decoded token, one expert's rows
  of a prefill chunk, and a prefill chunk's router and static projections.

Weights and inputs are random with the distributions of the benchmark (synth.py):
activations N(0, 1), router N(0, 0.02), bias by ``bias``, MXFP4 codes uniform with
E8M0 bytes 119..123, int8 uniform with block scales U(1e-4, 1e-3).
"""
import ctypes
import math

import numpy as np
import torch

from moonshine_b200 import _native, ops, replay, synth
from moonshine_b200.layer import MoELayer
from moonshine_b200.store import PartialStore, span_layout

HIDDEN, EXPERTS, TOP_K, SHARED = 7168, 896, 16, 2048
LATENT, LATENT_I = 3584, 3072              # the reference's expert shape
STORE_EXPERTS = 60                         # experts kept in host memory in the store cases (1 GiB)
EPSILON = 1e-5


def listed():
    return [
        # one decoded token: the serving loop's step, bound by the weights it reads and by launches
        {"name": "layer_1", "kind": "layer", "tokens": 1, "bias": "uniform", "form": "swiglu"},
        # a handful of sequences decoded together, with the norm and residual of the engine's block
        {"name": "block_5", "kind": "block", "tokens": 5, "bias": "uniform", "form": "situ"},
        # a larger decode batch
        {"name": "layer_24", "kind": "layer", "tokens": 24, "bias": "zipf", "form": "swiglu"},
        # the 512-token prefill of the benchmark
        {"name": "layer_512", "kind": "layer", "tokens": 512, "bias": "uniform", "form": "swiglu"},
        # the headline workload: layer-major prefill of 8192 tokens, skewed expert load
        {"name": "layer_8192", "kind": "layer", "tokens": 8192, "bias": "zipf", "form": "swiglu"},
        # the stress sweep's largest batch: four experts that every token selects
        {"name": "layer_16384", "kind": "layer", "tokens": 16384, "bias": "hot4", "form": "swiglu"},
        # one decoded token at the reference's own shape
        {"name": "latent_1", "kind": "latent", "tokens": 1, "bias": "uniform", "form": "situ"},
        # a prompt of odd length at the reference's own shape
        {"name": "latent_1021", "kind": "latent", "tokens": 1021, "bias": "zipf", "form": "situ"},
        # decode out of a partially resident table: hits run at once, misses are copied in first
        {"name": "store_8", "kind": "store", "tokens": 8, "slots": 40},
        # a host that composes the token itself from the operator interface (77 calls)
        {"name": "ops_token", "kind": "ops_token", "experts": 896},
        # one expert's rows of a prefill chunk through the operators (8192 tokens: 146 on average)
        {"name": "ops_expert_147", "kind": "ops_expert", "rows": 147},
        # router and static projections of a prefill chunk through the operators
        {"name": "ops_static_200", "kind": "ops_static", "tokens": 200},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(["layer", "block", "latent", "store", "ops_token", "ops_expert", "ops_static"],
                       [9, 4, 6, 1, 1, 2, 1])[0]
    if kind == "store":
        return {"kind": kind, "tokens": rng.randint(2, 8), "slots": rng.randint(24, 48)}
    if kind == "ops_token":
        return {"kind": kind, "experts": rng.randint(64, EXPERTS)}
    if kind == "ops_expert":
        return {"kind": kind, "rows": _log_int(rng, 1, 512)}
    if kind == "ops_static":
        return {"kind": kind, "tokens": _log_int(rng, 2, 512)}
    return {"kind": kind, "tokens": _log_int(rng, 1, 8192 if kind == "latent" else 16384),
            "bias": rng.choice(["uniform", "zipf", "hot4"]), "form": rng.choice(["swiglu", "situ"])}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(g, shape, sigma=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * sigma).to(torch.bfloat16)


def _int8(g, rows, cols):
    return torch.randint(-127, 128, (rows, cols), generator=g, device="cuda", dtype=torch.int8)


def _scales(g, rows, blocks, dtype):
    return (torch.rand((rows, blocks), generator=g, device="cuda") * 9e-4 + 1e-4).to(dtype)


def _codes(g, rows, cols):
    packed = torch.randint(0, 256, (rows, cols // 2), generator=g, device="cuda", dtype=torch.uint8)
    scales = torch.randint(119, 124, (rows, cols // 32), generator=g, device="cuda", dtype=torch.uint8)
    return packed, scales


def _config(case, **sizes):
    """swiglu: the benchmark's layer (Q8 blocks of 32, f16 scales).  situ: the reference's
    activation and static format (Q8 blocks of 128, f32 scales)."""
    if case.get("form", "situ") == "swiglu":
        return synth.baseline_config(bias_mode=case.get("bias", "uniform"), **sizes)
    return synth.baseline_config(bias_mode=case.get("bias", "uniform"), activation=synth.ACT_SITU, q8_block=128,
                                 q8_scale_type=synth.Q8_F32, route_scale=1.0, **sizes)


def _host(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16) if t.dtype is torch.bfloat16 else t.cpu().numpy()


def _q8(g, cfg, rows, cols):
    dtype = torch.float16 if cfg["q8_scale_type"] == synth.Q8_F16 else torch.float32
    return _int8(g, rows, cols), _scales(g, rows, cols // cfg["q8_block"], dtype)


def _static_weights(g, cfg, seed, shared=True):
    """Router and shared expert as MoELayer takes them; the expert tables it fills on the device."""
    w = {"router_weight": _host(_normal(g, (cfg["experts"], cfg["hidden"]), 0.02)),
         "router_bias": synth.router_bias(cfg, seed)}
    if shared:
        for name, (_, _, rows, cols) in synth.shared_tensor_specs(cfg).items():
            q, s = _q8(g, cfg, rows, cols)
            w[name + "_q"], w[name + "_s"] = _host(q), _host(s)
    return w


def prepare(case, seed):
    g = _generator(seed)
    return {"layer": _prepare_layer, "block": _prepare_layer, "latent": _prepare_latent, "store": _prepare_store,
            "ops_token": _prepare_ops_token, "ops_expert": _prepare_ops_expert,
            "ops_static": _prepare_ops_static}[case["kind"]](case, seed, g)


def _prepare_layer(case, seed, g):
    cfg, tokens = _config(case), case["tokens"]
    layer = MoELayer(cfg, _static_weights(g, cfg, seed), seed=seed, max_tokens=tokens if case["kind"] == "layer" else 1)
    state = {"kind": case["kind"], "layer": layer, "x": _normal(g, (tokens, HIDDEN)), "tokens": tokens}
    if case["kind"] == "block":
        state["norm"] = (1.0 + 0.1 * torch.randn(HIDDEN, generator=g, device="cuda")).to(torch.bfloat16)
        state["out"] = torch.empty_like(state["x"])
        state["workspace"] = torch.empty(ops.k3_moe_block_workspace_bytes(layer.desc, tokens), dtype=torch.uint8,
                                         device="cuda")
    return state


def _prepare_latent(case, seed, g):
    tokens = case["tokens"]
    cfg = _config(case, expert_hidden=LATENT_I)
    inner = dict(cfg, hidden=LATENT, shared_hidden=0)
    tables = MoELayer(inner, _static_weights(g, inner, seed, shared=False), seed=seed, max_tokens=1)
    t = {"router_weight": _normal(g, (EXPERTS, HIDDEN), 0.02),
         "router_bias": torch.from_numpy(synth.router_bias(cfg, seed)).cuda(),
         "norm_weight": (1.0 + 0.1 * torch.randn(LATENT, generator=g, device="cuda")).to(torch.bfloat16)}
    for name, (_, _, rows, cols) in synth.shared_tensor_specs(cfg).items():
        t[name + "_q"], t[name + "_s"] = _q8(g, cfg, rows, cols)
    t["down_q"], t["down_s"] = _q8(g, cfg, LATENT, HIDDEN)
    t["up_q"], t["up_s"] = _q8(g, cfg, HIDDEN, LATENT)
    desc = _native.LatentDesc(latent=LATENT, norm_epsilon=EPSILON,
                              **{k: t[k].data_ptr() for k in ("down_q", "down_s", "norm_weight", "up_q", "up_s")})
    ctypes.memmove(ctypes.byref(desc.layer), ctypes.byref(tables.desc), ctypes.sizeof(_native.LayerDesc))
    desc.layer.hidden, desc.layer.shared_hidden = HIDDEN, SHARED
    for name in t:
        if name.startswith(("router_", "shared_")):
            setattr(desc.layer, name, t[name].data_ptr())
    x = _normal(g, (tokens, HIDDEN))
    need = ops.k3_moe_latent_workspace_bytes(desc, tokens)
    return {"kind": "latent", "desc": desc, "tables": tables, "t": t, "x": x, "tokens": tokens,
            "out": torch.empty_like(x), "workspace": torch.empty(need, dtype=torch.uint8, device="cuda")}


def _prepare_store(case, seed, g):
    cfg = _config({}, hidden=LATENT, expert_hidden=LATENT_I, experts=STORE_EXPERTS, shared_hidden=0)
    offsets, total = span_layout(LATENT, LATENT_I)
    spans = torch.empty((STORE_EXPERTS, total), dtype=torch.uint8, pin_memory=True)
    for expert in range(STORE_EXPERTS):
        raw = torch.randint(0, 256, (total,), generator=g, device="cuda", dtype=torch.uint8)
        for scale, end in ((1, 2), (3, 4), (5, 6)):          # w1, w2, w3 scale bytes: 119..123
            part = raw[offsets[scale]:offsets[end] if end < 6 else total]
            part.copy_(119 + part % 5)
        spans[expert].copy_(raw)
    routes = replay.synthetic_routes(case["tokens"], 1, experts=STORE_EXPERTS, seed=seed)
    weights = torch.rand((case["tokens"], TOP_K), generator=g, device="cuda") * 0.1
    return {"kind": "store", "store": PartialStore(cfg, spans, slots=case["slots"]), "experts": routes.experts,
            "x": _normal(g, (case["tokens"], 1, LATENT)), "weights": weights}


def _ops_static_tensors(g, experts):
    t = {"router": _normal(g, (experts, HIDDEN), 0.02),
         "bias": torch.rand(experts, generator=g, device="cuda") * 0.2 - 0.1,
         "norm": (1.0 + 0.1 * torch.randn(LATENT, generator=g, device="cuda")).to(torch.bfloat16)}
    for name, rows, cols in (("down", LATENT, HIDDEN), ("up", HIDDEN, LATENT), ("sh_gate", SHARED, HIDDEN),
                             ("sh_up", SHARED, HIDDEN), ("sh_down", HIDDEN, SHARED)):
        t[name] = (_int8(g, rows, cols), _scales(g, rows, cols // 128, torch.float32))
    return t


def _bf16(*shape):
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda")


def _prepare_ops_token(case, seed, g):
    experts = case["experts"]
    b = {"logits": torch.empty(experts, device="cuda"), "ids": torch.empty(TOP_K, dtype=torch.int32, device="cuda"),
         "weights": torch.empty(TOP_K, device="cuda"), "latent": _bf16(LATENT), "gate": _bf16(LATENT_I),
         "up": _bf16(LATENT_I), "act": _bf16(LATENT_I), "vectors": _bf16(TOP_K, LATENT), "routed": _bf16(LATENT),
         "normed": _bf16(LATENT), "full": _bf16(HIDDEN), "sh_gate": _bf16(SHARED), "sh_up": _bf16(SHARED),
         "sh_act": _bf16(SHARED), "sh_out": _bf16(HIDDEN), "out": _bf16(HIDDEN)}
    slots = [[_codes(g, *shape) for shape in ((LATENT_I, LATENT), (LATENT_I, LATENT), (LATENT, LATENT_I))]
             for _ in range(TOP_K)]
    return {"kind": "ops_token", "experts": experts, "t": _ops_static_tensors(g, experts), "slots": slots,
            "x": _normal(g, (HIDDEN,)), "b": b, "rows": [b["vectors"][r] for r in range(TOP_K)]}


def _prepare_ops_expert(case, seed, g):
    rows, tokens = case["rows"], max(512, case["rows"])
    ids = torch.randperm(tokens, generator=g, device="cuda")[:rows].sort().values.to(torch.int32)
    return {"kind": "ops_expert", "rows": rows, "ids": ids, "x": _normal(g, (tokens, LATENT)),
            "w": [_codes(g, *shape) for shape in ((LATENT_I, LATENT), (LATENT_I, LATENT), (LATENT, LATENT_I))],
            "in": _bf16(rows, LATENT), "gate": _bf16(rows, LATENT_I), "up": _bf16(rows, LATENT_I),
            "act": _bf16(rows, LATENT_I), "down": _bf16(rows, LATENT),
            "out": torch.zeros((tokens, LATENT), dtype=torch.bfloat16, device="cuda")}


def _prepare_ops_static(case, seed, g):
    n = case["tokens"]
    b = {"logits": torch.empty((n, EXPERTS), device="cuda"),
         "ids": torch.empty((n, TOP_K), dtype=torch.int32, device="cuda"),
         "weights": torch.empty((n, TOP_K), device="cuda"), "latent": _bf16(n, LATENT), "routed": _bf16(n, LATENT),
         "normed": _bf16(n, LATENT), "full": _bf16(n, HIDDEN), "sh_gate": _bf16(n, SHARED), "sh_up": _bf16(n, SHARED),
         "sh_act": _bf16(n, SHARED), "sh_out": _bf16(n, HIDDEN), "out": _bf16(n, HIDDEN)}
    return {"kind": "ops_static", "tokens": n, "t": _ops_static_tensors(g, EXPERTS), "x": _normal(g, (n, HIDDEN)),
            "vectors": _normal(g, (n * TOP_K, LATENT)), "b": b}


# --------------------------------------------------------------------- run
def _ok(*results):
    if not all(results):
        raise RuntimeError("an entry point returned false")


def run(state):
    return _RUN[state["kind"]](state)


def _run_layer(s):
    return s["layer"].forward(s["x"])


def _run_block(s):
    _ok(ops.k3_moe_block_forward(s["layer"].desc, s["out"], s["x"], s["norm"], EPSILON, s["tokens"], s["workspace"],
                                 s["workspace"].numel()))
    return s["out"]


def _run_latent(s):
    _ok(ops.k3_moe_latent_layer_forward(s["desc"], s["out"], s["x"], s["tokens"], s["workspace"],
                                        s["workspace"].numel(), None, None))
    return s["out"]


def _run_store(s):
    return [s["store"].token(s["x"][i], s["experts"][i], s["weights"][i])[0] for i in range(len(s["experts"]))]


def _run_ops_token(s):
    t, b, x = s["t"], s["b"], s["x"]
    _ok(ops.k3_rocm_bf16_gemv_f32(b["logits"], t["router"], x, s["experts"], HIDDEN),
        ops.k3_rocm_router_topk_f32(b["ids"], b["weights"], b["logits"], t["bias"], s["experts"], TOP_K, 1.0),
        ops.k3_rocm_q8_128_gemv_bf16(b["latent"], *t["down"], x, LATENT, HIDDEN))
    for row, (w1, w3, w2) in zip(s["rows"], s["slots"]):
        _ok(ops.k3_rocm_mxfp4_gemv_bf16(b["gate"], *w1, b["latent"], LATENT_I, LATENT),
            ops.k3_rocm_mxfp4_gemv_bf16(b["up"], *w3, b["latent"], LATENT_I, LATENT),
            ops.k3_rocm_situ_bf16(b["act"], b["gate"], b["up"], LATENT_I, 4.0, 25.0),
            ops.k3_rocm_mxfp4_gemv_bf16(row, *w2, b["act"], LATENT, LATENT_I))
    _ok(ops.k3_rocm_weighted_sum_bf16(b["routed"], b["vectors"], b["weights"], TOP_K, LATENT),
        ops.k3_rocm_rms_norm_bf16(b["normed"], b["routed"], t["norm"], 1, LATENT, EPSILON),
        ops.k3_rocm_q8_128_gemv_bf16(b["full"], *t["up"], b["normed"], HIDDEN, LATENT),
        ops.k3_rocm_q8_128_gemv_bf16(b["sh_gate"], *t["sh_gate"], x, SHARED, HIDDEN),
        ops.k3_rocm_q8_128_gemv_bf16(b["sh_up"], *t["sh_up"], x, SHARED, HIDDEN),
        ops.k3_rocm_situ_bf16(b["sh_act"], b["sh_gate"], b["sh_up"], SHARED, 4.0, 25.0),
        ops.k3_rocm_q8_128_gemv_bf16(b["sh_out"], *t["sh_down"], b["sh_act"], HIDDEN, SHARED),
        ops.k3_rocm_add_bf16(b["out"], b["full"], b["sh_out"], HIDDEN))
    return [b["ids"], b["weights"], b["vectors"], b["out"]]


def _run_ops_expert(s):
    n, (w1, w3, w2) = s["rows"], s["w"]
    _ok(ops.k3_rocm_gather_rows_bf16(s["in"], s["x"], s["ids"], n, LATENT),
        ops.k3_rocm_mxfp4_gemm_tiled_bf16(s["gate"], *w1, s["in"], n, LATENT_I, LATENT, 32),
        ops.k3_rocm_mxfp4_gemm_tiled_bf16(s["up"], *w3, s["in"], n, LATENT_I, LATENT, 32),
        ops.k3_rocm_situ_bf16(s["act"], s["gate"], s["up"], n * LATENT_I, 4.0, 25.0),
        ops.k3_rocm_mxfp4_gemm_tiled_bf16(s["down"], *w2, s["act"], n, LATENT, LATENT_I, 32),
        ops.k3_rocm_scatter_rows_bf16(s["out"], s["down"], s["ids"], n, LATENT))
    return s["out"]


def _run_ops_static(s):
    n, t, b, x = s["tokens"], s["t"], s["b"], s["x"]
    _ok(ops.k3_rocm_bf16_gemm_tiled_f32(b["logits"], t["router"], x, n, EXPERTS, HIDDEN, 32),
        ops.k3_rocm_router_topk_f32_batch(b["ids"], b["weights"], b["logits"], t["bias"], n, EXPERTS, TOP_K, 1.0),
        ops.k3_rocm_q8_128_gemm_tiled_bf16(b["latent"], *t["down"], x, n, LATENT, HIDDEN, 32),
        ops.k3_rocm_weighted_sum_bf16_batch(b["routed"], s["vectors"], b["weights"], n, TOP_K, LATENT),
        ops.k3_rocm_rms_norm_bf16(b["normed"], b["routed"], t["norm"], n, LATENT, EPSILON),
        ops.k3_rocm_q8_128_gemm_tiled_bf16(b["full"], *t["up"], b["normed"], n, HIDDEN, LATENT, 32),
        ops.k3_rocm_q8_128_gemm_tiled_bf16(b["sh_gate"], *t["sh_gate"], x, n, SHARED, HIDDEN, 32),
        ops.k3_rocm_q8_128_gemm_tiled_bf16(b["sh_up"], *t["sh_up"], x, n, SHARED, HIDDEN, 32),
        ops.k3_rocm_situ_bf16(b["sh_act"], b["sh_gate"], b["sh_up"], n * SHARED, 4.0, 25.0),
        ops.k3_rocm_q8_128_gemm_tiled_bf16(b["sh_out"], *t["sh_down"], b["sh_act"], n, HIDDEN, SHARED, 32),
        ops.k3_rocm_add_bf16(b["out"], b["full"], b["sh_out"], n * HIDDEN))
    return [b["ids"], b["weights"], b["latent"], b["out"]]


_RUN = {"layer": _run_layer, "block": _run_block, "latent": _run_latent, "store": _run_store,
        "ops_token": _run_ops_token, "ops_expert": _run_ops_expert, "ops_static": _run_ops_static}


# -------------------------------------------------------------------- work
def _mx_bytes(rows, cols):
    return rows * cols // 2 + rows * cols // 32


def _q8_bytes(cfg, rows, cols):
    return rows * cols + rows * cols // cfg["q8_block"] * (2 if cfg["q8_scale_type"] == synth.Q8_F16 else 4)


def _touched(case, cfg):
    """Experts that a batch of this size selects, by drawing logits of the same distribution."""
    rng = np.random.default_rng(1)
    bias, hit = synth.router_bias(cfg, 1), np.zeros(EXPERTS, bool)
    sigma = 0.02 * math.sqrt(HIDDEN)
    for at in range(0, case["tokens"], 512):
        n = min(512, case["tokens"] - at)
        choice = 1.0 / (1.0 + np.exp(-rng.normal(0.0, sigma, (n, EXPERTS)))) + bias
        hit[np.argpartition(-choice, TOP_K, axis=1)[:, :TOP_K].ravel()] = True
    return int(hit.sum())


def work(case):
    kind = case["kind"]
    if kind == "store":
        # the 16 experts of every token, read from the slots; what must be copied in depends on the slots' history
        span, n = span_layout(LATENT, LATENT_I)[1], case["tokens"]
        return {"bytes": n * (TOP_K * span + 4 * LATENT), "flops": n * TOP_K * 6 * LATENT * LATENT_I}
    if kind == "ops_expert":
        n, matrix = case["rows"], _mx_bytes(LATENT_I, LATENT)
        return {"bytes": 3 * matrix + n * (4 * LATENT + 4), "flops": n * 6 * LATENT * LATENT_I}
    if kind in ("ops_token", "ops_static"):
        cfg = _config({})
        n, experts = (1, case["experts"]) if kind == "ops_token" else (case["tokens"], EXPERTS)
        params = 2 * LATENT * HIDDEN + 3 * SHARED * HIDDEN
        static = 2 * _q8_bytes(cfg, LATENT, HIDDEN) + 3 * _q8_bytes(cfg, SHARED, HIDDEN) + experts * (2 * HIDDEN + 4)
        flops = 2 * n * (params + experts * HIDDEN)
        if kind == "ops_token":
            return {"bytes": static + TOP_K * 3 * _mx_bytes(LATENT_I, LATENT) + 4 * HIDDEN + 2 * TOP_K * LATENT,
                    "flops": flops + TOP_K * 6 * LATENT * LATENT_I}
        return {"bytes": static + n * (4 * HIDDEN + 2 * TOP_K * LATENT + 2 * LATENT + 8 * TOP_K),
                "flops": flops + 2 * n * TOP_K * LATENT}
    cfg, n = _config(case), case["tokens"]
    width, inner = (LATENT, LATENT_I) if kind == "latent" else (HIDDEN, cfg["expert_hidden"])
    static = EXPERTS * (2 * HIDDEN + 4) + 3 * _q8_bytes(cfg, SHARED, HIDDEN)
    flops = n * (TOP_K * 6 * width * inner + 6 * SHARED * HIDDEN + 2 * EXPERTS * HIDDEN)
    if kind == "latent":
        static += 2 * _q8_bytes(cfg, LATENT, HIDDEN)
        flops += n * 4 * LATENT * HIDDEN
    return {"bytes": _touched(case, cfg) * 3 * _mx_bytes(width, inner) + static + n * 4 * HIDDEN, "flops": flops}


def tolerance(case):
    """bf16 results of sums whose order is free, with intermediate values rounded to bf16: the layer's
    stated 1e-2.  A batch's expert choice is compared exactly (ids are whole numbers)."""
    return {"rel": 1e-2}
