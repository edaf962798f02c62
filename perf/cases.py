"""Performance cases of the framework: the calls that a decode or prefill program makes, through the public Python
entry points of `runtime/`, with synthetic weights and activations of the distributions they meet in use.

A case is a dict of plain values.  `op` names the entry point:

  mxfp4_gemv   one MXFP4 matrix times one token                    (N, K)
  fp8_gemv     one FP8 matrix times one token                      (N, K, scale: e8m0 | f32)
  fp8_batched  an FP8 projection for several tokens / groups       (N, K, groups, tokens)
  shared       the FP8 shared expert for one token                 (K, H, O)
  decode       router + routed experts of one layer, one token     (K, H, E, k, score)
  grouped      routed experts of one token, six stacked experts    (K, H, O)
  moe          router + routed experts of one layer, T tokens      (T, K, H, E, k, routing, path)

`layers` (dense ops): how many layers' matrices one pass goes through, one call each, as a token does.
"""
from __future__ import annotations

import importlib
import math

import torch

_PKG = "dsv4-flash-gb10-runtime_b200"
rt = importlib.import_module(_PKG + ".runtime")
qz = importlib.import_module(_PKG + ".runtime.quantize")
_grouped_workspace_bytes = importlib.import_module(_PKG + ".runtime.mxfp4_grouped_gemv_binding").workspace_bytes

DEV = "cuda:0"
TOP_K = 6
EXPERTS = 256


def listed():
    return [
        # The smallest call: one MXFP4 projection of one token (4.5 MB of weights), latency and launch bound.
        {"name": "mxfp4_gemv_2048x4096", "op": "mxfp4_gemv", "N": 2048, "K": 4096, "layers": 1},
        # A ragged one (row count not a multiple of anything, K not a multiple of a warp's 1024), several layers.
        {"name": "mxfp4_gemv_10007x2912", "op": "mxfp4_gemv", "N": 10007, "K": 2912, "layers": 8},
        # FP8 attention projection of one token over several layers: 33.6 MB per call, streamed from HBM.
        {"name": "fp8_gemv_8192x4096", "op": "fp8_gemv", "N": 8192, "K": 4096, "scale": "e8m0", "layers": 8},
        # The query projection wq_b for four tokens in flight (a small decode batch or a drafted run of tokens).
        {"name": "fp8_batched_wq_b_4_tokens", "op": "fp8_batched", "N": 32768, "K": 1024, "groups": 1, "tokens": 4,
         "layers": 8},
        # The shared expert that runs beside the routed ones in every layer, one token.
        {"name": "shared_expert_1_token", "op": "shared", "K": 4096, "H": 2048, "O": 4096, "layers": 8},
        # The decode step itself: one token through one routed layer, top-6 of 256 experts (80 MB of weights).
        {"name": "decode_layer_top6_of_256", "op": "decode", "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "score": "softmax"},
        # The stacked six-expert entry (what an engine that gathers its experts calls) at a width of another model
        # size: neither dimension a power of two.
        {"name": "grouped_6_experts_2880x1440", "op": "grouped", "K": 2880, "H": 1440, "O": 2880},
        # Batched decode: few tokens, nearly every one with experts of its own.
        {"name": "moe_5_tokens", "op": "moe", "T": 5, "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "routing": "uniform", "path": "default"},
        # Batched decode under a hot set: 64 tokens, Zipf(1.1) routing.
        {"name": "moe_64_tokens_zipf", "op": "moe", "T": 64, "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "routing": "zipf", "path": "default"},
        # A prefill chunk of an odd length through the path with fp16 operands.
        {"name": "moe_1003_tokens_fp16_path", "op": "moe", "T": 1003, "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "routing": "uniform", "path": "fp16"},
        # Prefill of 4096 tokens.
        {"name": "moe_4096_tokens", "op": "moe", "T": 4096, "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "routing": "uniform", "path": "default"},
        # The largest: a 16 384-token prefill.
        {"name": "moe_16384_tokens", "op": "moe", "T": 16384, "K": 4096, "H": 2048, "E": EXPERTS, "k": TOP_K,
         "routing": "uniform", "path": "default"},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["mxfp4_gemv", "fp8_gemv", "fp8_batched", "shared", "decode", "grouped", "moe", "moe", "moe", "moe"])
    layers = rng.choice([1, 2, 4, 8])
    if op == "mxfp4_gemv":
        return {"op": op, "N": _log_int(rng, 100, 20000), "K": _log_int(rng, 512, 8192, 32), "layers": layers}
    if op == "fp8_gemv":
        return {"op": op, "N": _log_int(rng, 256, 16384, 128), "K": _log_int(rng, 512, 8192, 128),
                "scale": rng.choice(["e8m0", "e8m0", "f32"]), "layers": layers}
    if op == "fp8_batched":
        groups = rng.choice([1, 1, 1, 2, 8])
        top = 32768 if groups == 1 else 2048
        return {"op": op, "N": _log_int(rng, 512, top, 128), "K": _log_int(rng, 1024, 4096, 128), "groups": groups,
                "tokens": _log_int(rng, 1, 17), "layers": layers}
    if op == "shared":
        K = _log_int(rng, 1024, 4096, 128)
        return {"op": op, "K": K, "H": _log_int(rng, 1024, 2048, 128), "O": K, "layers": layers}
    if op == "decode":
        return {"op": op, "K": rng.choice([4096, 4096, 2048, _log_int(rng, 1024, 4096, 32)]),
                "H": rng.choice([2048, 2048, 1024, _log_int(rng, 512, 2048, 32)]), "E": rng.choice([64, 128, 256]),
                "k": rng.choice([4, 6, 6, 8]), "score": rng.choice(["softmax", "sqrt_softplus"])}
    if op == "grouped":
        K = _log_int(rng, 1024, 4096, 32)
        return {"op": op, "K": K, "H": _log_int(rng, 512, 2048, 32), "O": K}
    K, H = rng.choice([(4096, 2048), (4096, 2048), (2048, 1024), (_log_int(rng, 1024, 4096, 256), _log_int(rng, 512, 2048, 256))])
    path = rng.choice(["default", "default", "default", "fp16"])
    return {"op": op, "T": _log_int(rng, 1, 16384 if path == "default" else 4096), "K": K, "H": H,
            "E": rng.choice([32, 64, 256, 256]), "k": rng.choice([2, 4, 6, 6]),
            "routing": rng.choice(["uniform", "zipf"]), "path": path}


# ---------------------------------------------------------------------------------------------------- inputs

def _mxfp4(n, k, gen):
    return qz.quantize_mxfp4((torch.randn(n, k, generator=gen, device=DEV) * 0.02).to(torch.bfloat16))


def _fp8(n, k, gen, scale="e8m0"):
    return qz.quantize_fp8_block128(torch.randn(n, k, generator=gen, device=DEV) * 0.02, scale)


def _bank(n_experts, K, H, seed):
    """A resident bank of N(0, 0.02) experts.  A few experts are quantised and the others are those with their rows
    rotated, each by another amount: the bytes of real experts at a fraction of the time."""
    few = min(n_experts, 4)
    pool = qz.make_expert_bank(few, K, H, DEV, seed)
    if n_experts == few:
        return pool
    bank = {}
    for name, t in pool.items():
        big = torch.empty((n_experts,) + tuple(t.shape[1:]), dtype=t.dtype, device=DEV)
        for e in range(n_experts):
            r = (e // few) * 37 % t.shape[1]
            big[e, : t.shape[1] - r] = t[e % few, r:]
            if r:
                big[e, t.shape[1] - r:] = t[e % few, :r]
        bank[name] = big
    return bank


def _logits(T, E, routing, gen):
    """Router logits: N(0, 1), or log-probabilities of a Zipf(1.1) law plus Gumbel noise, so that the top k of a row
    are k draws from that law without replacement."""
    if routing == "zipf":
        p = -1.1 * torch.log(torch.arange(1, E + 1, device=DEV, dtype=torch.float32))
        u = torch.rand(T, E, generator=gen, device=DEV).clamp_(1e-7, 1 - 1e-7)
        return (p - torch.log(-torch.log(u))).contiguous()
    return torch.randn(T, E, generator=gen, device=DEV)


def _x(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEV).to(torch.bfloat16)


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    op, c = case["op"], case
    st = {"case": dict(case)}
    if op == "mxfp4_gemv":
        st["w"] = [_mxfp4(c["N"], c["K"], gen) for _ in range(c["layers"])]
        st["x"] = _x(gen, c["K"])
    elif op == "fp8_gemv":
        st["w"] = [_fp8(c["N"], c["K"], gen, c["scale"]) for _ in range(c["layers"])]
        st["x"] = _x(gen, c["K"])
    elif op == "fp8_batched":
        st["w"] = [_fp8(c["groups"] * c["N"], c["K"], gen) for _ in range(c["layers"])]
        st["x"] = _x(gen, c["tokens"], c["groups"] * c["K"])
    elif op == "shared":
        st["w"] = []
        for _ in range(c["layers"]):
            d = {}
            for name, n, k in (("w1", c["H"], c["K"]), ("w3", c["H"], c["K"]), ("w2", c["O"], c["H"])):
                d[name], d[name + "s"] = _fp8(n, k, gen)
            st["w"].append(d)
        st["x"] = _x(gen, c["K"])
    elif op == "decode":
        st["bank"] = _bank(c["E"], c["K"], c["H"], seed)
        st["logits"] = _logits(1, c["E"], "uniform", gen)[0]
        st["x"] = _x(gen, c["K"])
        st["out"] = torch.empty(c["K"], dtype=torch.bfloat16, device=DEV)
        st["workspace"] = torch.empty(rt.decode_workspace_bytes(c["k"], c["H"], c["K"]), dtype=torch.uint8, device=DEV)
    elif op == "grouped":
        b = _bank(6, c["K"], c["H"], seed)
        st["W"] = [{"packed": b[n + "p"], "scale": b[n + "s"]} for n in ("w1", "w3", "w2")]
        st["x"] = _x(gen, c["K"])
        st["r"] = torch.softmax(torch.randn(6, generator=gen, device=DEV), 0)
        st["out"] = torch.empty(c["O"], dtype=torch.bfloat16, device=DEV)
        st["workspace"] = torch.empty(_grouped_workspace_bytes(6, c["H"], c["O"]), dtype=torch.uint8, device=DEV)
    else:
        st["bank"] = _bank(c["E"], c["K"], c["H"], seed)
        st["logits"] = _logits(c["T"], c["E"], c["routing"], gen)
        st["x"] = _x(gen, c["T"], c["K"])
        st["out"] = torch.empty(c["T"], c["K"], dtype=torch.bfloat16, device=DEV)
        st["workspace"] = torch.empty(rt.forward_workspace_bytes(c["T"], c["k"], c["K"], c["H"], c["K"], c["E"]),
                                      dtype=torch.uint8, device=DEV)
    return st


# ------------------------------------------------------------------------------------------------------- a pass

def run(state):
    c, x = state["case"], state.get("x")
    op = c["op"]
    if op == "mxfp4_gemv":
        return [rt.mxfp4_gemv(p, s, x) for p, s in state["w"]]
    if op == "fp8_gemv":
        call = rt.fp8_e4m3_gemv if c["scale"] == "e8m0" else rt.fp8_e4m3_gemv_f32scale
        return [call(p, s, x) for p, s in state["w"]]
    if op == "fp8_batched":
        return [rt.fp8_e4m3_gemv_batched(p, s, x, n_groups=c["groups"]) for p, s in state["w"]]
    if op == "shared":
        return [rt.fp8_shared_swiglu(d, x) for d in state["w"]]
    if op == "decode":
        return rt.moe_decode_layer(state["bank"], state["logits"], x, k=c["k"], score_func=c["score"],
                                   out=state["out"], workspace=state["workspace"])
    if op == "grouped":
        w1, w3, w2 = state["W"]
        return rt.mxfp4_grouped_gemv(w1, w3, w2, None, x, state["r"], out=state["out"], workspace=state["workspace"])
    ids, w = rt.moe_route_topk(state["logits"], k=c["k"], score_func="softmax")
    out = rt.moe_forward(state["bank"], x, ids, w, out=state["out"], workspace=state["workspace"],
                         path=None if c["path"] == "default" else c["path"])
    return {"ids": ids, "weights": w, "out": out}


# ---------------------------------------------------------------------------------------- what a pass cannot avoid

def _experts_used(T, E, k, routing):
    """Expected number of distinct experts of T tokens with k different experts each."""
    if routing == "uniform":
        return E * (1.0 - (1.0 - k / E) ** T)
    p = [1.0 / (e + 1) ** 1.1 for e in range(E)]
    lo, hi = 0.0, 1e6                       # inclusion probability 1 - exp(-c p_e), c such that they add up to k
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        if sum(1.0 - math.exp(-mid * q) for q in p) < k:
            lo = mid
        else:
            hi = mid
    return sum(1.0 - math.exp(-lo * q * T) for q in p)


def work(case):
    c, op = case, case["op"]
    if op == "mxfp4_gemv":
        one = c["N"] * c["K"] * 17 / 32 + 2 * (c["K"] + c["N"])
        return {"bytes": c["layers"] * one, "flops": c["layers"] * 2 * c["N"] * c["K"]}
    if op in ("fp8_gemv", "fp8_batched"):
        g, t = c.get("groups", 1), c.get("tokens", 1)
        scale = 4 if c.get("scale") == "f32" else 1
        one = g * c["N"] * c["K"] * (1 + scale / 16384) + 2 * t * g * (c["K"] + c["N"])
        return {"bytes": c["layers"] * one, "flops": c["layers"] * 2 * g * t * c["N"] * c["K"]}
    K, H = c["K"], c["H"]
    if op == "shared":
        n = 2 * H * K + c["O"] * H
        return {"bytes": c["layers"] * (n * (1 + 1 / 16384) + 2 * (K + c["O"])), "flops": c["layers"] * 2 * n}
    expert = 3 * H * K
    if op == "decode":
        return {"bytes": c["k"] * expert * 17 / 32 + 4 * K + 4 * c["E"], "flops": 2 * c["k"] * expert}
    if op == "grouped":
        return {"bytes": 6 * expert * 17 / 32 + 4 * K, "flops": 12 * expert}
    T = c["T"]
    used = _experts_used(T, c["E"], c["k"], c["routing"])
    return {"bytes": used * expert * 17 / 32 + 4 * T * K + 4 * T * c["E"] + 8 * T * c["k"],
            "flops": 2 * T * c["k"] * expert}


def tolerance(case):
    # Every operator rounds its result to bf16 (relative error up to 2^-9 a value) after FP32 sums; the decode kernels
    # add 8-term fp16 chains inside a 32-element block, the batched layer rounds its SwiGLU intermediate, and the
    # shared expert rounds gate, up and activation to bf16.
    return {"rel": 1e-2, "max": 5e-2}
