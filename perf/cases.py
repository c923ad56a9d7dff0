"""Workloads that stand for the use of this library: what a program that deploys FLUX or SDXL transformers on INT8
Linears has it do, through the public entry points of ``pyraquant_b200``.

Kinds of case
  linear   one ``Int8Linear`` forward (per-token INT8 activations, per-channel INT8 weights, with or without the rank-32
           branch), bf16 for the FLUX layers and fp16 for the SDXL ones.  M runs from one text prompt to the 4K stage.
  block    the Linear path of one FLUX single-stream block: adaLN, the shared-input group (proj_mlp, to_q, to_k, to_v), GELU
           behind proj_mlp, proj_out on the two tensors with gate and residual.  Attention itself is not part of the library;
           the query projection stands in for its output, as in the benchmark.
  g32      one ``Int8LinearG32`` forward (one scale per 32 channels on both operands, the SDXL round-to-nearest arm).
  routed   the routed executor's MLP on a token canvas: gather of the active leaves and their halo, up projection, down
           projection (two weight tiers each), feathered scatter over the cached background.

Sizes are those of the benchmark workloads (FLUX 1K / 2K / 4K stages, SDXL 640- and 1280-channel levels, routed 4K),
the shapes of the tests, and odd ones in between.  Distributions are the configurations' too: activations N(0,1) with
0.5 % of the channels times 20 (N(0,1) for SDXL), weights and low-rank factors N(0,0.02), bias N(0,0.01).
"""
import math

import numpy as np
import torch
import torch.nn as nn

from pyraquant_b200 import int8_exec, ops, routing

RANK = 32
_DT = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # SDXL cross-attention projection of the text tokens (2 prompts x 77): the smallest call, all launch and latency
        {"name": "sdxl_text", "kind": "linear", "M": 154, "K": 640, "N": 1280, "dtype": "fp16", "lowrank": False},
        # FLUX text stream of a double-stream block: 512 tokens through the feed-forward's second Linear
        {"name": "flux_text_down", "kind": "linear", "M": 512, "K": 12288, "N": 3072, "dtype": "bf16", "lowrank": True},
        # FLUX 1K stage, square attention projection (4096 + 512 tokens)
        {"name": "flux_1k_proj", "kind": "linear", "M": 4608, "K": 3072, "N": 3072, "dtype": "bf16", "lowrank": True},
        # FLUX 2K stage, feed-forward's second Linear
        {"name": "flux_2k_down", "kind": "linear", "M": 16896, "K": 12288, "N": 3072, "dtype": "bf16", "lowrank": True},
        # FLUX 4K stage: the headline layers (fused QKV + MLP-in, proj-out)
        {"name": "flux_4k_in", "kind": "linear", "M": 66048, "K": 3072, "N": 21504, "dtype": "bf16", "lowrank": True},
        {"name": "flux_4k_out", "kind": "linear", "M": 66048, "K": 15360, "N": 3072, "dtype": "bf16", "lowrank": True},
        # SDXL 4K stage, 640-channel level, GEGLU up projection on the per-channel deployment arm
        {"name": "sdxl_geglu", "kind": "linear", "M": 65536, "K": 640, "N": 5120, "dtype": "fp16", "lowrank": False},
        # ragged sizes: a crop's token count, feature counts that are no multiple of a tile in either direction
        {"name": "ragged", "kind": "linear", "M": 3001, "K": 1808, "N": 2376, "dtype": "bf16", "lowrank": False},
        # one single-stream block at the 2K stage, the Linear path with the block-level entry points
        {"name": "block_2k", "kind": "block", "M": 16896, "D": 3072, "MLP": 12288},
        # SDXL group-32 arm: 1280-channel GEGLU at the 4K stage, and a 640-channel output projection at a small size
        {"name": "g32_geglu", "kind": "g32", "M": 16384, "K": 1280, "N": 10240, "dtype": "fp16"},
        {"name": "g32_small", "kind": "g32", "M": 1024, "K": 2560, "N": 640, "dtype": "fp16"},
        # routed 4K stage: 16 x 16-token leaves, 30 % active, two-token halo, two weight tiers
        {"name": "routed_4k", "kind": "routed", "side": 256, "leaf": 16, "p": 0.3, "halo": 2, "D": 3072, "MLP": 12288,
         "geometry": 0},
    ]


def _log_int(rng, lo, hi, mult=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / mult)) * mult))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "g32", "g32", "block", "routed"])
    if kind == "linear":
        while True:
            flux = rng.random() < 0.6
            M = _log_int(rng, 64, 66048)
            # feature counts: multiples of 32 (every layer with a low-rank branch), of 16 / 8 otherwise (the ragged ones)
            ragged = rng.random() < 0.3
            if flux:
                K = _log_int(rng, 1024, 15360, 16 if ragged else 128)
                N = _log_int(rng, 1024, 21504, 8 if ragged else 128)
            else:
                K = _log_int(rng, 320, 5120, 16 if ragged else 64)
                N = _log_int(rng, 320, 10240, 8 if ragged else 64)
            if M * K * N <= 66048 * 3072 * 21504 and M * K <= 66048 * 15360 and M * N <= 66048 * 21504:
                break
        return {"kind": "linear", "M": M, "K": K, "N": N, "dtype": "bf16" if flux else "fp16",
                "lowrank": bool(flux and not ragged and rng.random() < 0.7)}
    if kind == "g32":
        return {"kind": "g32", "M": _log_int(rng, 77, 32768), "K": _log_int(rng, 256, 5120, 128),
                "N": _log_int(rng, 320, 10240, 64 if rng.random() < 0.7 else 8), "dtype": "fp16"}
    if kind == "block":
        return {"kind": "block", "M": _log_int(rng, 1024, 20000), "D": rng.choice([1536, 2048, 3072]),
                "MLP": rng.choice([6144, 8192, 12288])}
    side = rng.choice([48, 64, 96, 128, 160, 192, 256])
    return {"kind": "routed", "side": side, "leaf": rng.choice([8, 16]), "p": round(rng.uniform(0.1, 0.6), 2),
            "halo": rng.choice([0, 1, 2, 3]), "D": rng.choice([1536, 3072]), "MLP": rng.choice([6144, 12288]),
            "geometry": rng.randrange(1 << 20)}


# ------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _act(g, M, K, dtype, outliers):
    x = torch.randn(M, K, generator=g, device="cuda")
    if outliers:
        n = max(1, int(round(K * 0.005)))
        x[:, torch.randperm(K, generator=g, device="cuda")[:n]] *= 20.0
    return x.to(dtype)


def _linear(g, K, N, dtype):
    lin = nn.Linear(K, N, bias=True, device="cuda", dtype=dtype)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(N, K, generator=g, device="cuda") * 0.02)
        lin.bias.copy_(torch.randn(N, generator=g, device="cuda") * 0.01)
    return lin


def _factors(g, K, N, dtype):
    A = (torch.randn(K, RANK, generator=g, device="cuda") * 0.02).to(dtype)
    B = (torch.randn(RANK, N, generator=g, device="cuda") * 0.02).to(dtype)
    return A, B


def _layer(g, K, N, dtype, lowrank, cls=int8_exec.Int8Linear):
    return cls(_linear(g, K, N, dtype), device=torch.device("cuda"), lowrank=_factors(g, K, N, dtype) if lowrank else None)


def _plan(case):
    """Route plan of a case: leaves drawn from the case's own geometry number; a leaf above the median score of the
    active ones is high precision, its tokens' rows run against the 8-bit weights."""
    side, leaf = case["side"], case["leaf"]
    n = side // leaf
    r = np.random.default_rng(case["geometry"])
    sel = (r.random((n, n)) < case["p"]).astype(np.float32)
    sel[0, 0] = 1.0                                       # at least one leaf
    scores = r.random((n, n)).astype(np.float32)
    hi = routing.inner_split_median(scores, sel, 1.0)
    tier = routing.leaf_tier_to_token_map(hi, (side, side))
    boxes = routing.leaf_run_boxes(sel, 2 * leaf)
    return routing.build_route_plan((side, side), boxes, case["halo"], token_tier_hi=tier)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "linear":
        dtype = _DT[case["dtype"]]
        layer = _layer(g, case["K"], case["N"], dtype, case["lowrank"])
        return {"kind": kind, "layer": layer, "x": _act(g, case["M"], case["K"], dtype, case["dtype"] == "bf16")}
    if kind == "g32":
        dtype = _DT[case["dtype"]]
        layer = int8_exec.Int8LinearG32(_linear(g, case["K"], case["N"], dtype), device=torch.device("cuda"))
        return {"kind": kind, "layer": layer, "x": _act(g, case["M"], case["K"], dtype, False)}
    if kind == "block":
        M, D, F = case["M"], case["D"], case["MLP"]
        bf = torch.bfloat16
        mlp, q, k, v = (_layer(g, D, n, bf, True) for n in (F, D, D, D))
        out = _layer(g, D + F, D, bf, True)
        group = int8_exec.share_input_quantisation([mlp, q, k, v])
        h = _act(g, M, D, bf, True).reshape(1, M, D)
        shift, scale, gate = ((torch.randn(1, D, generator=g, device="cuda") * 0.3).to(bf) for _ in range(3))
        return {"kind": kind, "layers": (mlp, q, k, v, out), "group": group, "h": h, "shift": shift, "scale": scale,
                "gate": gate}
    bf = torch.bfloat16
    side, D, F = case["side"], case["D"], case["MLP"]
    plan = _plan(case)
    plan.to("cuda")
    up = _layer(g, D, F, bf, True, int8_exec.Int8LinearRouted)
    down = _layer(g, F, D, bf, True, int8_exec.Int8LinearRouted)
    canvas = _act(g, side * side, D, bf, True)
    background = torch.randn(1, side, side, D, generator=g, device="cuda").to(bf)
    return {"kind": kind, "plan": plan, "up": up, "down": down, "canvas": canvas, "background": background,
            "row_idx": plan.to(canvas.device)["row_idx"]}


def run(state):
    kind = state["kind"]
    if kind in ("linear", "g32"):
        return state["layer"](state["x"])
    if kind == "block":
        mlp, q, k, v, out = state["layers"]
        h = state["h"]
        residual = h.clone()                              # the block's input stays usable for the next pass
        z = state["group"].prime_adaln(h, state["scale"], state["shift"])
        ff = mlp.forward_ex(z, ops.EPI_GELU_TANH)
        yq, yk, yv = q(z), k(z), v(z)
        state["group"].clear()
        out.forward_gated_residual(yq, state["gate"], residual, x_more=ff)
        return {"mlp": ff, "q": yq, "k": yk, "v": yv, "hidden": residual}
    plan = state["plan"]
    mid = state["up"].forward_gathered(state["canvas"], state["row_idx"], plan.m_hi)
    y = state["down"].forward_rows(mid, plan.m_hi)
    return {"mid": mid, "rows": y, "fused": routing.fuse_rows(state["background"], y, plan)}


# ------------------------------------------------------------------------------------------------------- bounds
def _linear_work(M, K, N, lowrank, x_bytes=2, out_bytes=2):
    b = x_bytes * M * K + N * K + 8 * N + out_bytes * M * N
    f = 2.0 * M * K * N
    if lowrank:
        b += 2 * RANK * (K + N)
        f += 2.0 * M * RANK * (K + N)
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["M"], case["K"], case["N"], case["lowrank"])
    elif kind == "g32":
        M, K, N = case["M"], case["K"], case["N"]
        b, f = _linear_work(M, K, N, False)
        b += 4 * N * (K // 32) - 4 * N                    # one weight scale per 32 channels instead of one per row
    elif kind == "block":
        M, D, F = case["M"], case["D"], case["MLP"]
        # h in; mlp, q, k, v and the new hidden state out; every weight once
        b = 2 * M * D + 2 * M * (F + 4 * D) + (F + 3 * D) * D + (D + F) * D
        f = 2.0 * M * D * (F + 3 * D) + 2.0 * M * (D + F) * D
        b += 2 * RANK * (4 * D + F + 3 * D + (D + F) + D)
        f += 2.0 * M * RANK * (4 * D + F + 3 * D + (D + F) + D)
    else:
        plan = _plan(case)
        D, F, M, T = case["D"], case["MLP"], plan.n_rows, case["side"] ** 2
        b1, f1 = _linear_work(M, D, F, True, x_bytes=0)
        b2, f2 = _linear_work(M, F, D, True, x_bytes=0)
        uniq = int(np.unique(plan.row_idx).size)
        # canvas rows in (each once), both weight sets of both layers, mid and rows out, background in, fused out
        b = 2 * uniq * D + b1 + b2 + 2 * F * D + 4 * T * D
        f = f1 + f2
    return {"bytes": int(b), "flops": float(f)}


def tolerance(case):
    # 16-bit outputs: the rounding of the result, and of the rank-32 term's 16-bit intermediate
    if case["kind"] in ("linear", "g32"):
        return {"rel": 7e-3 if case["dtype"] == "bf16" else 9e-4}
    # the chained layers quantise a 16-bit intermediate again: a rounding of it moves codes of the next layer
    return {"rel": 8e-3}


# ------------------------------------------------------------------------------------------------------- 64-bit restatement
def _codes(x):
    """Per-row symmetric codes and scales of x (the quantiser is part of the path's definition, its scale is fp32)."""
    amax = x.float().abs().amax(1, keepdim=True).clamp_min(1e-8)
    s = (amax / torch.full_like(amax, 127.0)).double()
    return torch.round(x.double() / s).clamp_(-127, 127), s


def _weight(layer):
    return layer.weight_int8.double() * layer.w_scale.double()[:, None]


def _exact_rows(x, layer, w64, out):
    """Rows of one per-channel Linear in 64 bits, in pieces; the low-rank intermediate is a 16-bit tensor by definition."""
    bias = layer.bias.double()
    for i in range(0, x.shape[0], 8192):
        xs = x[i:i + 8192]
        q, s = _codes(xs)
        y = (q @ w64.t()).mul_(s)
        if layer.lr_A is not None:
            t = (xs.double() @ layer.lr_A.double()).to(xs.dtype)
            y += t.double() @ layer.lr_B.double()
        y += bias
        out[i:i + 8192] = y
    return out


def _exact_linear(x, layer):
    return _exact_rows(x, layer, _weight(layer), torch.empty(x.shape[0], layer.out_features, dtype=torch.float64, device="cuda"))


def exact(case, seed):
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "linear":
        return _exact_linear(st["x"], st["layer"])
    if kind == "g32":
        x, layer = st["x"], st["layer"]
        M, K = x.shape
        wd = (layer.weight_int8.double().reshape(-1, K // 32, 32) * layer.w_scale.double()[..., None]).reshape(-1, K)
        out = torch.empty(M, layer.out_features, dtype=torch.float64, device="cuda")
        for i in range(0, M, 8192):
            xs = x[i:i + 8192]
            q, s = _codes(xs.reshape(-1, 32))
            out[i:i + 8192] = (q * s).reshape(xs.shape) @ wd.t() + layer.bias.double()
        return out
    if kind == "block":
        # what follows the 16-bit activations is their function: a rounding of z moves codes, so the layers' exact
        # values are taken from z rounded as the block's own tensors are
        mlp, q, k, v, out = st["layers"]
        D = case["D"]
        h = st["h"].reshape(-1, D)
        mu = h.double().mean(1, keepdim=True)
        var = (h.double() - mu).pow(2).mean(1, keepdim=True)
        y = ((h.double() - mu) / torch.sqrt(var + 1e-6)).to(h.dtype)
        z = y * (1 + st["scale"]) + st["shift"]
        shape = st["h"].shape[:-1]
        first = _exact_linear(z, mlp).to(h.dtype).double()
        ff = torch.nn.functional.gelu(first, approximate="tanh")
        yq, yk, yv = (_exact_linear(z, m) for m in (q, k, v))
        proj = _exact_linear(torch.cat([yq.to(h.dtype), ff.to(h.dtype)], dim=1), out)
        hidden = h.double() + st["gate"].double() * proj
        return {"mlp": ff.reshape(*shape, -1), "q": yq.reshape(*shape, -1), "k": yk.reshape(*shape, -1),
                "v": yv.reshape(*shape, -1), "hidden": hidden.reshape(*shape, -1)}
    plan, up, down = st["plan"], st["up"], st["down"]
    m_hi = plan.m_hi

    def two_tier(x, layer):
        out = torch.empty(x.shape[0], layer.out_features, dtype=torch.float64, device="cuda")
        _exact_rows(x[:m_hi], layer, _weight(layer), out[:m_hi])
        lo = layer.weight_lo.double() * layer.w_scale_lo.double()[:, None]
        _exact_rows(x[m_hi:], layer, lo, out[m_hi:])
        return out

    mid = two_tier(st["canvas"][st["row_idx"].long()], up)
    y = two_tier(mid.to(torch.bfloat16), down)
    # the blend is the reference's 16-bit arithmetic on 16-bit rows; it has no 64-bit value of its own
    return {"mid": mid, "rows": y, "fused": None}
