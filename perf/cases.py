"""The work that users of this framework have it do, as measurable cases.

Every case is one call (or one short sequence of calls) of the public entry points: whole images through
``BasedXLPipeline``, and the patched operators and matrix products that other code binds one by one
(``basedxl_b200.ops``, ``cascaded_lowp_matmul``, ``BasedXLLowPLinear``).  ``listed()`` holds representative
sizes, ``draw()`` more of the same ranges.
"""
from __future__ import annotations

import math

import torch

from basedxl_b200 import BasedXLConfig, BasedXLPipeline, ops
from basedxl_b200.cascaded_lowp_matmul import cascaded_lowp_matmul
from basedxl_b200.flops import unet_flops
from basedxl_b200.modules.lowp_linear import BasedXLLowPLinear
from basedxl_b200.sdxl_unet import sdxl_config

TEXT_TOKENS, TEXT_DIM, POOLED_DIM = 77, 2048, 1280
UNET_PARAMETERS = 2_567_463_684
HEAD_DIM = 64
GROUPS = 32
# The most that a drawn case may cost, in pixels x steps and in operations: below the largest listed ones.
MAX_PIXEL_STEPS = 4 * 2048 * 2048
MAX_OP_FLOPS = 1.0e12


def listed():
    return [
        # The headline workload: a 1024x1024 image with guidance, denoising steps replayed from CUDA graphs as
        # sample.py runs them.  Ten steps: the length of that program's warm-up image.
        {"name": "image 1024x1024", "kind": "image", "width": 1024, "height": 1024, "steps": 10, "graph": True},
        # The high-resolution workload: 16384-token self-attention, activations larger than L2.
        {"name": "image 2048x2048", "kind": "image", "width": 2048, "height": 2048, "steps": 4, "graph": True},
        # A small image with the pipeline's defaults, which launch every kernel of a step from the host.
        {"name": "image 512x512 eager", "kind": "image", "width": 512, "height": 512, "steps": 4, "graph": False},
        # Key/value projection of the text conditioning (2 x 77 tokens): the smallest linear layer of an image.
        {"name": "linear text k/v", "kind": "linear", "m": 154, "k": 2048, "n": 2560, "bias": False, "residual": False},
        # Feed-forward output projection at the 32x32 level, with the block's bias and residual.
        {"name": "linear ff out", "kind": "linear", "m": 2048, "k": 5120, "n": 1280, "bias": True, "residual": True},
        # The largest of the matmul shapes that the reference's wrapper is used at, through its Linear replacement.
        {"name": "lowp linear 2048x1280x10240", "kind": "lowp_linear", "m": 2048, "k": 1280, "n": 10240, "bias": True},
        # fp32 operands, same wrapper: the split-operand product.
        {"name": "matmul f32 8192x640x640", "kind": "matmul", "m": 8192, "k": 640, "n": 640, "dtype": "f32"},
        # Extents that are no multiple of anything, as a general matmul function meets them.
        {"name": "matmul f16 ragged", "kind": "matmul", "m": 1000, "k": 1003, "n": 1501, "dtype": "f16"},
        # Displaced step on one of four strips: 3x3 convolution with the neighbours' stale boundary rows.
        {"name": "conv strip 2x640x16x64", "kind": "conv", "b": 2, "cin": 640, "cout": 640, "h": 16, "w": 64, "stride": 1,
         "top": True, "bot": True, "time_bias": True, "residual": False},
        # Displaced step on one of four strips: GroupNorm + SiLU with stale moments, which also leaves the boundary
        # rows for the convolution that follows.
        {"name": "norm strip 2x1280x8x32", "kind": "norm", "b": 2, "c": 1280, "h": 8, "w": 32, "mode": "stale", "strips": 4},
        # Displaced step on one of four strips: local queries against the four strips' key/value slots.
        {"name": "attention strip 4x1024", "kind": "attention", "b": 2, "heads": 10, "lq": 1024, "slots": 4, "lslot": 1024},
        # Cross-attention of all 4096 image tokens with the 77 text tokens.
        {"name": "attention text 4096x77", "kind": "attention", "b": 2, "heads": 10, "lq": 4096, "slots": 1, "lslot": 77},
    ]


def _log_int(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _multiple(rng, lo, hi, of):
    """A multiple of ``of`` from lo to hi, spread over its logarithm."""
    return min(hi // of, max(-(-lo // of), int(round(_log_int(rng, lo, hi) / of)))) * of


def draw(rng):
    while True:
        case = _draw(rng)
        if case["kind"] == "image" or work(case)["flops"] <= MAX_OP_FLOPS:
            return case


def _draw(rng):
    # as often as the listed cases have them
    kind = rng.choice(["image"] * 3 + ["linear"] * 2 + ["lowp_linear"] + ["matmul"] * 2 + ["conv", "norm"] + ["attention"] * 2)
    flag = lambda share=0.5: rng.random() < share
    if kind == "image":
        # latents are a multiple of 4 on each side (two down-samplings): image sides a multiple of 32
        w, h = _multiple(rng, 256, 2048, 32), _multiple(rng, 256, 2048, 32)
        steps = min(_log_int(rng, 2, 12), MAX_PIXEL_STEPS // (w * h))
        return {"kind": kind, "width": w, "height": h, "steps": steps, "graph": flag(2 / 3)}
    if kind == "linear":
        return {"kind": kind, "m": _log_int(rng, 2, 32768), "k": _multiple(rng, 320, 5120, 8), "n": _multiple(rng, 320, 10240, 8),
                "bias": flag(), "residual": flag()}
    if kind == "lowp_linear":
        return {"kind": kind, "m": _log_int(rng, 2, 32768), "k": _multiple(rng, 320, 5120, 8), "n": _multiple(rng, 320, 10240, 8), "bias": flag()}
    if kind == "matmul":
        if flag():  # fp32 operands: K and N are multiples of 8
            return {"kind": kind, "m": _log_int(rng, 16, 16384), "k": _multiple(rng, 64, 4096, 8), "n": _multiple(rng, 64, 8192, 8), "dtype": "f32"}
        return {"kind": kind, "m": _log_int(rng, 16, 16384), "k": _log_int(rng, 64, 8192), "n": _log_int(rng, 64, 8192), "dtype": "f16"}
    if kind == "conv":
        stride = rng.choice([1, 1, 1, 2])
        return {"kind": kind, "b": rng.choice([1, 2]), "cin": _multiple(rng, 64, 2560, 64), "cout": _multiple(rng, 64, 1280, 64),
                "h": _multiple(rng, 4, 256, stride), "w": _multiple(rng, 8, 256, stride), "stride": stride,
                "top": flag(), "bot": flag(), "time_bias": flag(), "residual": flag()}
    if kind == "norm":
        return {"kind": kind, "b": rng.choice([1, 2]), "c": GROUPS * rng.choice([10, 20, 30, 40, 60, 80]), "h": _log_int(rng, 4, 256),
                "w": _log_int(rng, 8, 256), "mode": rng.choice(["local", "stale", "sync"]), "strips": rng.choice([2, 4, 8])}
    if flag():  # cross-attention: one slot of text tokens (one or several 77-token prompts)
        slots, lslot = 1, TEXT_TOKENS * rng.choice([1, 1, 2, 3])
        lq = _log_int(rng, 64, 16384)
    else:       # self-attention of a strip: the query count is the slot length
        slots = rng.choice([1, 2, 4, 8])
        lslot = lq = _log_int(rng, 64, 16384 // slots)
    return {"kind": kind, "b": rng.choice([1, 2]), "heads": rng.choice([5, 10, 20]), "lq": lq, "slots": slots, "lslot": lslot}


def _normal(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *shape, scale=1.0, dtype=torch.float16: (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def prepare(case, seed):
    return {"case": case, **_PREPARE[case["kind"]](case, _normal(seed))}


def _prepare_image(c, rn):
    # the loaded model (seeded random weights of the full architecture) and one prompt's embeddings and noise
    pipe = BasedXLPipeline.from_config(BasedXLConfig(width=c["width"], height=c["height"]), seed=0)
    pipe.set_progress_bar_config(disable=True)
    if c["graph"]:
        pipe.unet.enable_cuda_graph()
    return {"pipe": pipe, "prompt": rn(1, TEXT_TOKENS, TEXT_DIM), "negative": rn(1, TEXT_TOKENS, TEXT_DIM), "pooled": rn(1, POOLED_DIM),
            "negative_pooled": rn(1, POOLED_DIM), "latents": rn(1, 4, c["height"] // 8, c["width"] // 8, dtype=torch.float32)}


def _prepare_linear(c, rn):
    m, k, n = c["m"], c["k"], c["n"]
    return {"x": rn(m, k), "weight": rn(n, k, scale=k**-0.5), "bias": rn(n) if c["bias"] else None,
            "residual": rn(m, n) if c["residual"] else None}


def _prepare_lowp_linear(c, rn, wrap=BasedXLLowPLinear):
    layer = torch.nn.Linear(c["k"], c["n"], bias=c["bias"], device="cuda", dtype=torch.float16).requires_grad_(False)
    layer.weight.copy_(rn(c["n"], c["k"], scale=c["k"] ** -0.5))
    if c["bias"]:
        layer.bias.copy_(rn(c["n"]))
    return {"x": rn(c["m"], c["k"]), "layer": wrap(layer)}


def _prepare_matmul(c, rn):
    dtype = {"f16": torch.float16, "f32": torch.float32}[c["dtype"]]
    return {"a": rn(c["m"], c["k"], dtype=dtype), "b": rn(c["k"], c["n"], dtype=dtype)}


def _prepare_conv(c, rn, pack=ops.conv_weight_pack):
    b, ci, co, h, w = c["b"], c["cin"], c["cout"], c["h"], c["w"]
    halo = rn(2, b, 1, w, ci)  # the staging range of a neighbouring strip: [side, image, row, column, channel]
    return {"x": rn(b, h, w, ci), "weight": pack(rn(co, ci, 3, 3, scale=(9 * ci) ** -0.5)), "bias": rn(co),
            "top": halo[1] if c["top"] else None, "bot": halo[0] if c["bot"] else None,
            "time_bias": rn(b, co) if c["time_bias"] else None,
            "residual": rn(b, h // c["stride"], w // c["stride"], co) if c["residual"] else None}


def _prepare_norm(c, rn):
    b, ch, h, w = c["b"], c["c"], c["h"], c["w"]
    x = rn(b, h, w, ch)
    # every strip's published (mean, mean of squares): near those of N(0, 1) activations
    stale = rn(c["strips"], 2, b, GROUPS, scale=0.02, dtype=torch.float32)
    stale[:, 1] += 1.0
    return {"x": x, "gamma": rn(ch, scale=0.2) + 1, "beta": rn(ch, scale=0.2), "peers": list(stale.unbind(0)), "own": c["strips"] // 2,
            "moments": torch.empty(2, b, GROUPS, device="cuda"), "halo": torch.empty(2, b, 1, w, ch, device="cuda", dtype=torch.float16)}


def _prepare_attention(c, rn):
    cq = c["heads"] * HEAD_DIM
    return {"q": rn(c["b"], c["lq"], cq), "slots": [rn(c["b"], c["lslot"], 2 * cq) for _ in range(c["slots"])]}


_PREPARE = {"image": _prepare_image, "linear": _prepare_linear, "lowp_linear": _prepare_lowp_linear, "matmul": _prepare_matmul,
            "conv": _prepare_conv, "norm": _prepare_norm, "attention": _prepare_attention}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "image":
        return state["pipe"](state["prompt"], state["pooled"], state["negative"], state["negative_pooled"],
                             num_inference_steps=c["steps"], guidance_scale=5.0, latents=state["latents"]).latents
    if kind == "linear":
        return ops.linear(state["x"], state["weight"], bias=state["bias"], residual=state["residual"])
    if kind == "lowp_linear":
        return state["layer"](state["x"])
    if kind == "matmul":
        return cascaded_lowp_matmul(state["a"], state["b"])
    if kind == "conv":
        return ops.conv3x3(state["x"], state["weight"], state["bias"], stride=c["stride"], top=state["top"], bot=state["bot"],
                           bias_rows=state["time_bias"], residual=state["residual"])
    if kind == "attention":
        return ops.attention(state["q"], state["slots"], c["heads"])
    return _run_norm(state, c["mode"])


def _run_norm(s, mode):
    if mode == "sync":  # moments first (they are exchanged between the two calls), then the normalisation
        fresh = ops.groupnorm_stats(s["x"], GROUPS, out=s["moments"])
        y = ops.groupnorm_apply(s["x"], GROUPS, 1e-5, s["gamma"], s["beta"], fresh, s["peers"], s["own"], ops.MODE_SYNC, silu=True)
        return {"y": y, "moments": fresh, "halo": ops.halo_pack(y, 1, out=s["halo"])}
    if mode == "local":
        return ops.groupnorm_fused(s["x"], GROUPS, 1e-5, s["gamma"], s["beta"], silu=True)
    y = ops.groupnorm_fused(s["x"], GROUPS, 1e-5, s["gamma"], s["beta"], s["peers"], s["own"], ops.MODE_STALE, silu=True,
                            fresh_out=s["moments"], halo_out=s["halo"])
    return {"y": y, "moments": s["moments"], "halo": s["halo"]}


def exact(case, seed):
    """``run``'s outputs for the same inputs in 64 bits; an image would take minutes."""
    return _EXACT[case["kind"]](case, _normal(seed)) if case["kind"] in _EXACT else None


def _wide(state):
    return {k: v.double() if isinstance(v, torch.Tensor) else v for k, v in state.items()}


def _exact_linear(c, rn):
    s = _wide(_prepare_linear(c, rn))
    y = s["x"] @ s["weight"].T
    if c["bias"]:
        y += s["bias"]
    return y + s["residual"] if c["residual"] else y


def _exact_lowp_linear(c, rn):
    s = _prepare_lowp_linear(c, rn, wrap=lambda layer: layer)
    y = s["x"].double() @ s["layer"].weight.double().T
    return y + s["layer"].bias.double() if c["bias"] else y


def _exact_matmul(c, rn):
    s = _wide(_prepare_matmul(c, rn))
    return s["a"] @ s["b"]


def _exact_conv(c, rn):
    s = _wide(_prepare_conv(c, rn, pack=lambda w: w))
    b, h, w, st = c["b"], c["h"], c["w"], c["stride"]
    x = torch.zeros(b, h + 2, w + 2, c["cin"], device="cuda", dtype=torch.float64)
    x[:, 1:-1, 1:-1] = s["x"]
    if c["top"]:
        x[:, :1, 1:-1] = s["top"]
    if c["bot"]:
        x[:, -1:, 1:-1] = s["bot"]
    y = torch.zeros(b, h // st, w // st, c["cout"], device="cuda", dtype=torch.float64) + s["bias"]
    for ky in range(3):
        for kx in range(3):
            y += x[:, ky : ky + h : st, kx : kx + w : st] @ s["weight"][:, :, ky, kx].T
    if c["time_bias"]:
        y += s["time_bias"][:, None, None, :]
    return y + s["residual"] if c["residual"] else y


def _exact_norm(c, rn):
    raw = _prepare_norm(c, rn)
    peers = torch.stack(raw["peers"]).double()
    s = _wide(raw)
    b, ch, h, w, own = c["b"], c["c"], c["h"], c["w"], s["own"]
    x = s["x"].view(b, h * w, GROUPS, ch // GROUPS)
    fresh = torch.stack([x.mean(dim=(1, 3)), (x * x).mean(dim=(1, 3))])
    full = fresh
    if c["mode"] == "stale":
        full = peers.mean(dim=0) + fresh - peers[own]
    elif c["mode"] == "sync":
        peers[own] = fresh
        full = peers.mean(dim=0)
    var = full[1] - full[0] ** 2
    var = torch.where(var < 0, fresh[1] - fresh[0] ** 2, var)
    n = h * w * ch // GROUPS
    rstd = (var * n / (n - 1) + 1e-5).rsqrt()
    y = ((x - full[0][:, None, :, None]) * rstd[:, None, :, None]).reshape(b, h, w, ch)
    y = torch.nn.functional.silu(y * s["gamma"] + s["beta"])
    return y if c["mode"] == "local" else {"y": y, "moments": fresh, "halo": torch.stack([y[:, :1], y[:, -1:]])}


def _exact_attention(c, rn):
    s = _prepare_attention(c, rn)
    b, lq, heads = c["b"], c["lq"], c["heads"]
    split = lambda t: t.double().unflatten(-1, (heads, HEAD_DIM)).transpose(1, 2)
    k, v = (split(t) for t in torch.cat(s["slots"], dim=1).chunk(2, dim=-1))
    q = split(s["q"])
    out = torch.empty(b, heads, lq, HEAD_DIM, device="cuda", dtype=torch.float64)
    for i in range(0, lq, 1024):  # scores of 1024 queries at a time
        for j in range(b):
            p = (q[j, :, i : i + 1024] @ k[j].transpose(1, 2) * HEAD_DIM**-0.5).softmax(dim=-1)
            out[j, :, i : i + 1024] = p @ v[j]
    return out.transpose(1, 2).reshape(b, lq, heads * HEAD_DIM)


_EXACT = {"linear": _exact_linear, "lowp_linear": _exact_lowp_linear, "matmul": _exact_matmul, "conv": _exact_conv,
          "norm": _exact_norm, "attention": _exact_attention}


def work(case):
    c, kind = case, case["kind"]
    if kind == "image":
        h, w = c["height"] // 8, c["width"] // 8
        # the weights (fp16) are larger than any cache: every step reads them once
        step_bytes = 2.0 * UNET_PARAMETERS + 2 * 4 * h * w * 4 + 4 * 4 * h * w
        return {"bytes": c["steps"] * step_bytes, "flops": c["steps"] * unet_flops(sdxl_config(), h, w, batch=2)}
    if kind in ("linear", "lowp_linear", "matmul"):
        m, k, n = c["m"], c["k"], c["n"]
        size = 4 if c.get("dtype") == "f32" else 2
        extra = n * bool(c.get("bias")) + m * n * bool(c.get("residual"))
        return {"bytes": float(size * (m * k + k * n + m * n + extra)), "flops": 2.0 * m * k * n}
    if kind == "conv":
        b, ci, co, h, w, s = c["b"], c["cin"], c["cout"], c["h"], c["w"], c["stride"]
        out = b * (h // s) * (w // s) * co
        rows = b * w * ci * (c["top"] + c["bot"])
        return {"bytes": 2.0 * (b * h * w * ci + rows + 9 * ci * co + co + b * co * c["time_bias"] + out * (1 + c["residual"])),
                "flops": 2.0 * 9 * ci * out}
    if kind == "norm":
        n = c["b"] * c["c"] * c["h"] * c["w"]
        halo = 0 if c["mode"] == "local" else 2 * c["b"] * c["c"] * c["w"]
        return {"bytes": 2.0 * (2 * n + halo + 2 * c["c"]), "flops": 10.0 * n}
    lkv, cq = c["slots"] * c["lslot"], c["heads"] * HEAD_DIM
    return {"bytes": 2.0 * c["b"] * cq * (2 * c["lq"] + 2 * lkv), "flops": 4.0 * c["b"] * c["lq"] * lkv * cq}


def tolerance(case):
    kind = case["kind"]
    if kind == "image":
        # fp16 rounding (2^-11 per value) of several hundred layers' activations in every step
        return {"rel": 5e-3}
    if kind == "matmul" and case["dtype"] == "f32":
        # 22-bit operands, fp32 accumulation in the tensor core
        return {"rel": 2e-5, "max": 1e-3}
    if kind == "attention":
        # fp16 probabilities and fp16 results
        return {"rel": 2e-3}
    # fp32 accumulation, one rounding to fp16 (at most 2^-11 of the value)
    return {"rel": 1e-3}
