"""The work that a user of this package has it do, as cases that can be timed and compared.

Three paths, each through the entry points an inference engine calls between two attention layers:

``norm``  ``rmsnorm_fp4quant`` / ``add_rmsnorm_fp4quant``: one call per normalisation, a decode step has a few rows and a
          prefill step thousands; scale factors tiled (the GEMM's operand) or row-major.
``gemm``  ``mm_fp4`` / ``nvfp4_gemm`` / ``mxfp8_gemm``: the dense projections.  M is the number of tokens of the step
          (one to a few dozen in decode, thousands in prefill), N and K are the layer's.
``moe``   ``B12xMoEWrapper.run`` with the router inside, or ``topk_route`` + ``b12x_fused_moe``: the routed experts of a
          layer, weights packed once when the model is loaded.

Inputs are drawn as the layers see them: activations and residuals ~ N(0, 1), norm weights 1 + 0.1 N(0, 1), GEMM
operands N(0, 1) quantised with a per-tensor global scale, expert weights N(0, 0.02) quantised per expert, router logits
~ N(0, 1).
"""
import math

import torch

import cutedsl_fully_opensourced_b200 as b200
from cutedsl_fully_opensourced_b200.gemm import quantize_operand
from cutedsl_fully_opensourced_b200.layout import pack_e2m1, swizzle_sf

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "f32": torch.float32}
_DISTINCT_EXPERTS = 8        # weight matrices that are quantised; the other experts hold copies under their own alphas


def listed():
    return [
        # -- norms -------------------------------------------------------------------------------------------------
        # a decode step's residual norm: eight sequences, nothing but latency and launch cost
        {"name": "norm_add_8x7168", "path": "norm", "add": True, "rows": 8, "hidden": 7168, "dtype": "bf16", "sf": "tiled"},
        # a prompt of ordinary length, fp16 model, plain norm, row-major scale factors
        {"name": "norm_4096x5120_fp16", "path": "norm", "add": False, "rows": 4096, "hidden": 5120, "dtype": "fp16",
         "sf": "rows"},
        # a large prefill step: the benchmark's norm configuration
        {"name": "norm_add_8192x7168", "path": "norm", "add": True, "rows": 8192, "hidden": 7168, "dtype": "bf16",
         "sf": "tiled"},
        # -- dense projections -------------------------------------------------------------------------------------
        # decode: sixteen sequences against one weight matrix, a weight stream
        {"name": "gemm_16x8192x8192", "path": "gemm", "kind": "nvfp4", "m": 16, "n": 8192, "k": 8192, "out": "bf16"},
        # a short prompt on a mid-size layer: too few tiles for many waves
        {"name": "gemm_1024x4096x4096_fp16", "path": "gemm", "kind": "nvfp4", "m": 1024, "n": 4096, "k": 4096,
         "out": "fp16"},
        # a mixed batch of prompts: row count ragged, 8-bit operands
        {"name": "gemm_mxfp8_3001x5120x4096", "path": "gemm", "kind": "mxfp8", "m": 3001, "n": 5120, "k": 4096,
         "out": "bf16"},
        # the benchmark's large GEMM
        {"name": "gemm_8192x8192x8192", "path": "gemm", "kind": "nvfp4", "m": 8192, "n": 8192, "k": 8192, "out": "bf16"},
        # -- routed experts ----------------------------------------------------------------------------------------
        # decode of the large configuration: one sequence, and a full decode batch
        {"name": "moe_decode_1", "path": "moe", "tokens": 1, "experts": 256, "hidden": 7168, "inter": 2048, "top_k": 8,
         "route": "inside", "rows": "bf16"},
        {"name": "moe_decode_64", "path": "moe", "tokens": 64, "experts": 256, "hidden": 7168, "inter": 2048, "top_k": 8,
         "route": "inside", "rows": "bf16"},
        # a short prompt: a ragged number of tokens, a few dozen rows per expert, routed by a call of its own
        {"name": "moe_333", "path": "moe", "tokens": 333, "experts": 128, "hidden": 2048, "inter": 768, "top_k": 8,
         "route": "before", "rows": "bf16"},
        # prefill of the small-expert configuration (the benchmark's) and of one with few wide experts
        {"name": "moe_prefill_4096", "path": "moe", "tokens": 4096, "experts": 128, "hidden": 2048, "inter": 768,
         "top_k": 8, "route": "inside", "rows": "bf16"},
        {"name": "moe_wide_4096", "path": "moe", "tokens": 4096, "experts": 32, "hidden": 4096, "inter": 1024, "top_k": 4,
         "route": "before", "rows": "bf16"},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same three paths, over the ranges that the listed ones stand for."""
    path = rng.choice(("norm", "norm", "norm", "gemm", "gemm", "gemm", "gemm", "moe", "moe", "moe"))
    if path == "norm":
        # any number of rows, any hidden size of a real layer: round ones and odd multiples of a scale block
        hidden = 16 * round(_log_uniform(rng, 1024, 8192) / 16)
        if rng.random() < 0.6:
            hidden = 512 * round(hidden / 512)
        rows = min(round(_log_uniform(rng, 1, 16384)), 8192 * 7168 // hidden)
        return {"path": "norm", "add": rng.random() < 0.6, "rows": rows, "hidden": hidden,
                "dtype": rng.choice(("bf16", "bf16", "fp16")), "sf": rng.choice(("tiled", "tiled", "rows", "both"))}
    if path == "gemm":
        # any number of tokens against layers of 1024 to 8192, round or not
        step_n, step_k = rng.choice(((512, 512), (128, 128), (8, 32)))
        return {"path": "gemm", "kind": rng.choice(("nvfp4", "nvfp4", "nvfp4", "nvfp4", "mxfp4", "mxfp8")),
                "m": round(_log_uniform(rng, 1, 8192)),
                "n": max(1024, step_n * round(_log_uniform(rng, 1024, 8192) / step_n)),
                "k": max(1024, step_k * round(_log_uniform(rng, 1024, 8192) / step_k)),
                "out": rng.choice(("bf16", "bf16", "bf16", "fp16", "f32"))}
    if rng.random() < 0.35:
        # the large decode configuration
        shape = {"tokens": round(_log_uniform(rng, 1, 64)), "experts": 256, "hidden": 7168, "inter": 2048, "top_k": 8}
    else:
        experts, hidden, inter, top_k = rng.choice(((128, 2048, 768, 8), (128, 2048, 768, 8), (32, 4096, 1024, 4),
                                                    (64, 2048, 1408, 6), (60, 2560, 1280, 4), (8, 4096, 3584, 2)))
        shape = {"tokens": round(_log_uniform(rng, 1, 4096)), "experts": experts, "hidden": hidden, "inter": inter,
                 "top_k": top_k}
    return {"path": "moe", **shape, "route": rng.choice(("inside", "before")),
            "rows": rng.choice(("bf16", "bf16", "bf16", "f32"))}


# ---------------------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mx_operand(x, kind):
    """[rows, k] f32 -> (operand, tiled ue8m0 scale bytes): one power-of-two scale per 32 elements."""
    rows, k = x.shape
    pad = -k % 32                      # k is a multiple of 32 for e2m1 operands, of 16 for 8-bit ones
    blocks = torch.nn.functional.pad(x, (0, pad)).view(rows, -1, 32)
    largest = 4.0 if kind == "mxfp4" else 256.0        # power of two of the largest value of the type
    exponent = torch.floor(torch.log2(blocks.abs().amax(-1).clamp_min(1e-20) / largest)).clamp(-127, 127)
    scaled = (blocks / torch.exp2(exponent)[..., None]).view(rows, k + pad)[:, :k]
    sf = swizzle_sf((exponent + 127).to(torch.uint8))
    if kind == "mxfp8":
        return scaled.clamp(-448.0, 448.0).to(torch.float8_e4m3fn), sf
    midpoints = torch.tensor((0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0), device=x.device)
    codes = torch.bucketize(scaled.abs(), midpoints).to(torch.uint8)
    return pack_e2m1(codes | ((scaled < 0).to(torch.uint8) << 3)), sf


def _prepare_norm(case, g):
    rows, hidden, dt = case["rows"], case["hidden"], _DTYPES[case["dtype"]]
    x = torch.randn(rows, hidden, generator=g, device="cuda").to(dt)
    residual = torch.randn(rows, hidden, generator=g, device="cuda").to(dt) if case["add"] else None
    weight = (1 + 0.1 * torch.randn(hidden, generator=g, device="cuda")).to(dt)
    # a calibrated per-tensor scale: a normalised value stays below about six
    gs = torch.full((1,), 448.0, dtype=torch.float32, device="cuda")
    return {"x": x, "residual": residual, "weight": weight, "gs": gs}


def _prepare_gemm(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    a, b = (torch.randn(r, k, generator=g, device="cuda") for r in (m, n))
    if case["kind"] == "nvfp4":
        (a, sfa, gsa), (b, sfb, gsb) = quantize_operand(a), quantize_operand(b)
        alpha = torch.full((1,), 1.0 / (gsa * gsb), dtype=torch.float32, device="cuda")
    else:
        (a, sfa), (b, sfb) = _mx_operand(a, case["kind"]), _mx_operand(b, case["kind"])
        alpha = None
    return {"a": a, "b": b, "sfa": sfa, "sfb": sfb, "alpha": alpha, "out": _DTYPES[case["out"]]}


def _prepare_moe(case, g):
    t, e, h, i, k = (case[x] for x in ("tokens", "experts", "hidden", "inter", "top_k"))
    distinct = min(e, _DISTINCT_EXPERTS)
    w1 = 0.02 * torch.randn(distinct, 2 * i, h, generator=g, device="cuda")
    w2 = 0.02 * torch.randn(distinct, h, i, generator=g, device="cuda")
    packed = b200.pack_moe_weights(w1, w2)
    del w1, w2
    which = torch.arange(e, device="cuda") % distinct
    weights = {}
    for name in ("w1", "w2"):
        weights[name + "_weight"] = packed[name + "_weight"][which]
        tiles = packed[name + "_weight_sf"].permute(5, 2, 4, 0, 1, 3).view(torch.uint8)     # expert outermost in memory
        weights[name + "_weight_sf"] = tiles[which].view(torch.float8_e4m3fn).permute(3, 4, 1, 5, 2, 0)
        weights[name + "_alpha"] = packed[name + "_alpha"][which] * (0.8 + 0.4 * torch.rand(e, generator=g, device="cuda"))
    x = torch.randn(t, h, generator=g, device="cuda").to(torch.bfloat16)
    logits = torch.randn(t, e, generator=g, device="cuda")
    hot = torch.rand(t, generator=g, device="cuda") < 0.01          # a few tokens agree on one expert
    logits[:, 0] += 8.0 * hot
    state = {"x": x, "logits": logits, "weights": weights, "experts": e, "top_k": k,
             "rows": torch.float32 if case["rows"] == "f32" else None}
    if case["route"] == "inside":
        state["moe"] = b200.B12xMoEWrapper(e, k, h, i, max_num_tokens=t, slot_rows_dtype=state["rows"])
    return state


def prepare(case, seed):
    g = _generator(seed)
    state = {"norm": _prepare_norm, "gemm": _prepare_gemm, "moe": _prepare_moe}[case["path"]](case, g)
    state["case"] = case
    return state


def run(state):
    case = state["case"]
    if case["path"] == "norm":
        tiled, both = case["sf"] != "rows", case["sf"] == "both"
        if not case["add"]:
            return b200.rmsnorm_fp4quant(state["x"], state["weight"], global_scale=state["gs"], is_sf_swizzled_layout=tiled)
        out = b200.add_rmsnorm_fp4quant(state["x"], state["residual"], state["weight"], global_scale=state["gs"],
                                        is_sf_swizzled_layout=tiled, output_both_sf_layouts=both)
        return (*out, state["residual"])
    if case["path"] == "gemm":
        a, b, sfa, sfb, alpha = (state[n] for n in ("a", "b", "sfa", "sfb", "alpha"))
        if case["kind"] == "nvfp4":
            return b200.mm_fp4(a, b.t(), sfa, sfb, alpha, state["out"])
        if case["kind"] == "mxfp4":
            return b200.nvfp4_gemm(a, b, sfa, sfb, out_dtype=state["out"], sf_vec_size=32)
        return b200.mxfp8_gemm(a, b, sfa, sfb, out_dtype=state["out"])
    w = state["weights"]
    if case["route"] == "inside":
        return state["moe"].run(state["x"], w["w1_weight"], w["w1_weight_sf"], w["w2_weight"], w["w2_weight_sf"],
                                router_logits=state["logits"], w1_alpha=w["w1_alpha"], w2_alpha=w["w2_alpha"])
    ids, scales = b200.topk_route(state["logits"], state["top_k"])
    out = b200.b12x_fused_moe(state["x"], w["w1_weight"], w["w1_weight_sf"], w["w2_weight"], w["w2_weight_sf"], ids, scales,
                              state["experts"], state["top_k"], w1_alpha=w["w1_alpha"], w2_alpha=w["w2_alpha"],
                              slot_rows_dtype=state["rows"])
    return out, ids, scales


def work(case):
    if case["path"] == "norm":
        elements = case["rows"] * case["hidden"]
        per_element = (6.0 if case["add"] else 2.0) + 0.5 + 0.0625 * (2 if case["add"] and case["sf"] == "both" else 1)
        return {"bytes": elements * per_element + 2 * case["hidden"], "flops": 0}
    if case["path"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        operand = {"nvfp4": 0.5 + 1 / 16, "mxfp4": 0.5 + 1 / 32, "mxfp8": 1 + 1 / 32}[case["kind"]]
        return {"bytes": (m + n) * k * operand + m * n * (4 if case["out"] == "f32" else 2), "flops": 2.0 * m * n * k}
    t, e, h, i, k = (case[x] for x in ("tokens", "experts", "hidden", "inter", "top_k"))
    active = e * (1.0 - (1.0 - k / e) ** t)             # experts that are named at least once
    return {"bytes": active * 3 * h * i * (0.5 + 1 / 16) + t * (2 * h * 2 + 4 * e), "flops": 6.0 * t * k * h * i}


def tolerance(case):
    if case["path"] == "norm":
        # the residual is exact; a code or scale byte next to a rounding boundary may move with the order of the f32 sum
        return {"rel": 0.0, "max": 0.0, "differ": 1e-4}
    if case["path"] == "gemm":
        return {"rel": {"bf16": 4e-3, "fp16": 1e-3, "f32": 1e-5}[case["out"]]}
    # activations are re-quantised to four bits between the two GEMMs
    return {"rel": 1e-2, "differ": 1e-4}
