"""The work this framework is used for, as cases that can be timed and compared.

Five kinds of pass, each through the public entry points as a program calls them
(launchers built once, specialised with ``flyc.compile`` and kept, weights quantised and
preshuffled once, outputs written into buffers the program owns):

``gemm``      one A8W8 (or 16-bit) preshuffle GEMM whose activations are already quantised:
              a norm or activation kernel upstream wrote the codes and scales.
``linear``    a linear layer on bf16 activations: per-token quantiser, then the GEMM.
``moe``       a mixture-of-experts layer (routing table, gate-up stage, quantiser, down
              stage, top-k sum) through ``ExpertParallelMoe`` on one GPU.
``stages``    the same two stages through ``compile_moe_gemm1`` / ``compile_moe_gemm2``
              with atomic accumulation, the form the reference's own tests drive.
``mx``        a block-scaled linear layer on bf16 activations: per-1x32 quantiser, scale
              image, block-scaled GEMM (MXFP8 x MXFP8, MXFP4 x MXFP4, MXFP6 x MXFP4).

Sizes: the benchmark's configurations and the sizes of the tests, plus ragged ones.
"""

import math

import torch

from flydsl_b200 import compile_preshuffle_gemm, pertoken_quant, shuffle_weight
from flydsl_b200 import compiler as flyc
from flydsl_b200.expert_parallel import ExpertParallelMoe
from flydsl_b200.kernels.gemm import mxfp4_preshuffle as mx4
from flydsl_b200.kernels.gemm import mxfp8_preshuffle as mx8
from flydsl_b200.kernels.moe.moe_gemm_2stage import compile_moe_gemm1, compile_moe_gemm2, moe_sorting

EIGHT_BIT = {"fp8": torch.float8_e4m3fn, "int8": torch.int8}
SIXTEEN_BIT = {"bf16": torch.bfloat16, "fp16": torch.float16}
MX_BITS = {"mxfp8": (8, 8), "mxfp4": (4, 4), "mxfp6": (6, 4)}  # bits of an activation and of a weight code


def _gemm(kind, name, m, n, k, in_dtype="fp8", out_dtype="bf16", epilogue="none"):
    return dict(name=name, kind=kind, m=m, n=n, k=k, in_dtype=in_dtype, out_dtype=out_dtype, epilogue=epilogue)


def _moe(kind, name, tokens, model, inter, experts, topk, tile_m, in_dtype="fp8"):
    return dict(name=name, kind=kind, tokens=tokens, model=model, inter=inter, experts=experts, topk=topk, tile_m=tile_m,
                in_dtype=in_dtype)


def _mx(name, fmt, m, n, k):
    return dict(name=name, kind="mx", fmt=fmt, m=m, n=n, k=k)


def listed():
    return [
        # one token of a decode step through a projection: the smallest call, two launches
        _gemm("linear", "linear_fp8_1x8192x8192", 1, 8192, 8192),
        # a small projection of a batch of 128: the benchmark's first configuration
        _gemm("gemm", "gemm_fp8_128x4096x4096", 128, 4096, 4096),
        # a decode batch of 32 on the weight stream: the benchmark's second configuration
        _gemm("gemm", "gemm_int8_32x8192x8192", 32, 8192, 8192, "int8"),
        # a chunk of ragged prefill with bias and activation, fp16 output, no size a multiple of a tile
        _gemm("linear", "linear_int8_997x10208x5120_gelu", 997, 10208, 5120, "int8", "fp16", "bias_gelu"),
        # unquantised layers: the reference's example, 16-bit operands
        _gemm("gemm", "gemm_fp16_4096x4096x4096", 4096, 4096, 4096, "fp16", "fp16"),
        # prefill of the wide up-projection: the benchmark's third configuration, the largest pass
        _gemm("linear", "linear_fp8_8192x28672x8192", 8192, 28672, 8192),
        # a decode batch through a mixture-of-experts layer
        _moe("moe", "moe_fp8_32tok", 32, 4096, 2048, 8, 2, 16),
        # prefill through the same layer
        _moe("moe", "moe_fp8_4096tok", 4096, 4096, 2048, 8, 2, 128),
        # many small experts, a ragged batch, int8, atomic accumulation, the reference's default block of 64
        _moe("stages", "stages_int8_515tok_16experts", 515, 2048, 1408, 16, 4, 64, "int8"),
        # block-scaled layers at the sizes of the reference's tests: prefill, decode, long K
        _mx("mxfp8_1024x8192x8192", "mxfp8", 1024, 8192, 8192),
        _mx("mxfp4_64x8192x8192", "mxfp4", 64, 8192, 8192),
        _mx("mxfp6_256x4096x14336", "mxfp6", 256, 4096, 14336),
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


MOST_FLOPS = 2.0 * 8192 * 28672 * 8192  # the largest listed case


def draw(rng):
    kind = rng.choice(["gemm", "linear", "gemm", "linear", "moe", "stages", "mx", "mx"])
    if kind in ("gemm", "linear"):
        in_dtype = rng.choice(["fp8", "fp8", "int8"] if kind == "linear" else ["fp8", "fp8", "int8", "fp16", "bf16"])
        m = _log_int(rng, 1, 8192)
        n = _log_int(rng, 1024, 28672, rng.choice([16, 128, 1024]))
        k = _log_int(rng, 1024, 14336, rng.choice([128, 1024]))
        m = max(1, min(m, int(MOST_FLOPS / (2.0 * n * k) / (1 if in_dtype in EIGHT_BIT else 2))))
        return _gemm(kind, "drawn", m, n, k, in_dtype, rng.choice(["bf16", "bf16", "fp16"]),
                     rng.choice(["none", "none", "bias", "bias_relu", "bias_silu", "bias_gelu"]))
    if kind in ("moe", "stages"):
        experts = rng.choice([8, 16, 32])
        tokens = _log_int(rng, 1, 4096)
        topk = rng.choice([2, 4])
        rows = tokens * topk / experts  # routed rows an expert sees
        tile_m = 16 if rows < 24 else 32 if rows < 48 else 64 if rows < 200 else 128
        return _moe(kind, "drawn", tokens, _log_int(rng, 1024, 4096, 256), _log_int(rng, 768, 2048, 128), experts, topk,
                    tile_m, rng.choice(["fp8", "int8"]))
    k = _log_int(rng, 1024, 14336, 256)
    return _mx("drawn", rng.choice(["mxfp8", "mxfp4", "mxfp6"]), _log_int(rng, 1, 1024 * 8192 // k),
               _log_int(rng, 1024, 14336, 128), k)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape, dtype=torch.float32, std=1.0):
        return torch.randn(*shape, generator=g, device=dev, dtype=dtype) * std

    if case["kind"] in ("gemm", "linear"):
        return _prepare_gemm(case, dev, normal)
    if case["kind"] == "mx":
        return _prepare_mx(case, dev, normal)
    return _prepare_moe(case, dev, normal)


def _prepare_gemm(case, dev, normal):
    m, n, k, in_dtype = case["m"], case["n"], case["k"], case["in_dtype"]
    eight = in_dtype in EIGHT_BIT
    out_t = SIXTEEN_BIT[case["out_dtype"]]
    x = normal(m, k, dtype=torch.bfloat16 if eight else SIXTEEN_BIT[in_dtype])
    w = normal(n, k, dtype=torch.bfloat16 if eight else SIXTEEN_BIT[in_dtype], std=0.02)
    launch = compile_preshuffle_gemm(N=n, K=k, tile_m=128, tile_n=128, tile_k=64, in_dtype=in_dtype,
                                     out_dtype=case["out_dtype"], epilogue=case["epilogue"])
    c = torch.empty(m, n, dtype=out_t, device=dev)
    bias = normal(n, dtype=out_t) if case["epilogue"] != "none" else torch.empty(0, dtype=out_t, device=dev)
    if eight:
        w_q, sw = pertoken_quant(w, quant_dtype=EIGHT_BIT[in_dtype])
        x_q, sx = pertoken_quant(x, quant_dtype=EIGHT_BIT[in_dtype])
        w_img, a = shuffle_weight(w_q).view(torch.int8).view(-1), x_q.view(torch.int8).view(-1)
        sx, sw = sx.view(-1), sw.view(-1)
    else:
        w_img, a = shuffle_weight(w).view(-1), x.view(-1)
        sx = sw = torch.empty(0, dtype=torch.float32, device=dev)
    fn = flyc.compile(launch, c.view(-1), a, w_img, sx, sw, bias, m, n, torch.cuda.current_stream(dev))
    return dict(case=case, fn=fn, c=c, x=x, a=a, w=w_img, sx=sx, sw=sw, bias=bias)


def _prepare_moe(case, dev, normal):
    t, d, i, e, topk, tile_m = (case[v] for v in ("tokens", "model", "inter", "experts", "topk", "tile_m"))
    qd = EIGHT_BIT[case["in_dtype"]]
    x_q, sx = pertoken_quant(normal(t, d, dtype=torch.bfloat16), quant_dtype=qd)
    w1_q, sw1 = pertoken_quant(normal(e, 2 * i, d, dtype=torch.bfloat16, std=0.02), quant_dtype=qd)
    w2_q, sw2 = pertoken_quant(normal(e, d, i, dtype=torch.bfloat16, std=0.02), quant_dtype=qd)
    # a router's choice: unequal load over the experts, softmax weights over the chosen ones
    vals, ids = torch.topk(normal(t, e) + normal(e, std=0.5), k=topk, dim=1)
    s = dict(case=case, x=x_q, sx=sx.view(-1), ids=ids.to(torch.int32), wts=torch.softmax(vals, dim=1))
    if case["kind"] == "moe":
        layer = ExpertParallelMoe(model_dim=d, inter_dim=i, experts=e, topk=topk, tile_m=tile_m, in_dtype=case["in_dtype"],
                                  out_dtype="bf16", rank=0, world=1)
        layer.load_expert_weights(w1_q, sw1, w2_q, sw2)
        s["layer"] = layer
        return s
    kw = dict(model_dim=d, inter_dim=i, experts=e, topk=topk, tile_m=tile_m, tile_n=128, tile_k=128, out_dtype="f16",
              in_dtype=case["in_dtype"])
    s["g1"] = flyc.compile(compile_moe_gemm1(**kw, doweight_stage1=False))
    s["g2"] = flyc.compile(compile_moe_gemm2(**kw, doweight_stage2=True, accumulate=True))
    s["w1"], s["w2"] = shuffle_weight(w1_q).view(-1), shuffle_weight(w2_q).view(-1)
    s["sw1"], s["sw2"] = sw1.view(-1), sw2.view(-1)
    s["h"] = torch.empty(t, topk, i, dtype=torch.float16, device=dev)
    s["y"] = torch.empty(t, d, dtype=torch.float16, device=dev)
    return s


def _mx_quant(fmt, x):
    """Activation codes and row-major E8M0 scales of one format."""
    if fmt == "mxfp8":
        return mx8.per_1x32_f8_quant(x)
    if fmt == "mxfp4":
        return mx4.per_1x32_f4_quant(x)
    return mx4.per_1x32_f6_quant(x)[:2]


def _prepare_mx(case, dev, normal):
    m, n, k, fmt = case["m"], case["n"], case["k"], case["fmt"]
    x = normal(m, k, dtype=torch.bfloat16)
    w = normal(n, k, dtype=torch.bfloat16, std=0.02)
    if fmt == "mxfp8":
        launch = mx8.compile_mxfp8_preshuffle_gemm(N=n, K=k)
        w_q, sw = mx8.per_1x32_f8_quant(w)
        w_img, sw_img = shuffle_weight(w_q), mx8.shuffle_scale(sw)
    else:
        a_dtype = "fp4" if fmt == "mxfp4" else "fp6"
        launch = mx4.compile_mxfp4_preshuffle_gemm(N=n, K=k, a_dtype=a_dtype, b_dtype="fp4")
        w_q, sw = mx4.per_1x32_f4_quant(w)
        w_img, sw_img = mx4.shuffle_weight_w4(w_q, for_a_dtype=a_dtype), mx4.shuffle_scale_w4(sw)
    return dict(case=case, fn=flyc.compile(launch), x=x, w=w_img.view(torch.uint8).view(-1), sw=sw_img,
                c=torch.empty(m, n, dtype=torch.bfloat16, device=dev))


def run(state):
    case = state["case"]
    stream = torch.cuda.current_stream()
    if case["kind"] in ("gemm", "linear"):
        a, sx, c = state["a"], state["sx"], state["c"]
        if case["kind"] == "linear":
            a, sx = pertoken_quant(state["x"], quant_dtype=EIGHT_BIT[case["in_dtype"]])
            a, sx = a.view(torch.int8).view(-1), sx.view(-1)
        state["fn"](c.view(-1), a, state["w"], sx, state["sw"], state["bias"], case["m"], case["n"], stream)
        return c
    if case["kind"] == "mx":
        c = state["c"]
        a, sa = _mx_quant(case["fmt"], state["x"])
        sa_img = mx8.shuffle_scale(sa) if case["fmt"] == "mxfp8" else mx4.shuffle_scale_w4(sa)
        state["fn"](c.view(-1), a.view(torch.uint8).view(-1), state["w"], sa_img, state["sw"], None, case["m"], case["n"], stream)
        return c
    if case["kind"] == "moe":
        return state["layer"].forward(state["x"], state["sx"], state["ids"], state["wts"])
    t, d, i = case["tokens"], case["model"], case["inter"]
    ids, wts, e_ids, n_valid = moe_sorting(state["ids"], state["wts"], num_experts=case["experts"], block_size=case["tile_m"])
    blocks = e_ids.numel()
    h, y = state["h"], state["y"]
    state["g1"](h, state["x"].view(-1), state["w1"], state["sx"], state["sw1"], ids, e_ids, wts, n_valid, t, i, d, blocks, stream)
    a2, sa2 = pertoken_quant(h, quant_dtype=EIGHT_BIT[case["in_dtype"]])
    y.zero_()
    state["g2"](y, a2.view(-1), state["w2"], sa2.view(-1), state["sw2"], ids, e_ids, wts, n_valid, t, d, i, blocks, stream)
    return y


def work(case):
    """Inputs read once, outputs written once (weights of the experts that can be hit), products of the routed rows."""
    if case["kind"] in ("gemm", "linear"):
        m, n, k = case["m"], case["n"], case["k"]
        eight = case["in_dtype"] in EIGHT_BIT
        w_e = 1 if eight else 2
        a_e = 2 if case["kind"] == "linear" else w_e
        scales = (4 * n + (4 * m if case["kind"] == "gemm" else 0)) if eight else 0
        bias = 2 * n if case["epilogue"] != "none" else 0
        return {"bytes": m * k * a_e + n * k * w_e + 2 * m * n + scales + bias, "flops": 2.0 * m * n * k}
    if case["kind"] == "mx":
        m, n, k = case["m"], case["n"], case["k"]
        w_bits = MX_BITS[case["fmt"]][1]
        return {"bytes": 2 * m * k + n * k * w_bits // 8 + n * k // 32 + 2 * m * n, "flops": 2.0 * m * n * k}
    t, d, i, e, topk = (case[v] for v in ("tokens", "model", "inter", "experts", "topk"))
    used = min(e, t * topk)
    return {"bytes": t * d + 4 * t + 8 * t * topk + used * (3 * i * d + 4 * (2 * i + d)) + 2 * t * d,
            "flops": 2.0 * t * topk * 3 * i * d}


# Four times the distance of the listed cases from the same operands multiplied and summed in
# float64.  A product with exact or fp32 accumulation differs from that by the rounding of its
# output (bf16: 1.66e-3 of the norm, 3.9e-3 of one value; fp16: an eighth).  The two stages of a
# mixture of experts also round and quantise in between, where a code next to a rounding boundary
# may fall either way (bf16: 2.4e-3 and 2.5e-2; fp16: 3.9e-4 and 2.7e-3).
def tolerance(case):
    if case["kind"] == "moe":
        return {"rel": 1e-2, "max": 1e-1}
    if case["kind"] == "stages":
        return {"rel": 1.6e-3, "max": 1.1e-2}
    if case.get("out_dtype") == "fp16":
        return {"rel": 8.3e-4, "max": 2e-3}
    return {"rel": 6.7e-3, "max": 1.6e-2}
