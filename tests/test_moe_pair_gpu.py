"""The grouped GEMM on CTA pairs (FLYB200_MOE_KERNEL=3) against the form with one CTA per 128-row item (2): the same
products in the same order, so the same bits."""

import pytest
import torch

from flydsl_b200 import _lib, shuffle_weight
from flydsl_b200.kernels.moe.moe_gemm_2stage import compile_moe_gemm1, compile_moe_gemm2, moe_sorting
from oracle import moe_oracle

pytestmark = pytest.mark.gpu

OUT_T = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def stage(number, codes, scales, w, sw, routing, *, model, inter, experts, topk, tile_m, in_dtype, out_dtype, accumulate, n_valid=None):
    ids, wts, e_ids, post = routing
    tokens = codes.shape[0] if number == 1 else codes.shape[0] // topk
    rows, dim = (tokens * topk, inter) if number == 1 else (tokens if accumulate else tokens * topk, model)
    out = torch.zeros(rows + 5, dim, dtype=OUT_T[out_dtype], device="cuda")
    out[rows:] = 7.0
    kw = dict(model_dim=model, inter_dim=inter, experts=experts, topk=topk, tile_m=tile_m, tile_n=128, tile_k=128, in_dtype=in_dtype,
              out_dtype=out_dtype)
    exe = compile_moe_gemm1(**kw, doweight_stage1=False) if number == 1 else compile_moe_gemm2(**kw, doweight_stage2=True, accumulate=accumulate)
    n, k = (inter, model) if number == 1 else (model, inter)
    exe(out, codes.view(-1), w, scales, sw, ids, e_ids, wts, post if n_valid is None else n_valid, tokens, n, k, e_ids.numel(),
        torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    assert bool((out[rows:] == 7.0).all())
    return out


def inputs(tokens, model, inter, experts, topk, in_dtype, skew, seed):
    g = torch.Generator().manual_seed(seed)
    draw = lambda *s: (torch.randint(-127, 128, s, generator=g, dtype=torch.int8).cuda() if in_dtype == "int8"  # noqa: E731
                       else torch.randn(*s, generator=g).cuda().to(torch.float8_e4m3fn))
    scale = lambda n: (torch.rand(n, generator=g) / 64).cuda()  # noqa: E731
    ids = torch.topk(torch.randn(tokens, experts, generator=g) + skew * torch.arange(experts), k=topk, dim=1).indices.int().cuda()
    wts = torch.rand(tokens, topk, generator=g).cuda()
    return dict(ids=ids, wts=wts, x=draw(tokens, model), sx=scale(tokens), a2=draw(tokens * topk, inter), sa2=scale(tokens * topk),
                w1=shuffle_weight(draw(experts, 2 * inter, model)).view(-1), sw1=scale(experts * 2 * inter),
                w2=shuffle_weight(draw(experts, model, inter)).view(-1) if inter % 128 == 0 else None, sw2=scale(experts * model))


@pytest.mark.parametrize(
    "tokens,model,inter,experts,topk,tile_m,in_dtype,skew",
    [
        (1, 256, 128, 4, 1, 64, "fp8", 0.0),  # one row, one tile
        (400, 2944, 1408, 7, 2, 64, "fp8", 0.0),  # 77 items in the gate-up stage: the last three in four strips each
        (1500, 1024, 1424, 4, 2, 256, "int8", 0.1),  # a partial channel tile (gate-up stage alone); experts of several tiles
        (700, 512, 640, 9, 3, 128, "int8", 0.4),  # unequal experts: half-filled last tiles, empty experts
        (90, 256, 384, 40, 2, 64, "fp8", 0.0),  # a tile of few rows per expert
        (300, 2688, 1024, 10, 1, 64, "int8", 0.0),  # 110 items in the down stage: 36 of them in two strips; a half channel pair
    ],
)
def test_pairs_equal_single_ctas(monkeypatch, tokens, model, inter, experts, topk, tile_m, in_dtype, skew):
    d = inputs(tokens, model, inter, experts, topk, in_dtype, skew, seed=tokens)
    routing = moe_sorting(d["ids"], d["wts"], num_experts=experts, block_size=tile_m)
    kw = dict(model=model, inter=inter, experts=experts, topk=topk, tile_m=tile_m, in_dtype=in_dtype)
    # (accumulation of one route per token alone has a fixed order)
    stages = [(1, "bf16", False), (1, "f16", False), (2, "bf16", False), (2, "f16", False)]
    if topk == 1:
        stages += [(2, "f32", True), (2, "bf16", True)]
    for number, out_dtype, accumulate in stages:
        if number == 2 and d["w2"] is None:
            continue
        args = (number, d["x"], d["sx"], d["w1"], d["sw1"]) if number == 1 else (number, d["a2"], d["sa2"], d["w2"], d["sw2"])
        got = []
        for form in "23":
            monkeypatch.setenv("FLYB200_MOE_KERNEL", form)
            got.append(stage(*args, routing, **kw, out_dtype=out_dtype, accumulate=accumulate))
        assert torch.equal(got[0], got[1]), (number, out_dtype)


def test_blocks_without_expert_and_a_shorter_list(monkeypatch):
    """A run of blocks that loses one in the middle, blocks of no expert at either end, and a list cut short inside a tile."""
    tokens, model, inter, experts, topk, tile_m = 600, 512, 256, 3, 2, 64
    d = inputs(tokens, model, inter, experts, topk, "int8", 0.0, seed=3)
    ids, wts, e_ids, post = moe_sorting(d["ids"], d["wts"], num_experts=experts, block_size=tile_m)
    e_ids = e_ids.clone()
    e_ids[0] = e_ids[3] = -1
    e_ids[int(post[0]) // tile_m - 1] = experts  # out of range: no expert either
    cut = torch.tensor([int(post[0]) // tile_m // 2 * tile_m + tile_m], dtype=torch.int32, device="cuda")
    for n_valid in (None, cut):
        got = []
        for form in "23":
            monkeypatch.setenv("FLYB200_MOE_KERNEL", form)
            got.append(stage(2, d["a2"], d["sa2"], d["w2"], d["sw2"], (ids, wts, e_ids, post), model=model, inter=inter, experts=experts,
                             topk=topk, tile_m=tile_m, in_dtype="int8", out_dtype="bf16", accumulate=False, n_valid=n_valid))
        assert torch.equal(got[0], got[1])
        assert int((got[0] == 0).all(dim=1).sum()) > 0  # some routes had no expert


def test_longer_lists_than_the_pair_form_holds(monkeypatch):
    """7200 experts of one route each are 7200 routing blocks; the pair form's list has room for 7168, so the request for it
    runs one CTA per item."""
    experts, model, inter = 7200, 16, 128
    d = moe_oracle.make_inputs(experts, 128, inter, 2, 1, "int8", seed=5)  # activations and scales of the second stage
    g = torch.Generator().manual_seed(5)
    ids = torch.randperm(experts, generator=g).view(-1, 1).int()
    w2, sw2 = torch.randint(-127, 128, (experts, model, inter), generator=g, dtype=torch.int8), torch.rand(experts, model, 1, generator=g) / 64
    routing = moe_sorting(ids.cuda(), d["topk_weights"].cuda(), num_experts=experts, block_size=64)
    assert routing[2].numel() > 7168 and int(routing[3][0]) == 64 * experts
    monkeypatch.setenv("FLYB200_MOE_KERNEL", "3")
    got = stage(2, d["a2_q"].view(experts, inter).cuda(), d["scale_a2"].reshape(-1).cuda(), shuffle_weight(w2.cuda()).view(-1), sw2.view(-1).cuda(),
                routing, model=model, inter=inter, experts=experts, topk=1, tile_m=64, in_dtype="int8", out_dtype="f32", accumulate=True)
    args = (d["scale_a2"], sw2, ids.long(), d["topk_weights"], model)
    ref, size = moe_oracle.moe_gemm2(d["a2_q"], w2, *args), moe_oracle.moe_gemm2(d["a2_q"].int().abs(), w2.int().abs(), *args)
    # the kernel's sum of integers is exact; the oracle rounds both operands, 128 products and sums; four roundings of factors here
    assert bool(((got[:experts].cpu() - ref).abs() <= (2 * 128 + 6) * 2**-24 * size).all())
