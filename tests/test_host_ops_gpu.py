"""The operators' host path (csrc/ops.cpp): every form it accepts or leaves to the Python statements gives
what those statements give, and what they refuse stays refused."""

import threading

import pytest
import torch

from flydsl_b200 import _lib, pertoken_quant, shuffle_weight
from flydsl_b200.expert_parallel import ExpertParallelMoe
from flydsl_b200.kernels.gemm import mxfp4_preshuffle as mx4
from flydsl_b200.kernels.gemm import mxfp8_preshuffle as mx8
from flydsl_b200.kernels.moe.moe_gemm_2stage import moe_sorting

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


def same(a, b):
    return a.shape == b.shape and a.dtype == b.dtype and torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


def forms(dtype):
    """Orders, strides and alignments: contiguous, 3-D, transposed, sliced, offset by one element, one row, odd K."""
    base = torch.randn(70, 512, device="cuda", dtype=torch.float32).to(dtype)
    flat = torch.randn(64 * 256 + 1, device="cuda", dtype=torch.float32).to(dtype)
    return [base, base.view(7, 10, 512), base.t(), base[:, :256], base[::2], flat[1:].view(64, 256), base[:1], base[0], base[:, :100].contiguous(),
            base[:0], base.requires_grad_(True)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float64])
@pytest.mark.parametrize("qd", [FP8, torch.int8, torch.float8_e5m2])
def test_pertoken_quant_forms(dtype, qd):
    for x in forms(dtype):
        if x.numel() == 0:
            continue
        y, s = pertoken_quant(x, quant_dtype=qd)
        y0, s0 = pertoken_quant(x, quant_dtype=qd, use_kernel=False)
        assert same(y, y0) and same(s, s0)
    with pytest.raises(ValueError):
        pertoken_quant(forms(dtype)[2], quant_dtype=qd, use_kernel=True)  # transposed: the kernel cannot take it
    with pytest.raises(_lib.FlyB200Error):
        pertoken_quant(torch.empty(0, 64, device="cuda"), quant_dtype=torch.int8)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float64])
def test_block_quantiser_forms(dtype):
    for x in forms(dtype):
        if x.shape[-1] % 32 != 0 or x.numel() == 0:
            continue
        for q, ref in ((mx8.per_1x32_f8_quant, mx8.per_1x32_f8_quant_torch), (mx4.per_1x32_f4_quant, mx4.per_1x32_f4_quant_torch)):
            assert all(same(a, b) for a, b in zip(q(x.detach()), ref(x.detach())))
        if x.dim() == 2:
            assert all(same(a, b) for a, b in zip(mx4.per_1x32_f6_quant(x.detach()), mx4.per_1x32_f6_quant_torch(x.detach())))
    with pytest.raises(ValueError):
        mx8.per_1x32_f8_quant(torch.zeros(4, 48, device="cuda"))


def test_scale_image_forms():
    s = torch.randint(0, 256, (200, 64), device="cuda", dtype=torch.uint8)
    want = mx8.shuffle_scale(s)
    wide = torch.zeros(200, 96, device="cuda", dtype=torch.uint8)
    wide[:, 32:] = s
    assert torch.equal(mx8.shuffle_scale(wide[:, 32:]), want) and torch.equal(mx8.shuffle_scale(s.t().contiguous().t()), want)
    for bad in (s[:, :62], s.cpu(), s.view(-1), s.float()):
        with pytest.raises(ValueError):
            mx8.shuffle_scale(bad)


@pytest.mark.parametrize("a_dtype", ["fp8x8", "fp4", "fp6", "fp8"])
def test_block_scaled_gemm_refuses_what_it_refused(a_dtype):
    m, n, k = 20, 256, 512
    x, w = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda")
    if a_dtype == "fp8x8":
        fn, (a, sa), (b, sb) = mx8.compile_mxfp8_preshuffle_gemm(N=n, K=k), mx8.per_1x32_f8_quant(x), mx8.per_1x32_f8_quant(w)
        b = shuffle_weight(b)
    else:
        fn = mx4.compile_mxfp4_preshuffle_gemm(N=n, K=k, a_dtype=a_dtype, b_dtype="fp4")
        a, sa = {"fp4": mx4.per_1x32_f4_quant, "fp6": lambda t: mx4.per_1x32_f6_quant(t)[:2], "fp8": mx8.per_1x32_f8_quant}[a_dtype](x)
        b, sb = mx4.per_1x32_f4_quant(w)
        b = mx4.shuffle_weight_w4(b, for_a_dtype=a_dtype)
    c = torch.zeros(m, n, device="cuda", dtype=torch.bfloat16)
    st = torch.cuda.current_stream()
    good = dict(c=c, a=a.view(torch.uint8), b=b.view(torch.uint8), sa=mx8.shuffle_scale(sa), sb=mx8.shuffle_scale(sb), bias=None, m=m, n=n)
    call = lambda **kw: fn(*{**good, **kw}.values(), st)  # noqa: E731
    call()
    want = c.clone()
    for kw in (dict(c=c[:4]), dict(c=c.float()), dict(c=c.t()), dict(a=good["a"][:4]), dict(a=good["a"].cpu()), dict(b=good["b"].view(-1)[:64]),
               dict(sa=good["sa"][:64]), dict(sb=good["sb"][:64]), dict(bias=torch.zeros(n, device="cuda")), dict(m=-1), dict(n=n + 128),
               dict(a=None)):
        with pytest.raises(ValueError):
            call(**kw)
    call(m=0)
    # another stream than the current one
    side = torch.cuda.Stream()
    side.wait_stream(st)
    out = torch.zeros_like(c)
    fn(out, *list(good.values())[1:], side)
    side.synchronize()
    assert torch.equal(out, want)


def layer_and_inputs(tokens=37, in_dtype="fp8", experts=8, rank=0, world=1):
    d, i, topk = 512, 256, 2
    g = torch.Generator(device="cuda").manual_seed(tokens)
    qd = FP8 if in_dtype == "fp8" else torch.int8
    layer = ExpertParallelMoe(model_dim=d, inter_dim=i, experts=experts, topk=topk, tile_m=16, in_dtype=in_dtype, rank=rank, world=world)
    el = experts // world
    w1, s1 = pertoken_quant(torch.randn(el, 2 * i, d, generator=g, device="cuda"), quant_dtype=qd)
    w2, s2 = pertoken_quant(torch.randn(el, d, i, generator=g, device="cuda"), quant_dtype=qd)
    layer.load_expert_weights(w1, s1, w2, s2)
    x, sx = pertoken_quant(torch.randn(tokens, d, generator=g, device="cuda"), quant_dtype=qd)
    v, ids = torch.topk(torch.rand(tokens, experts, generator=g, device="cuda"), k=topk, dim=1)
    return layer, x, sx, ids, torch.softmax(v, dim=1)


@pytest.mark.parametrize("in_dtype,rank,world", [("fp8", 0, 1), ("int8", 1, 2)])
def test_moe_layer_forms(monkeypatch, in_dtype, rank, world):
    layer, x, sx, ids, wts = layer_and_inputs(in_dtype=in_dtype, rank=rank, world=world)
    want = layer.forward_local(x, sx, ids, wts)
    wide = torch.zeros(x.shape[0], 2 * x.shape[1], device="cuda", dtype=torch.uint8)
    wide[:, : x.shape[1]] = x.view(torch.uint8)
    strided = wide[:, : x.shape[1]].view(x.dtype)
    variants = [(x, sx.view(-1), ids.int(), wts), (x, sx, ids.to(torch.int16), wts.double()), (strided, sx, ids, wts),
                (x, sx, ids.t().contiguous().t(), wts.t().contiguous().t()), (x, sx.view(1, -1), ids, wts)]
    for v in variants:
        assert torch.equal(layer.forward_local(*v), want)
    rounded = layer.forward_local(x, sx.view(1, -1), ids, wts.half())
    assert not torch.equal(rounded, want)
    monkeypatch.setattr(layer, "_forward_native", lambda *a: None)  # the statements one by one
    assert torch.equal(layer.forward_local(x, sx, ids, wts), want)
    assert torch.equal(layer.forward_local(x, sx, ids, wts.half()), rounded)


def test_moe_layer_on_streams_threads_and_in_a_graph():
    layer, x, sx, ids, wts = layer_and_inputs(tokens=64)
    want = layer.forward_local(x, sx, ids, wts)
    torch.cuda.synchronize()
    results = {}

    def work(key):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for _ in range(20):
                results[key] = layer.forward_local(x, sx, ids, wts)
        st.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(results) == 4 and all(torch.equal(r, want) for r in results.values())
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        layer.forward_local(x, sx, ids, wts)
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            y = layer.forward_local(x, sx, ids, wts)
        y.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    with pytest.raises(RuntimeError):  # a shape whose scratch does not exist yet
        big = layer_and_inputs(tokens=640)
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            big[0].forward_local(*big[1:])


def test_routing_table_forms():
    g = torch.Generator(device="cuda").manual_seed(1)
    ids = torch.topk(torch.rand(90, 16, generator=g, device="cuda"), k=4, dim=1).indices
    wts = torch.rand(90, 4, generator=g, device="cuda")
    want = moe_sorting(ids.cpu(), wts.cpu(), num_experts=16, block_size=32)
    for i, w in ((ids, wts), (ids.int(), wts.double()), (ids.to(torch.uint8), wts), (ids.t().contiguous().t(), wts.t().contiguous().t())):
        got = moe_sorting(i, w, num_experts=16, block_size=32)
        used = int(want[3][0])
        assert all(torch.equal(a.cpu(), b) for a, b in zip(got, want)), used


def test_wide_ids_count_as_int32():
    """64-bit ids: the low half counts, in the table and in the masked top-k sum alike."""
    layer, x, sx, ids, wts = layer_and_inputs(tokens=45)
    want = layer.forward_local(x, sx, ids.int(), wts)
    wide = ids.clone()
    wide[::3] += 1 << 32
    wide[1::3] -= 1 << 40
    assert torch.equal(layer.forward_local(x, sx, wide, wts), want)
    for bad in (torch.full_like(ids, (1 << 32) + 8), torch.full_like(ids, 1 << 31)):  # no expert's number, negative
        assert not layer.forward_local(x, sx, bad, wts).any()
    for got, ref in zip(moe_sorting(wide, wts, num_experts=8, block_size=16), moe_sorting(ids.int(), wts, num_experts=8, block_size=16)):
        assert torch.equal(got, ref)
    odd = torch.empty(wide.numel() + 1, device="cuda", dtype=torch.int64)[1:].view_as(wide).copy_(wide)  # a base of 8 bytes
    for got, ref in zip(moe_sorting(odd, wts, num_experts=8, block_size=16), moe_sorting(ids.int(), wts, num_experts=8, block_size=16)):
        assert torch.equal(got, ref)
