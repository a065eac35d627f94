"""Without the host extension (no compiler, other headers) every operator still runs, on the same kernels, and
objects that are not tensors but have a device address are still taken."""

import pytest
import torch

from flydsl_b200 import _lib, compile_preshuffle_gemm, host_statements, pertoken_quant, shuffle_weight
from flydsl_b200 import compiler as flyc
from flydsl_b200.expert_parallel import ExpertParallelMoe
from flydsl_b200.kernels.gemm import mxfp4_preshuffle as mx4
from flydsl_b200.kernels.gemm import mxfp8_preshuffle as mx8
from flydsl_b200.kernels.moe.moe_gemm_2stage import compile_moe_gemm1, moe_sorting
from flydsl_b200.utils import pertoken_quant_kernel


@pytest.fixture
def no_extension(monkeypatch):
    def refuse(force=False):
        raise RuntimeError("no compiler")

    monkeypatch.setattr(_lib, "_ops", None)
    monkeypatch.setattr(_lib._build, "build_ops", refuse)
    with pytest.warns(RuntimeWarning, match="no compiler"):
        assert _lib.ops() is host_statements


def test_the_statements_have_every_function(no_extension, monkeypatch):
    monkeypatch.undo()
    names = [n for n in dir(_lib.ops()) if not n.startswith("_")]
    assert "moe_layer" in names and all(callable(getattr(host_statements, n, None)) for n in names)


def outputs():
    g = torch.Generator(device="cuda").manual_seed(7)
    dev, st = torch.device("cuda", 0), torch.cuda.current_stream()
    m, n, k = 37, 512, 1024
    x = torch.randn(m, k, generator=g, device=dev, dtype=torch.float32).to(torch.bfloat16)
    w = torch.randn(n, k, generator=g, device=dev, dtype=torch.float32).to(torch.bfloat16)
    out = []
    for qd, name in ((torch.float8_e4m3fn, "fp8"), (torch.int8, "int8")):
        (a, sa), (b, sb) = pertoken_quant(x, quant_dtype=qd), pertoken_quant(w, quant_dtype=qd)
        launch = compile_preshuffle_gemm(N=n, K=k, tile_m=64, tile_n=128, tile_k=128, in_dtype=name)
        c, none = torch.empty(m, n, device=dev, dtype=torch.bfloat16), torch.empty(0, device=dev, dtype=torch.bfloat16)
        args = (c.view(-1), a.view(torch.int8).view(-1), shuffle_weight(b).view(torch.int8).view(-1), sa.view(-1), sb.view(-1), none, m, n, st)
        flyc.compile(launch, *args)(*args)
        out += [a, sa, c]
    kw = dict(model_dim=512, inter_dim=256, experts=8, topk=2, tile_m=16, in_dtype="fp8")
    (w1, s1), (w2, s2) = (pertoken_quant(torch.randn(8, r, c_, generator=g, device=dev), quant_dtype=torch.float8_e4m3fn)
                          for r, c_ in ((512, 512), (512, 256)))
    xm, sm = pertoken_quant(torch.randn(20, 512, generator=g, device=dev), quant_dtype=torch.float8_e4m3fn)
    v, ids = torch.topk(torch.rand(20, 8, generator=g, device=dev), k=2, dim=1)
    for od in ("bf16", "f32"):
        layer = ExpertParallelMoe(**kw, out_dtype=od, rank=0, world=1)
        layer.load_expert_weights(w1, s1, w2, s2)
        out.append(layer.forward_local(xm, sm, ids, v))
    table = moe_sorting(ids, v, num_experts=8, block_size=16)
    g1 = compile_moe_gemm1(**kw, tile_n=128, tile_k=128, doweight_stage1=True, out_dtype="bf16")
    y = torch.zeros(20, 2, 256, device=dev, dtype=torch.bfloat16)
    g1(y, xm, shuffle_weight(w1), sm.view(-1), s1.view(-1), table[0], table[2], table[1], table[3], 20, 256, 512, int(table[2].numel()), st)
    out += [*table, y]
    for a_dtype in ("fp8x8", "fp4", "fp6", "fp8"):
        if a_dtype == "fp8x8":
            fn, (a, sa), (b, sb) = mx8.compile_mxfp8_preshuffle_gemm(N=n, K=k), mx8.per_1x32_f8_quant(x), mx8.per_1x32_f8_quant(w)
            b = shuffle_weight(b)
        else:
            fn = mx4.compile_mxfp4_preshuffle_gemm(N=n, K=k, a_dtype=a_dtype, b_dtype="fp4")
            a, sa = {"fp4": mx4.per_1x32_f4_quant, "fp6": lambda t: mx4.per_1x32_f6_quant(t)[:2], "fp8": mx8.per_1x32_f8_quant}[a_dtype](x)
            b, sb = mx4.per_1x32_f4_quant(w)
            b = mx4.shuffle_weight_w4(b, for_a_dtype=a_dtype)
        c = torch.zeros(m, n, device=dev, dtype=torch.bfloat16)
        fn(c, a.view(torch.uint8), b.view(torch.uint8), mx8.shuffle_scale(sa), mx8.shuffle_scale(sb), None, m, n, st)
        out += [a, sa, c]
    return out


def same(a, b):
    return a.shape == b.shape and a.dtype == b.dtype and torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


@pytest.mark.gpu
def test_same_results_without_the_extension(request):
    want = outputs()
    request.getfixturevalue("no_extension")
    got = outputs()
    assert len(got) == len(want) and all(same(a, b) for a, b in zip(got, want))


class Buffer:
    """A device buffer of another library."""

    def __init__(self, t):
        self.t, self.device = t, t.device

    def data_ptr(self):
        return self.t.data_ptr()

    def numel(self):
        return self.t.numel()


@pytest.mark.gpu
def test_buffers_that_are_not_tensors():
    n, k, m = 256, 512, 20
    g = torch.Generator(device="cuda").manual_seed(1)
    (a, sa), (b, sb) = (pertoken_quant(torch.randn(r, k, generator=g, device="cuda"), quant_dtype=torch.float8_e4m3fn) for r in (m, n))
    c = torch.zeros(2, m * n, device="cuda", dtype=torch.bfloat16)
    st = torch.cuda.current_stream()
    rest = [a.view(torch.int8).view(-1), shuffle_weight(b).view(torch.int8).view(-1), sa.view(-1), sb.view(-1), torch.empty(0, device="cuda")]
    fn = flyc.compile(compile_preshuffle_gemm(N=n, K=k, tile_m=64, tile_n=128, tile_k=128), c[0], *rest, m, n, st)
    fn(c[0], *rest, m, n, st)
    fn(Buffer(c[1]), *[Buffer(t) for t in rest], m, n, st)
    assert torch.equal(c[0], c[1]) and bool(c[0].any())
    with pytest.raises(AttributeError):
        fn(c[0], None, *rest[1:], m, n, st)


@pytest.mark.gpu
def test_quantiser_kernel_takes_2_31_elements_and_says_what_it_refuses():
    rows, k = 1 << 18, 8200
    x = torch.randn(1 << 8, k, device="cuda").to(torch.bfloat16).repeat(rows >> 8, 1)
    assert x.numel() >= 1 << 31
    y, s = pertoken_quant_kernel(x, torch.int8)
    want, ws = pertoken_quant(x[:256], quant_dtype=torch.int8)
    for r0 in (0, rows // 2, rows - 256):
        assert torch.equal(y[r0 : r0 + 256], want) and torch.equal(s[r0 : r0 + 256], ws)
    with pytest.raises(_lib.FlyB200Error) as e:
        pertoken_quant_kernel(x.view(-1)[1 : 1 + 64 * k].view(64, k), torch.int8)
    assert e.value.code == _lib.E_BAD_ALIGN
    for bad in (x[:8, :100], x[:8].double(), x[:8].cpu()):
        with pytest.raises(_lib.FlyB200Error):
            pertoken_quant_kernel(bad, torch.int8)
