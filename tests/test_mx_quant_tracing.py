"""The per-1x32 quantisers and the MXFP6 container conversion where torch has to see the operations: fake
tensors, tracing, compilation, subclasses and gradients give what the torch statements give."""

import pytest
import torch
from torch._subclasses import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx

from flydsl_b200.kernels.gemm import mxfp4_preshuffle as mx4
from flydsl_b200.kernels.gemm import mxfp8_preshuffle as mx8

PAIRS = [(mx8.per_1x32_f8_quant, mx8.per_1x32_f8_quant_torch), (mx4.per_1x32_f4_quant, mx4.per_1x32_f4_quant_torch),
         (mx4.per_1x32_f6_quant, mx4.per_1x32_f6_quant_torch)]


def same(a, b):
    return a.shape == b.shape and a.dtype == b.dtype and torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


@pytest.mark.parametrize("quant,ref", PAIRS)
def test_fake_cuda_tensors(quant, ref):
    with FakeTensorMode():
        x = torch.empty(8, 256, device="cuda", dtype=torch.bfloat16)
        got, want = quant(x), ref(x)
    assert [(t.shape, t.dtype, t.device) for t in got] == [(t.shape, t.dtype, t.device) for t in want]


def test_fake_cuda_containers():
    with FakeTensorMode():
        out = mx4.fp6_containers_from_padded(torch.empty(8, 256, device="cuda", dtype=torch.uint8))
    assert out.shape == (8, 256) and out.dtype == torch.uint8


@pytest.mark.gpu
@pytest.mark.parametrize("quant,ref", PAIRS)
def test_traced_and_compiled(quant, ref):
    x, other = torch.randn(2, 16, 256, device="cuda").unbind(0)
    graph = make_fx(quant)(x)
    assert all(same(a, b) for a, b in zip(graph(other), ref(other)))  # the trace holds operations, not x's results
    compiled = torch.compile(quant, backend="eager", fullgraph=True)
    assert all(same(a, b) for a, b in zip(compiled(other), ref(other)))


@pytest.mark.gpu
def test_traced_containers():
    a, b = torch.randint(0, 256, (2, 16, 256), device="cuda", dtype=torch.uint8).unbind(0)
    graph = make_fx(mx4.fp6_containers_from_padded)(a)
    assert torch.equal(graph(b), mx4.fp6_containers_from_padded(b))


@pytest.mark.gpu
def test_codes_carry_the_gradient():
    x = torch.randn(16, 256, device="cuda", requires_grad=True)
    got, want = mx8.per_1x32_f8_quant(x), mx8.per_1x32_f8_quant_torch(x)
    assert [t.requires_grad for t in got] == [t.requires_grad for t in want] == [True, False]
    assert all(same(a.detach(), b.detach()) for a, b in zip(got, want))
    up = torch.randn(16, 256, device="cuda")
    grads = [torch.autograd.grad(q[0].float(), x, up)[0] for q in (got, want)]
    assert torch.equal(*grads) and bool(grads[0].abs().max() > 0)
    with torch.no_grad():
        assert not mx8.per_1x32_f8_quant(x)[0].requires_grad
    import torch.autograd.forward_ad as fw

    with fw.dual_level():
        dual = fw.make_dual(x.detach(), up)
        tangents = [fw.unpack_dual(q(dual)[0].float()).tangent for q in (mx8.per_1x32_f8_quant, mx8.per_1x32_f8_quant_torch)]
        assert same(*tangents)  # bit by bit: tangents past the range of the codes are NaN


class Sub(torch.Tensor):
    pass


@pytest.mark.gpu
@pytest.mark.parametrize("quant,ref", PAIRS)
def test_subclasses_and_lazy_negation(quant, ref):
    x = torch.randn(16, 256, device="cuda")
    got, want = quant(x.as_subclass(Sub)), ref(x.as_subclass(Sub))
    assert [type(t) for t in got] == [type(t) for t in want] and all(same(a, b) for a, b in zip(got, want))
    neg = torch._neg_view(x)
    assert all(same(a, b) for a, b in zip(quant(neg), ref(-x)))
