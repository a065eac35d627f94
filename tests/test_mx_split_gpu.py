"""K split of the block-scaled large-M kernel over a cluster: every factor on ragged row tiles and k-block
counts that the factor does not divide, against the unsplit kernel and the oracle's operands."""

import pytest
import torch

from flydsl_b200 import _lib, shuffle_weight
from flydsl_b200.kernels.gemm.mxfp4_preshuffle import (compile_mxfp4_preshuffle_gemm, per_1x32_f4_quant, per_1x32_f6_quant,
                                                       shuffle_scale_w4, shuffle_weight_w4)
from flydsl_b200.kernels.gemm.mxfp8_preshuffle import compile_mxfp8_preshuffle_gemm, per_1x32_f8_quant, shuffle_scale
from oracle import mx_oracle

pytestmark = pytest.mark.gpu


def product(fmt, x, w, out_dtype):
    """The layer's output (guard rows behind it must stay untouched), the float64 product of the operands as
    the oracle dequantises them, and the sums of the products' magnitudes."""
    m, k = x.shape
    n = w.shape[0]
    c = torch.full((m + 8, n), 7.0, dtype=torch.bfloat16 if out_dtype == "bf16" else torch.float16, device=x.device)
    if fmt == "mxfp8":
        fn = compile_mxfp8_preshuffle_gemm(N=n, K=k, out_dtype=out_dtype)
        a, sa = per_1x32_f8_quant(x)
        b, sb = per_1x32_f8_quant(w)
        w_img, a_img, w_sc = shuffle_weight(b), shuffle_scale(sa), shuffle_scale(sb)
        fa, fw = mx_oracle.dequant(a.cpu(), sa.cpu()), mx_oracle.dequant(b.cpu(), sb.cpu())
    else:
        a_dtype = "fp4" if fmt == "mxfp4" else "fp6"
        fn = compile_mxfp4_preshuffle_gemm(N=n, K=k, out_dtype=out_dtype, a_dtype=a_dtype, b_dtype="fp4")
        a, sa, *raw = per_1x32_f4_quant(x) if fmt == "mxfp4" else per_1x32_f6_quant(x)
        b, sb = per_1x32_f4_quant(w)
        w_img, a_img, w_sc = shuffle_weight_w4(b, for_a_dtype=a_dtype), shuffle_scale_w4(sa), shuffle_scale_w4(sb)
        if fmt == "mxfp4":
            fa = mx_oracle.dequant_fp4(a.cpu(), sa.cpu())
        else:
            fa = mx_oracle.fp6_to_f32(raw[0].cpu()) * mx_oracle.e8m0_to_f32(sa.cpu()).repeat_interleave(32, dim=-1)
        fw = mx_oracle.dequant_fp4(b.cpu(), sb.cpu())
    fn(c.view(-1), a.view(torch.uint8).view(-1), w_img.view(torch.uint8).view(-1), a_img, w_sc, None, m, n, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    assert torch.all(c[m:] == 7.0), "guard rows were written"
    fa, fw = fa.double().to(x.device), fw.double().to(x.device)
    return c[:m].float(), fa @ fw.t(), fa.abs() @ fw.abs().t()


def bound(exact, magnitude, k, out_dtype):
    """Half a unit of the output (8 and 11 significant bits: at most 2^-8 and 2^-11 of the value), and the sum in
    fp32: one addition per 32 products and per part, each off by at most 2^-23 of what has been added so far,
    which the sum of the magnitudes bounds."""
    return 2.0 ** (-8 if out_dtype == "bf16" else -11) * exact.abs() + (k / 32 + 10) * 2.0**-23 * magnitude


@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "mxfp6"])
@pytest.mark.parametrize("m,n,k", [(129, 128, 2304), (300, 256, 4096), (1, 384, 8448), (640, 1024, 14336)])
@pytest.mark.parametrize("out_dtype", ["bf16", "fp16"])
def test_split_equals_unsplit_to_the_last_rounding(monkeypatch, fmt, m, n, k, out_dtype):
    """The parts are fp32 sums of the same products, so the outputs of two splits differ by the rounding of
    the sums (2^-24 of the largest partial sum per addition) and of the output (half a unit)."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    monkeypatch.setenv("FLYB200_MX_SMALL", "0")
    monkeypatch.setenv("FLYB200_MX_SPLIT", "1")
    whole, exact, magnitude = product(fmt, x, w, out_dtype)
    assert bool(((whole - exact).abs() <= bound(exact, magnitude, k, out_dtype)).all())
    unit = 2.0**-8 if out_dtype == "bf16" else 2.0**-11
    # sums of up to k products, each part rounded below k * 2^-24 of the root sum of squares
    slack = k * 2.0**-24 * float(whole.abs().max())
    for split in ("2", "4", "8"):
        monkeypatch.setenv("FLYB200_MX_SPLIT", split)
        got = product(fmt, x, w, out_dtype)[0]
        assert bool(((got - exact).abs() <= bound(exact, magnitude, k, out_dtype)).all())
        assert bool(((got - whole).abs() <= 2 * unit * whole.abs() + slack).all())
        assert torch.equal(got, product(fmt, x, w, out_dtype)[0])  # summed in rank order: repeatable


@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (17, 384, 4096), (128, 1024, 2304)])
def test_mixed_kinds_on_the_small_m_kernel(monkeypatch, m, n, k):
    """MXFP6 x MXFP4 of up to 128 tokens: the small-M kernel (weights on the other operand side) against
    the large-M kernel, apart from the rounding of sums and output, and both against the oracle's operands."""
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    monkeypatch.setenv("FLYB200_MX_SMALL", "0")
    large, exact, magnitude = product("mxfp6", x, w, "fp16")
    monkeypatch.setenv("FLYB200_MX_SMALL", "1")
    small = product("mxfp6", x, w, "fp16")[0]
    for c in (large, small):
        assert bool(((c - exact).abs() <= bound(exact, magnitude, k, "fp16")).all())
    assert bool(((small - large).abs() <= 2.0**-10 * large.abs() + k * 2.0**-24 * float(large.abs().max())).all())


@pytest.mark.parametrize("fmt,k", [("mxfp8", 128), ("mxfp8", 384), ("mxfp8", 512), ("mxfp6", 256), ("mxfp6", 768), ("mxfp4", 256), ("mxfp4", 1024)])
@pytest.mark.parametrize("split", ["2", "4", "8"])
def test_a_forced_split_leaves_no_part_empty(monkeypatch, fmt, k, split):
    """Fewer k-blocks than the forced factor: as many parts as there are k-blocks at most."""
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(150, k, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(256, k, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    monkeypatch.setenv("FLYB200_MX_SPLIT", split)
    c, exact, magnitude = product(fmt, x, w, "fp16")
    assert bool(((c - exact).abs() <= bound(exact, magnitude, k, "fp16")).all())
