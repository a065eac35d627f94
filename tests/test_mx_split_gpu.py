"""K split of the block-scaled large-M kernel over a cluster: every factor on ragged row tiles and k-block
counts that the factor does not divide, against the unsplit kernel and the CPU oracle."""

import pytest
import torch

from flydsl_b200 import _lib, shuffle_weight
from flydsl_b200.kernels.gemm.mxfp4_preshuffle import (compile_mxfp4_preshuffle_gemm, per_1x32_f4_quant, per_1x32_f6_quant,
                                                       shuffle_scale_w4, shuffle_weight_w4)
from flydsl_b200.kernels.gemm.mxfp8_preshuffle import compile_mxfp8_preshuffle_gemm, per_1x32_f8_quant, shuffle_scale

pytestmark = pytest.mark.gpu


def product(fmt, x, w, out_dtype):
    """The layer's output (guard rows behind it must stay untouched) and the float64 product of the
    dequantised operands."""
    m, k = x.shape
    n = w.shape[0]
    c = torch.full((m + 8, n), 7.0, dtype=torch.bfloat16 if out_dtype == "bf16" else torch.float16, device=x.device)
    if fmt == "mxfp8":
        fn = compile_mxfp8_preshuffle_gemm(N=n, K=k, out_dtype=out_dtype)
        a, sa = per_1x32_f8_quant(x)
        b, sb = per_1x32_f8_quant(w)
        w_img, a_img, w_sc = shuffle_weight(b), shuffle_scale(sa), shuffle_scale(sb)
    else:
        a_dtype = "fp4" if fmt == "mxfp4" else "fp6"
        fn = compile_mxfp4_preshuffle_gemm(N=n, K=k, out_dtype=out_dtype, a_dtype=a_dtype, b_dtype="fp4")
        a, sa = per_1x32_f4_quant(x) if fmt == "mxfp4" else per_1x32_f6_quant(x)[:2]
        b, sb = per_1x32_f4_quant(w)
        w_img, a_img, w_sc = shuffle_weight_w4(b, for_a_dtype=a_dtype), shuffle_scale_w4(sa), shuffle_scale_w4(sb)
    fn(c.view(-1), a.view(torch.uint8).view(-1), w_img.view(torch.uint8).view(-1), a_img, w_sc, None, m, n, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    assert torch.all(c[m:] == 7.0), "guard rows were written"
    return c[:m]


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
    whole = product(fmt, x, w, out_dtype).float()
    unit = 2.0**-8 if out_dtype == "bf16" else 2.0**-11
    # sums of up to k products, each part rounded below k * 2^-24 of the root sum of squares
    slack = k * 2.0**-24 * float(whole.abs().max())
    for split in ("2", "4", "8"):
        monkeypatch.setenv("FLYB200_MX_SPLIT", split)
        got = product(fmt, x, w, out_dtype).float()
        assert bool(((got - whole).abs() <= 2 * unit * whole.abs() + slack).all())
        assert torch.equal(got, product(fmt, x, w, out_dtype).float())  # summed in rank order: repeatable


@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (17, 384, 4096), (128, 1024, 2304)])
def test_mixed_kinds_on_the_small_m_kernel(monkeypatch, m, n, k):
    """MXFP6 x MXFP4 of up to 128 tokens: the small-M kernel (weights on the other operand side) against
    the large-M kernel, apart from the rounding of sums and output."""
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, generator=g, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda", dtype=torch.float32) * 0.05).to(torch.bfloat16)
    monkeypatch.setenv("FLYB200_MX_SMALL", "0")
    large = product("mxfp6", x, w, "fp16").float()
    monkeypatch.setenv("FLYB200_MX_SMALL", "1")
    small = product("mxfp6", x, w, "fp16").float()
    assert bool(((small - large).abs() <= 2.0**-10 * large.abs() + k * 2.0**-24 * float(large.abs().max())).all())
