"""The large-M kernel's epilogue: every activation on tile edges, with channel scales and bias that do
not start on 16 bytes, and the reciprocal it uses instead of a division."""

import numpy as np
import pytest
import torch

from flydsl_b200 import compile_preshuffle_gemm, shuffle_weight
from oracle import a8w8_oracle as oracle
from tests.test_gemm_parity_gpu import ATOL, ROWS, RTOL, TALL, run_gemm_generic


def test_one_newton_step_gives_the_ieee_reciprocal():
    """r + r (1 - x r) from any estimate within one unit in the last place, on every float of [1, 2)
    (powers of two scale exactly): the IEEE reciprocal but for at most 32 of the 2^23, which are one unit
    off, an error of 0.5 + 2^-20 units (Markstein's exceptions).  float64 holds the residual exactly."""
    x = (np.arange(1 << 23, dtype=np.uint32) + np.uint32(0x3F800000)).view(np.float32)
    exact = (np.float32(1) / x).astype(np.float32)
    for step in (-1, 0, 1):
        r = (exact.view(np.int32) + step).view(np.float32)
        e = (1.0 - x.astype(np.float64) * r).astype(np.float32)
        off = (r + r.astype(np.float64) * e).astype(np.float32).view(np.int32) - exact.view(np.int32)
        assert np.abs(off).max() <= 1 and np.count_nonzero(off) <= 32


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", ["none", "bias", "bias_relu", "bias_silu", "bias_gelu"])
@pytest.mark.parametrize("in_dtype,out_dtype,offset,hint", [("fp8", "bf16", 0, ROWS | 8), ("int8", "fp16", 1, ROWS | 7), ("int8", "bf16", 2, TALL | 5),
                                                            ("bf16", "fp16", 3, ROWS | 3), ("fp16", "bf16", 4, 0)])
def test_epilogue_on_tile_edges(epilogue, in_dtype, out_dtype, offset, hint):
    """Scales and bias as views `offset` elements into a buffer; N ends inside a tile, M inside a row block.
    Large negative and positive biases reach both ends of the exponentials."""
    dev = torch.device("cuda:0")
    m, n, k = 301, 1040, 512
    g = torch.Generator().manual_seed(offset)
    odt = torch.float16 if out_dtype == "fp16" else torch.bfloat16
    bias = torch.randn(n, generator=g) * 3
    bias[::7] = -95.0
    bias[1::7] = 60.0
    bias = bias.to(odt)
    if in_dtype in ("bf16", "fp16"):
        dt = torch.bfloat16 if in_dtype == "bf16" else torch.float16
        a, b = torch.randn(m, k, generator=g).to(dt), (torch.randn(n, k, generator=g) * 0.05).to(dt)
        sa = sb = sb_dev = None
    else:
        a, b, sa, sb = oracle.make_inputs(m, n, k, in_dtype, seed=offset)
        sb_buf = torch.empty(n + 8, dtype=torch.float32, device=dev)
        sb_dev = sb_buf[offset : offset + n]
        sb_dev.copy_(sb.view(-1))
    bias_buf = torch.empty(n + 8, dtype=odt, device=dev)
    bias_dev = bias_buf[offset : offset + n]
    bias_dev.copy_(bias)
    got = run_gemm_generic(dev, a, b, sa, sb_dev, bias_dev if epilogue != "none" else None, m, n, k, in_dtype, out_dtype=out_dtype,
                           epilogue=epilogue, hint=hint)
    acc = a.float() @ b.float().T
    ref = oracle.epilogue(acc, sa, sb, bias, epilogue, out_dtype=torch.float32)
    assert not torch.isnan(got).any() and oracle.strict_mismatches(got, ref, RTOL, ATOL) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,width", [(300, 12816, 8), (300, 12704, 8), (300, 14464, 8), (300, 6448, 4), (100, 19104, 4), (520, 7584, 8)])
@pytest.mark.parametrize("in_dtype", ["int8", "bf16"])
def test_last_round_in_strips_is_bit_identical(monkeypatch, m, n, width, in_dtype):
    """Tiles of 32 * width columns of which a few are left for the last round (2 and 4 strips; a last tile of
    16 columns whose other strips are empty; a strip that N ends in): every output is the same sum."""
    dev = torch.device("cuda:0")
    k = 256
    g = torch.Generator().manual_seed(n)
    bias = torch.randn(n, generator=g).to(torch.bfloat16)
    if in_dtype == "bf16":
        a, b, sa, sb = torch.randn(m, k, generator=g).bfloat16(), torch.randn(n, k, generator=g).bfloat16(), None, None
    else:
        a, b, sa, sb = oracle.make_inputs(m, n, k, in_dtype, seed=n)
    outs = []
    for tail in ("0", "1"):
        monkeypatch.setenv("FLYB200_ROWS_TAIL", tail)
        outs.append(run_gemm_generic(dev, a, b, sa, sb, bias, m, n, k, in_dtype, epilogue="bias_gelu", hint=ROWS | width))
    assert torch.equal(outs[0], outs[1])
    ref = oracle.epilogue(a.float() @ b.float().T, sa, sb, bias, "bias_gelu", out_dtype=torch.float32)
    assert oracle.strict_mismatches(outs[1], ref, RTOL, ATOL) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", ["none", "bias", "bias_relu", "bias_silu", "bias_gelu"])
@pytest.mark.parametrize("m", [1, 16, 40])
def test_direct_and_reduced_stores_of_the_small_m_kernel_agree(m, epilogue):
    """The same integer accumulators through the unsplit kernel (stored from the accumulator layout) and through
    K splits (summed exactly, stored after the reduction, four values at a time): the same bits."""
    n, k = 512, 4096
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int8)
    b = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    sa, sb = (torch.rand(r, generator=g, device="cuda") * 2e-3 + 1e-4 for r in (m, n))
    bias = torch.randn(n, generator=g, device="cuda").to(torch.float16)
    outs = []
    for hint in (1 << 8 | 1, 1 << 8 | 1 << 12 | 4, 1 << 8 | 2 << 12 | 4):  # unsplit, through a workspace, inside a cluster
        fn = compile_preshuffle_gemm(N=n, K=k, tile_m=64, tile_n=128, tile_k=128, in_dtype="int8", out_dtype="fp16", epilogue=epilogue,
                                     variant_hint=hint)
        c = torch.empty(m, n, device="cuda", dtype=torch.float16)
        fn(c.view(-1), a.view(-1), shuffle_weight(b).view(-1), sa, sb, bias, m, n, torch.cuda.current_stream())
        outs.append(c)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", ["none", "bias_silu"])
@pytest.mark.parametrize("in_dtype,out_dtype,hint", [("fp8", "bf16", ROWS | 8), ("int8", "fp16", ROWS | 7), ("fp16", "fp16", ROWS | 3), ("bf16", "bf16", ROWS | 1)])
def test_four_and_eight_epilogue_warps_store_the_same_bits(monkeypatch, in_dtype, out_dtype, epilogue, hint):
    """Tiles of 256, 224 (a 32-column tail), 96 and 32 columns, several rounds, ragged M and N."""
    dev = torch.device("cuda:0")
    m, n, k = 2300, 2064, 512
    g = torch.Generator().manual_seed(hint)
    bias = torch.randn(n, generator=g).to(torch.float16 if out_dtype == "fp16" else torch.bfloat16)
    if in_dtype in ("bf16", "fp16"):
        dt = torch.bfloat16 if in_dtype == "bf16" else torch.float16
        a, b, sa, sb = torch.randn(m, k, generator=g).to(dt), (torch.randn(n, k, generator=g) * 0.05).to(dt), None, None
    else:
        a, b, sa, sb = oracle.make_inputs(m, n, k, in_dtype, seed=hint)
    outs = []
    for warps in ("4", "8"):
        monkeypatch.setenv("FLYB200_ROWS_EPI", warps)
        outs.append(run_gemm_generic(dev, a, b, sa, sb, bias if epilogue != "none" else None, m, n, k, in_dtype, out_dtype=out_dtype,
                                     epilogue=epilogue, hint=hint))
    assert torch.equal(outs[0], outs[1])
    ref = oracle.epilogue(a.float() @ b.float().T, sa, sb, bias, epilogue, out_dtype=torch.float32)
    assert oracle.strict_mismatches(outs[0], ref, RTOL, ATOL) == 0
