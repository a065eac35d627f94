"""The quantiser that writes into sorted order against the quantiser and the gather in turn (bit for bit)."""

import pytest
import torch

from flydsl_b200 import _lib, pertoken_quant
from flydsl_b200.kernels.moe.moe_gemm_2stage import moe_sorting

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qd", [torch.float8_e4m3fn, torch.int8], ids=["fp8", "int8"])
# one to eight warps per row, few and many rows, K no multiple of a warp's vectors
@pytest.mark.parametrize("tokens,topk,experts,block,k", [(1, 2, 8, 16, 768), (33, 4, 16, 64, 1408), (700, 4, 8, 128, 2048), (1300, 2, 4, 32, 144),
                                                         (600, 2, 8, 64, 4096), (300, 2, 4, 16, 16384)])
def test_equals_quantiser_then_gather(qd, tokens, topk, experts, block, k):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(tokens + k)
    x = torch.randn(tokens * topk, k, generator=g, device=dev, dtype=torch.float32) * 3
    x[:: 7, 5] = float("inf")
    x[3 % (tokens * topk)] = 0.0
    x = x.to(torch.bfloat16)
    ids = torch.topk(torch.rand(tokens, experts, generator=g, device=dev), k=topk, dim=1).indices.to(torch.int32)
    ids[0, 0] = -1  # a route that belongs to nobody
    srt, _, e_ids, post = moe_sorting(ids, torch.ones(tokens, topk, device=dev), num_experts=experts, block_size=block)
    # the table is one block longer than what is in use: rows past its end are zero
    rows = e_ids.numel() * block
    srt = torch.cat([srt, srt.new_full((rows,), (topk << 24) | tokens)])[:rows].contiguous()
    st = torch.cuda.current_stream().cuda_stream
    got = torch.full((rows, k), 99, dtype=torch.uint8, device=dev), torch.full((rows,), -1.0, device=dev)
    ref = torch.empty_like(got[0]), torch.empty_like(got[1])
    dt = _lib.DT_INT8 if qd == torch.int8 else _lib.DT_FP8
    lib = _lib.load()
    _lib.check(lib.flyb200_moe_quant_sorted(got[0].data_ptr(), got[1].data_ptr(), x.data_ptr(), srt.data_ptr(), post.data_ptr(), tokens,
                                            topk, k, rows, dt, st))
    y, s = pertoken_quant(x, quant_dtype=qd)
    _lib.check(lib.flyb200_moe_gather_rows(ref[0].data_ptr(), ref[1].data_ptr(), y.data_ptr(), s.data_ptr(), srt.data_ptr(), post.data_ptr(),
                                           tokens, topk, 1, k, rows, st))
    torch.cuda.synchronize()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


def test_refused_arguments():
    lib = _lib.load()
    b = torch.zeros(64, dtype=torch.int32, device="cuda:0").data_ptr()
    ok = (b, b, b, b, b, 1, 1, 128, 0, _lib.DT_FP8, None)
    assert lib.flyb200_moe_quant_sorted(*ok) == 0
    for i, v, code in ((2, None, _lib.E_BAD_ARG), (7, 120, _lib.E_UNSUPPORTED), (7, 32768, _lib.E_UNSUPPORTED), (9, 2, _lib.E_BAD_ARG),
                       (2, b + 4, _lib.E_BAD_ALIGN), (8, -1, _lib.E_BAD_ARG)):
        assert lib.flyb200_moe_quant_sorted(*ok[:i], v, *ok[i + 1 :]) == code
