"""The per-1x32 quantiser kernels against the torch statements on the same GPU tensor: every byte of
codes, scales and (MXFP6) unpacked codes, and the two layout kernels beside them."""

import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200.kernels.gemm import mxfp4_preshuffle as mx4
from flydsl_b200.kernels.gemm import mxfp8_preshuffle as mx8

pytestmark = pytest.mark.gpu
FORMATS = {
    "fp8": (mx8.per_1x32_f8_quant, mx8.per_1x32_f8_quant_torch),
    "fp4": (mx4.per_1x32_f4_quant, mx4.per_1x32_f4_quant_torch),
    "fp6": (mx4.per_1x32_f6_quant, mx4.per_1x32_f6_quant_torch),
}


def edge_rows(k, fmt):
    """Rows that sit on the decisions of the quantisers: scale exponents over the whole fp32 range with
    mantissas around 1.5, code midpoints and their neighbours, zeros of both signs, subnormals, Inf, NaN."""
    g = torch.Generator().manual_seed(3)
    rows = []
    for e in list(range(-149, 128, 3)) + [-127, -126, -125, -100, -99, 126, 127]:
        mant = torch.tensor([1.0, 1.25, 1.4999999, 1.5, 1.5000001, 1.75, 1.9999999])[torch.randint(0, 7, (k // 32, 1), generator=g)]
        top = torch.ldexp(mant.double(), torch.tensor(e)).clamp(max=3.4028234e38)
        if fmt == "fp8":
            steps = torch.randint(-448, 449, (k // 32, 32), generator=g).double() / 448
        else:  # the midpoints between codes are eighths (E2M1) or sixteenths (E2M3) of the scale
            steps = torch.randint(-128, 129, (k // 32, 32), generator=g).double() / 128
        blk = top * steps
        blk[:, 0] = top[:, 0]
        blk[:, 1] = -0.0
        near = blk.float()
        near[:, 2::5] = torch.nextafter(near[:, 2::5], torch.full_like(near[:, 2::5], float("inf")))
        near[:, 3::5] = torch.nextafter(near[:, 3::5], torch.full_like(near[:, 3::5], float("-inf")))
        rows.append(near.reshape(1, k))
    x = torch.cat(rows)
    x[0] = 0.0
    x[1] = -0.0
    x[2, 5] = float("nan")
    x[3, 40] = float("inf")
    x[4, 41] = float("-inf")
    return x


def same(got, want):
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.dtype == b.dtype and a.is_contiguous()
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,k", [(1, 32), (3, 96), (129, 256), (1000, 8192)])
def test_random_rows_bit_identical_to_torch(fmt, dtype, rows, k):
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    x = (torch.randn(rows, k, generator=g, device="cuda") * torch.exp(4 * torch.randn(rows, 1, generator=g, device="cuda"))).to(dtype)
    kernel, statement = FORMATS[fmt]
    same(kernel(x), statement(x))


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_edges_bit_identical_to_torch(fmt, dtype):
    x = edge_rows(256, fmt).to(dtype).cuda()
    kernel, statement = FORMATS[fmt]
    same(kernel(x), statement(x))


@pytest.mark.parametrize("fmt", ["fp8", "fp4"])
def test_leading_dimensions_strides_and_odd_bases(fmt):
    kernel, statement = FORMATS[fmt]
    x = torch.randn(2, 3, 64, device="cuda")
    same(kernel(x), statement(x))
    t = torch.randn(64, 32, device="cuda", dtype=torch.bfloat16).t()  # not contiguous
    same(kernel(t), statement(t))
    odd = torch.randn(64 * 5 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(5, 64)  # base not 16-byte aligned
    same(kernel(odd), statement(odd))


@pytest.mark.parametrize("rows,k", [(1, 128), (31, 256), (129, 384), (1000, 4096)])
@pytest.mark.parametrize("offset", [0, 1])
def test_scale_image_layout(rows, k, offset):
    src = torch.randint(0, 256, (rows * (k // 32) + offset,), dtype=torch.uint8, device="cuda")[offset:].view(rows, k // 32)
    img = mx8.shuffle_scale(src).view(k // 128, -1, 32, 4, 4)  # [k-block][row tile][r % 32][r / 32][j]
    want = torch.zeros(img.shape[1] * 128, k // 32, dtype=torch.uint8, device="cuda")
    want[:rows] = src
    want = want.view(-1, 4, 32, k // 128, 4).permute(3, 0, 2, 1, 4)
    assert torch.equal(img, want)


@pytest.mark.parametrize("rows,k", [(1, 32), (7, 256), (300, 4096)])
def test_fp6_containers(rows, k):
    a = torch.randint(0, 256, (rows, k), dtype=torch.uint8)
    assert torch.equal(mx4.fp6_containers_from_padded(a.cuda()).cpu(), mx4.fp6_containers_from_padded(a))


@pytest.mark.parametrize("src_shift,dst_shift", [(0, 1), (1, 0), (3, 2), (0, 0)])
def test_scale_image_at_any_base(src_shift, dst_shift):
    rows, kb = 200, 16
    src = torch.randint(0, 256, (rows * kb + src_shift,), device="cuda", dtype=torch.uint8)[src_shift:].view(rows, kb)
    n = mx8.scale_image_bytes(rows, kb * 32)
    buf = torch.full((n + dst_shift + 3,), 77, device="cuda", dtype=torch.uint8)
    rc = _lib.load().flyb200_mx_scale_image(buf.data_ptr() + dst_shift, src.data_ptr(), rows, kb * 32, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(buf[dst_shift : dst_shift + n], mx8.shuffle_scale(src.clone()))
    assert torch.all(buf[:dst_shift] == 77) and torch.all(buf[dst_shift + n :] == 77)
