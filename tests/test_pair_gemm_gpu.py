"""The pair form of the large-M kernel (256 x bn tiles on two CTAs): every tile width, ragged edges, column strips
in the last round, and the rule that takes calls to it."""

import pytest
import torch

from flydsl_b200 import _lib, shuffle_weight
from oracle import a8w8_oracle as oracle
from tests.helpers import as_i8, device_status, gpu_acc

PAIR_FORM = 3 << 8
STRIPS = [  # 74 clusters: 80 tiles of 256 columns leave 6 (four strips each), 104 leave 30 (two)
    (1277, 4080, 256, 8),
    (1024, 6608, 128, 8),
    (1024, 3296, 384, 4),  # 104 tiles of 128 columns, two strips of 64
]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,width", [(m, n, k, w) for m, n, k in ((1, 16, 128), (129, 2064, 1152), (300, 1040, 640)) for w in range(2, 9)] + STRIPS)
def test_every_width_and_strip_bit_exact(m, n, k, width):
    """INT8 accumulators against the oracle: no width divides N, rows end inside either CTA's half."""
    a, b, _, _ = oracle.make_inputs(m, n, k, "int8", seed=width + m, rne_int8=True)
    assert _lib.pair_width(m, n, k, "int8", PAIR_FORM | width) == 32 * width
    acc = gpu_acc(a.cuda(), shuffle_weight(b.cuda()), m, n, k, "int8", variant_hint=PAIR_FORM | width)
    torch.cuda.synchronize()
    assert device_status() == 0
    assert torch.equal(acc.cpu(), oracle.int32_acc(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,width", STRIPS)
def test_last_round_whole_or_in_strips_is_bit_identical(monkeypatch, m, n, k, width):
    a, b, _, _ = oracle.make_inputs(m, n, k, "int8", seed=m, rne_int8=True)
    for tail, strips in (("0", {1}), ("1", {2, 4})):
        monkeypatch.setenv("FLYB200_ROWS_TAIL", tail)
        assert _lib.describe_plan(m, n, k, "int8", PAIR_FORM | width)["strips"] in strips
        acc = gpu_acc(a.cuda(), shuffle_weight(b.cuda()), m, n, k, "int8", variant_hint=PAIR_FORM | width)
        torch.cuda.synchronize()
        assert device_status() == 0
        assert torch.equal(acc.cpu(), oracle.int32_acc(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", ["none", "bias_gelu"])
@pytest.mark.parametrize("in_dtype,out_dtype", [("fp8", "bf16"), ("int8", "fp16"), ("bf16", "bf16"), ("fp16", "fp16")])
@pytest.mark.parametrize("m,n,k,width", [(200, 1040, 1024, 7), (513, 2064, 2048, 0)] + STRIPS[:1])
def test_stored_tiles_equal_those_of_the_one_cta_form(m, n, k, width, in_dtype, out_dtype, epilogue):
    """Same products in the same order, same epilogue: the 128-row form's output, and nothing past the last row."""
    from flydsl_b200 import compile_preshuffle_gemm

    g = torch.Generator().manual_seed(m + width)
    dt = torch.float16 if out_dtype == "fp16" else torch.bfloat16
    if in_dtype in ("fp8", "int8"):
        a, b, sa, sb = oracle.make_inputs(m, n, k, in_dtype, seed=m + width)
    else:
        a, b = (torch.randn(r, k, generator=g).to(dt) for r in (m, n))
        sa = sb = torch.empty(0)
    bias = torch.randn(n, generator=g).to(dt) if epilogue != "none" else torch.empty(0, dtype=dt)
    args = [as_i8(a.cuda()).view(-1), as_i8(shuffle_weight(b.cuda())).view(-1), sa.cuda(), sb.cuda(), bias.cuda(), m, n]
    out = []
    for hint in (2 << 8, PAIR_FORM | width):
        fn = compile_preshuffle_gemm(N=n, K=k, tile_m=128, tile_n=128, tile_k=128, in_dtype=in_dtype, out_dtype=out_dtype,
                                     epilogue=epilogue, variant_hint=hint)
        c = torch.full((m + 260, n), -8192.0, dtype=dt, device="cuda")
        fn(c.view(-1), *args, torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert device_status() == 0
        assert bool((c[m:] == -8192.0).all())
        out.append(c[:m])
    assert torch.equal(out[0], out[1])


def test_which_calls_run_as_pairs():
    """A pure host function: pairs from 129 tokens up where they are estimated to be faster."""
    w = _lib.pair_width
    assert w(4096, 4096, 4096, "fp16") == 256 and w(8192, 28672, 8192) == 256
    assert w(2048, 8192, 8192) == 224 and w(256, 8192, 8192) == 128  # whole rounds; one round of narrow tiles
    assert w(128, 8192, 8192) == 0  # half of the pair would have no rows
    assert w(512, 2048, 8192) == 0 and w(512, 2048, 4096) > 0  # K split in four over a long K stays on the small-M kernel
    assert w(320, 10208, 5120, "bf16") == 0  # 384 padded rows against 512
    assert w(8192, 8192, 1024) == 0 and w(8192, 8192, 2048) > 0  # few k-blocks: the epilogue is longer than the mainloop
    assert w(512, 8192, 2560) == 0  # one round: the set-up weighs more
    # what a caller asks for is not changed, and a request for the form is honoured at its width
    assert w(4096, 8192, 8192, variant_hint=2 << 8) == 0 and w(4096, 8192, 8192, variant_hint=5) == 0
    assert w(64, 256, 128, variant_hint=PAIR_FORM | 3) == 96 and w(64, 256, 128, variant_hint=PAIR_FORM) == 256
    assert w(4096, 8192, 8192, variant_hint=2 << 28) > 0  # (no dependent launch: the kernel is still open)
    assert w(4096, 8192, 8192, sm_count=1) == 0 and w(4096, 8200, 8192) == 0


@pytest.mark.parametrize("m,n,k", [(256, 1024, 8064), (256, 2048, 7936), (130, 1024, 6144), (200, 4096, 8064), (133, 5136, 14336), (256, 4096, 14336)])
def test_narrow_outputs_over_many_k_blocks_keep_the_k_split(m, n, k):
    """Pairs walk all k-blocks on few SMs there; the choice compares times on both sides of 64 k-blocks."""
    assert _lib.pair_width(m, n, k) == 0 and _lib.pair_width(m, n, k + 512) == 0


@pytest.mark.parametrize("m,n", [(130, 1024), (200, 2048), (256, 4096), (129, 16384)])
def test_few_k_blocks_do_not_run_as_pairs(m, n):
    """Eight k-blocks: the 128-row form needs 5.7 us at 200 x 4096, pairs 7.0, the small-M kernel 12.7."""
    assert _lib.pair_width(m, n, 1024) == 0


@pytest.mark.parametrize("m,n,k,width", [(180, 3152, 2048, 64), (184, 6352, 1024, 96), (208, 8240, 1408, 128)])
def test_silu_on_a_partial_last_tile_does_not_run_on_the_128_row_form(m, n, k, width):
    """Its last tile then takes the division's long way: 14.7 instead of 9.1 us on the first size."""
    d = _lib.describe_plan
    assert (d(m, n, k)["kernel"], d(m, n, k)["bn"]) == (2, width)
    assert [d(m, n, k, epilogue=e)["kernel"] for e in ("bias_relu", "bias_gelu", "bias_silu")] == [2, 2, 3]
    whole = n // width * width
    assert d(m, whole, k, epilogue="bias_silu")["kernel"] == 2
