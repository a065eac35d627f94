"""The functions of the host extension (csrc/ops.cpp) as Python statements over the C library: taken where the
extension cannot be built or loaded (no C++ compiler, other torch headers), and for arguments that are not
tensors but have a device address.  A function returns what the extension returns: None where the caller's own
statements take the call, an int for a library code."""

from __future__ import annotations

from . import _lib


def eager(x) -> bool:
    return False


def _left_to_the_caller(*args):
    return None


pertoken_quant = mx_quant = mx_scale_image = mx_gemm = moe_sort = moe_layer = _left_to_the_caller


def _ptr(t):
    return None if t is None else t.data_ptr()


def gemm_a8w8(c, a, b, scale_a, scale_b, bias, M, N, K, in_dtype, out_dtype, epilogue, hint, ws, ws_bytes, stream) -> int:
    return _lib.load().flyb200_gemm_a8w8(
        c.data_ptr(), a.data_ptr(), b.data_ptr(), _ptr(scale_a), _ptr(scale_b), _ptr(bias), M, N, K, in_dtype, out_dtype, epilogue, hint,
        ws or None, ws_bytes, stream or None,
    )  # fmt: skip


def moe_stage(out, x, w, scale_x, scale_w, ids, expert_ids, weights, valid, a_sorted, sa_sorted, stage, tokens, topk, gather, k, experts,
              model, inter, tile_m, blocks, in_dtype, out_dtype, doweight, accumulate, stream, all_experts) -> int:
    lib, s = _lib.load(), stream or None
    a, sa, i, v = a_sorted.data_ptr(), sa_sorted.data_ptr(), ids.data_ptr(), valid.data_ptr()
    rc = lib.flyb200_moe_gather_rows(a, sa, x.data_ptr(), scale_x.data_ptr(), i, v, tokens, topk, gather, k, blocks * tile_m, s)
    if rc:
        return rc
    return lib.flyb200_moe_gemm_shard(
        stage, out.data_ptr(), a, w.data_ptr(), sa, scale_w.data_ptr(), i, expert_ids.data_ptr(),
        weights.data_ptr() if weights is not None and weights.numel() else None, v, tokens, topk, experts, all_experts, model, inter, tile_m,
        blocks, in_dtype, out_dtype, int(doweight), int(accumulate), 1, s,
    )  # fmt: skip
