"""ctypes binding of libflyb200.so (the C ABI in include/flyb200.h).

There is no fallback: if the library cannot be loaded every operator of this
package raises.
"""

from __future__ import annotations

import contextlib
import ctypes
import importlib.machinery
import importlib.util
import threading
import warnings

import torch

from . import build as _build

OK = 0
E_BAD_ARG, E_BAD_ALIGN, E_CUDA, E_TIMEOUT, E_UNSUPPORTED, E_SMEM_ALIGN, E_WORKSPACE, E_SCRATCH_LIMIT = range(1, 9)

DT_FP8, DT_INT8, DT_FP16, DT_BF16 = range(4)
OUT_BF16, OUT_FP16, OUT_F32 = range(3)
EPI_NONE, EPI_BIAS, EPI_BIAS_RELU, EPI_BIAS_SILU, EPI_BIAS_GELU = range(5)
SRC_ROW_MAJOR, SRC_MFMA_16x16 = range(2)
MOE_QUANT_MAX_K = 16384

IN_DTYPES = {"fp8": DT_FP8, "int8": DT_INT8, "fp16": DT_FP16, "bf16": DT_BF16}
OUT_DTYPES = {"bf16": OUT_BF16, "fp16": OUT_FP16}
EPILOGUES = {
    "none": EPI_NONE,
    "bias": EPI_BIAS,
    "bias_relu": EPI_BIAS_RELU,
    "bias_silu": EPI_BIAS_SILU,
    "bias_gelu": EPI_BIAS_GELU,
}

_vp, _i, _sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t

# name -> (restype, argtypes): one row per declaration in include/flyb200.h
SIGNATURES = {
    "flyb200_gemm_a8w8": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _vp, _sz, _vp]),
    "flyb200_gemm_a8w8_acc": (_i, [_vp, _vp, _vp, _i, _i, _i, _i, _i, _vp, _sz, _vp]),
    "flyb200_gemm_a8w8_static_scratch": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _vp]),
    "flyb200_static_scratch_bytes": (_sz, []),
    "flyb200_gemm_a8w8_scatter": (
        _i,
        [ctypes.POINTER(_vp), _i, _i, ctypes.c_longlong, ctypes.c_longlong, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _vp],
    ),
    "flyb200_pertoken_quant": (_i, [_vp, _vp, _vp, _i, _i, _i, _i, _vp]),
    "flyb200_shuffle_weight": (_i, [_vp, _vp, _i, _i, _i, _i, _vp]),
    "flyb200_unshuffle_weight": (_i, [_vp, _vp, _i, _i, _i, _vp]),
    "flyb200_pair_width": (_i, [_i, _i, _i, _i, _i, _i]),
    "flyb200_describe_call": (_i, [_i, _i, _i, _i, _i, _i, _i, ctypes.POINTER(_i)]),
    "flyb200_describe_plan": (_i, [_i, _i, _i, _i, _i, _i, ctypes.POINTER(_i)]),
    "flyb200_layout_kind": (_i, [_i, _i, _i]),
    "flyb200_workspace_bytes": (_sz, [_i, _i, _i, _i, _i]),
    "flyb200_read_status": (_i, [ctypes.POINTER(_i)]),
    "flyb200_selftest_bounded_wait": (_i, [ctypes.c_uint, _vp]),
    "flyb200_moe_gather_rows": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _vp]),
    "flyb200_moe_quant_sorted": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _vp]),
    "flyb200_moe_gemm": (_i, [_i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp] + [_i] * 12 + [_vp]),
    "flyb200_moe_gemm_shard": (_i, [_i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp] + [_i] * 13 + [_vp]),
    "flyb200_moe_form": (_i, [_i] * 10),
    "flyb200_moe_reduce": (_i, [_vp, _vp, _i, _i, _i, _i, _vp, _vp, _i, _vp]),
    "flyb200_moe_sorting": (_i, [_vp, _vp, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _vp, _vp]),
    "flyb200_moe_sorting_range": (_i, [_vp, _i, _vp, _i, _i, _i, ctypes.c_longlong, _i, _vp, _vp, _vp, _vp, _vp]),
    "flyb200_gemm_mxfp8": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp]),
    "flyb200_gemm_mx_mixed": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp]),
    "flyb200_gemm_mxfp4": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp]),
    "flyb200_mx_quant": (_i, [_vp, _vp, _vp, _vp, ctypes.c_longlong, _i, _i, _vp]),
    "flyb200_mx_fp6_containers": (_i, [_vp, _vp, ctypes.c_longlong, _vp]),
    "flyb200_mx_scale_image": (_i, [_vp, _vp, _i, _i, _vp]),
    "flyb200_mx_scale_image_bytes": (_sz, [_i, _i]),
    "flyb200_strerror": (ctypes.c_char_p, [_i]),
    "flyb200_last_cuda_error": (ctypes.c_char_p, []),
    "flyb200_version": (_i, []),
}

_lock = threading.Lock()
_lib = None
_ops = None
_NO_GUARD = contextlib.nullcontext()


class FlyB200Error(RuntimeError):
    def __init__(self, code: int, what: str):
        self.code = code
        super().__init__(what)


def load() -> ctypes.CDLL:
    """Load (building first if the in-tree library is missing or stale)."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is None:
            path = _build.build_library()
            lib = ctypes.CDLL(path)
            for name, (res, args) in SIGNATURES.items():
                fn = getattr(lib, name)  # AttributeError if the symbol is not exported
                fn.restype = res
                fn.argtypes = args
            _lib = lib
    return _lib


def ops():
    """The CPython extension with the operators' host path (csrc/ops.cpp), loaded (built first if missing
    or stale) on first use.  Its functions return None for arguments that are not of the common form,
    an int for a library error.  Where it can be neither built nor loaded, host_statements.py stands for it:
    the same kernels, with more host time per call."""
    global _ops
    if _ops is not None:
        return _ops
    load()
    with _lock:
        if _ops is None:
            try:
                loader = importlib.machinery.ExtensionFileLoader("flyb200_ops", _build.build_ops())
                mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("flyb200_ops", loader))
                loader.exec_module(mod)
            except (RuntimeError, ImportError, OSError) as e:
                from . import host_statements as mod

                warnings.warn(f"flydsl_b200: no host extension, calls take more host time: {e}", RuntimeWarning, stacklevel=2)
            _ops = mod
    return _ops


def check(code: int, what: str = "libflyb200") -> None:
    if code == OK:
        return
    lib = load()
    msg = lib.flyb200_strerror(code).decode()
    if code == E_CUDA:
        msg += ": " + lib.flyb200_last_cuda_error().decode()
    raise FlyB200Error(code, f"{what}: {msg} (code {code})")


def on_device(device):
    """Context that makes ``device`` current, free of cost where it already is."""
    return _NO_GUARD if torch.cuda.current_device() == device.index else torch.cuda.device(device)


def current_stream(device) -> int:
    """Raw handle of torch's current stream on ``device`` (0 = default)."""
    return torch._C._cuda_getCurrentRawStream(device.index)


PLAN_FIELDS = ("kernel", "bn", "split_k", "kb_per_split", "reduce", "stages", "pdl", "token_blocks", "strips")


def describe_plan(m: int, n: int, k: int, in_dtype: str = "fp8", variant_hint: int = 0, sm_count: int = 148, epilogue: str = "none") -> dict:
    """The kernel variant that the call runs (no GPU needed)."""
    out = (_i * len(PLAN_FIELDS))()
    check(load().flyb200_describe_call(m, n, k, IN_DTYPES[in_dtype], EPILOGUES[epilogue], variant_hint, sm_count, out), "describe_plan")
    return dict(zip(PLAN_FIELDS, list(out)))


def pair_width(m: int, n: int, k: int, in_dtype: str = "fp8", variant_hint: int = 0, sm_count: int = 148, epilogue: str = "none") -> int:
    """Tile width with which the call runs as CTA pairs, 0 where it does not (no GPU needed)."""
    out = (_i * len(PLAN_FIELDS))()
    if load().flyb200_describe_call(m, n, k, IN_DTYPES[in_dtype], EPILOGUES[epilogue], variant_hint, sm_count, out):
        return 0
    return out[1] if out[0] == 3 else 0


def moe_form(stage: int, tokens: int, topk: int, experts: int, model_dim: int, inter_dim: int, tile_m: int, all_experts: int | None = None,
             sm_count: int = 148) -> int:
    """The kernel a mixture-of-experts stage runs on, numbered as in FLYB200_MOE_KERNEL (no GPU needed).  ``experts``: of the call,
    ``all_experts``: of all ranks."""
    blocks = -(-(tokens * topk + experts * tile_m - topk) // tile_m)  # as many as the routing table has room for
    return load().flyb200_moe_form(stage, tokens, topk, experts, all_experts or experts, model_dim, inter_dim, tile_m, blocks, sm_count)


_failure_hooks: list = []


def on_failure_status(fn) -> None:
    """Register a callback run whenever :func:`read_status` finds a failure recorded by a kernel."""
    _failure_hooks.append(fn)


def read_status() -> int:
    """Synchronise the current device and return (and clear) its status word.
    A non-zero status means a kernel gave up on a bounded wait; state that such
    a kernel may have left half-updated (split-K arrival counters) is reset."""
    out = _i(0)
    check(load().flyb200_read_status(ctypes.byref(out)), "read_status")
    if out.value != 0:
        for fn in _failure_hooks:
            fn()
    return out.value
