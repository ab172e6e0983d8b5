"""ctypes binding of ``lib/libaptserve_b200.so`` (the C ABI in
``include/aptserve_b200.h``).

There is no fallback: if the library is missing, every operator of this package
raises.  Build it with ``python -m apt_serve_b200.build``.  (The small host library beside it only
packs lists faster than numpy does and may be missing.)
"""
from __future__ import annotations

import ctypes
from ctypes import c_char_p, c_float, c_int, c_int64, c_size_t, c_void_p
import sysconfig
from pathlib import Path

import torch

LIB_PATH = Path(__file__).resolve().parent / "lib" / "libaptserve_b200.so"
# reads Python objects with the layout of the interpreter it was compiled for, whose tag it carries in its name
HOST_LIB_PATH = LIB_PATH.with_name("libaptserve_b200_host" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

APS_OK = 0
APS_ERR_NULL_POINTER = 1
APS_ERR_MISALIGNED = 2
APS_ERR_DTYPE = 3
APS_ERR_SHAPE = 4
APS_ERR_UNSUPPORTED = 5
APS_ERR_WORKSPACE = 6
APS_ERR_CUDA = 7
APS_ERR_DEVICE = 8

DTYPE_ENUM = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}

# name -> (restype, argtypes); kept in step with include/aptserve_b200.h
PROTOTYPES = {
    "aps_last_error": (c_char_p, []),
    "aps_version": (c_char_p, []),
    "aps_reshape_and_cache": (c_int, [c_void_p] * 5 + [c_int64, c_int, c_int, c_int, c_int64,
                                                       c_int64, c_int64, c_int, c_void_p]),
    "aps_hidden_to_cache": (c_int, [c_void_p] * 5 + [c_int64, c_int, c_int64, c_int64, c_int,
                                                     c_void_p]),
    "aps_gather_hidden_rows": (c_int, [c_void_p] * 5 + [c_int64, c_void_p, c_int64, c_int64, c_int] + [c_int64] * 3 + [c_void_p, c_int, c_void_p]),
    "aps_cache_to_hidden": (c_int, [c_void_p] * 4 + [c_int64, c_int, c_int64, c_int64, c_int,
                                                     c_void_p]),
    "aps_mixed_kv_to_cache": (c_int, [c_void_p] * 10 + [c_int64, c_int64, c_int, c_int, c_int,
                                                        c_int64, c_int64, c_int64, c_int64, c_int,
                                                        c_void_p]),
    "aps_prefill_cache_write": (c_int, [c_void_p] * 8 + [c_int64, c_void_p, c_int64] + [c_int] * 4 +
                                [c_int64] * 5 + [c_int, c_void_p]),
    "aps_copy_blocks": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_int64, c_int64, c_void_p]),
    "aps_swap_blocks": (c_int, [c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64,
                                c_int64, c_int, c_void_p, c_void_p]),
    "aps_attention_workspace_bytes": (c_size_t, [c_int] * 5),
    "aps_paged_decode_attention": (c_int, [c_void_p] * 6 + [c_int] * 5 + [c_int64] * 3 +
                                   [c_float, c_void_p, c_size_t, c_int, c_void_p]),
    "aps_paged_decode_attention_static": (c_int, [c_void_p] * 6 + [c_int] * 5 + [c_int64] * 3 +
                                          [c_float, c_int, c_void_p]),
    "aps_hybrid_decode_attention": (c_int, [c_void_p] * 12 + [c_int] * 6 + [c_int64] * 6 +
                                    [c_float, c_void_p, c_size_t, c_int, c_void_p]),
    "aps_kv_reprojection": (c_int, [c_void_p] * 3 + [c_int64] + [c_void_p] * 4 + [c_int] * 3 +
                            [c_int64] * 4 + [c_int, c_void_p, c_void_p]),
    "aps_decode_layer_step": (c_int, [c_void_p] * 15 + [c_int] * 6 + [c_int64] * 9 +
                              [c_float, c_void_p, c_size_t, c_int, c_void_p]),
    "aps_decode_layer_step_workspace_bytes": (c_size_t, [c_int] * 7),
    "aps_plain_decode_step": (c_int, [c_void_p] * 7 + [c_int64] + [c_void_p] * 2 + [c_int] * 5 + [c_int64] * 5 +
                              [c_float, c_void_p, c_size_t, c_int, c_void_p]),
    "aps_prefill_attention": (c_int, [c_void_p] * 5 + [c_int, c_int, c_int64, c_int, c_int] + [c_int64] * 4 +
                              [c_float, c_int, c_void_p]),
    "aps_attention_status": (c_int, [c_void_p, c_void_p, c_void_p]),
    "aps_reprojection_cycles": (c_int, [c_void_p, c_void_p, c_void_p]),
    "aps_cache_ops_status": (c_int, [c_void_p, c_void_p]),
    "aps_selftest_bounded_wait": (c_int, [c_void_p, c_size_t, ctypes.c_longlong, c_void_p] + [c_int] * 5 +
                                  [c_int64, c_int, c_void_p]),
    "aps_selftest_prefill_wait": (c_int, [ctypes.c_longlong, c_void_p]),
    "aps_selftest_tile_pieces": (c_int, [c_int, c_int, c_int, c_void_p]),
    "aps_set_profile_events": (c_int, [c_int, c_void_p, c_void_p]),
    "aps_absorbed_hidden_attention": (c_int, [c_void_p] * 9 + [c_int] * 5 + [c_int64, c_int64, c_int, c_void_p]),
    "aps_tp_unique_id": (c_int, [c_void_p]),
    "aps_tp_init": (c_int, [c_void_p, c_void_p, c_int, c_int]),
    "aps_tp_allreduce": (c_int, [c_void_p, c_void_p, c_int64, c_int, c_void_p]),
    "aps_tp_world_size": (c_int, [c_void_p, c_void_p]),
    "aps_tp_destroy": (c_int, [c_void_p]),
    "aps_decode_metadata_scratch_bytes": (c_size_t, [c_int]),
    "aps_derive_private_tables": (c_int, [c_void_p] * 4 + [c_int64, c_void_p, c_void_p, c_int64, c_void_p, c_int, c_int,
                                          c_int64, c_int, c_void_p]),
    "aps_expand_decode_lists": (c_int, [c_void_p] * 6 + [c_int] * 3 + [c_void_p] * 9 + [c_int64, c_int64, c_void_p]),
    "aps_expand_decode_metadata": (c_int, [c_void_p] * 4 + [c_int] * 3 + [c_void_p] * 8 +
                                   [c_int64, c_int64, c_void_p, c_void_p, c_size_t, c_void_p]),
}

_lib = None


def lib() -> ctypes.CDLL:
    """The loaded library; raises if it has not been built."""
    global _lib
    if _lib is None:
        if not LIB_PATH.exists():
            raise RuntimeError(
                f"{LIB_PATH} is missing: the CUDA extension has not been built "
                "(run `python -m apt_serve_b200.build`). There is no CPU or PyTorch fallback.")
        handle = ctypes.CDLL(str(LIB_PATH))
        for name, (restype, argtypes) in PROTOTYPES.items():
            fn = getattr(handle, name)
            fn.restype = restype
            fn.argtypes = argtypes
        _lib = handle
    return _lib


_host_lib = None


def host_lib():
    """The library that reads Python lists (called with the interpreter lock held), or None where it has not been built."""
    global _host_lib
    if _host_lib is None and HOST_LIB_PATH.exists():
        handle = ctypes.PyDLL(str(HOST_LIB_PATH))
        handle.aps_pack_block_tables.restype = c_int
        handle.aps_pack_block_tables.argtypes = [ctypes.py_object, ctypes.py_object, c_void_p, c_int64, c_int64,
                                                 c_void_p, c_void_p, c_void_p]
        handle.aps_measure_decode_batch.restype = c_int
        handle.aps_measure_decode_batch.argtypes = [ctypes.py_object] * 3 + [c_int64] + [c_void_p] * 3
        handle.aps_pack_decode_batch.restype = c_int
        handle.aps_pack_decode_batch.argtypes = [ctypes.py_object] * 2 + [c_void_p] * 2 + [c_int64] * 3 + [c_void_p]
        handle.aps_first_too_long.restype = c_int64
        handle.aps_first_too_long.argtypes = [ctypes.py_object] * 2 + [c_void_p] * 2 + [c_int64] * 2
        handle.aps_read_decode_lists.restype = ctypes.py_object
        handle.aps_read_decode_lists.argtypes = [ctypes.py_object] * 4 + [c_int64, c_int64, c_void_p]
        _host_lib = handle
    return _host_lib


def check(status: int) -> None:
    """Turn a non-zero ``aps_status`` into the exception the reference would
    raise: ``ValueError`` for unsupported head / block sizes and dtypes
    (aptserve_flash_attn.py:40-41, 278-288), ``RuntimeError`` otherwise
    (``TORCH_CHECK`` in mixed_cache.cu:202)."""
    if status == APS_OK:
        return
    msg = lib().aps_last_error().decode("utf-8", "replace")
    if status in (APS_ERR_UNSUPPORTED, APS_ERR_DTYPE):
        raise ValueError(f"aptserve_b200: {msg} (status {status})")
    raise RuntimeError(f"aptserve_b200: {msg} (status {status})")


def dtype_enum(t: torch.Tensor) -> int:
    try:
        return DTYPE_ENUM[t.dtype]
    except KeyError:
        raise ValueError(f"aptserve_b200: dtype {t.dtype} is not supported") from None


def require_cuda(*tensors: torch.Tensor) -> torch.device:
    dev, index = None, -1
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("aptserve_b200 operators run on CUDA tensors only "
                               "(there is no CPU path)")
        if dev is None:
            dev, index = t.device, t.get_device()
        elif t.get_device() != index:
            raise RuntimeError("aptserve_b200: tensors live on different devices")
    return dev


def ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def only_values(*tensors) -> bool:
    """Whether a call wants nothing of the tensors but their values: no graph for a backward pass, no tangents, trace, batching
    or other transform, no fake tensors or modes that watch the operators.  A native call would leave all of these out in
    silence, the library call is an operator that torch knows."""
    return not (torch.compiler.is_compiling() or torch.jit.is_tracing()
                or any(type(t) is not torch.Tensor and type(t) is not torch.nn.Parameter for t in tensors)
                or (torch.is_grad_enabled() and any(t.requires_grad for t in tensors))
                or torch.autograd.forward_ad._current_level >= 0 or torch._C._functorch.peek_interpreter_stack() is not None
                or torch._C._len_torch_dispatch_stack() > 0)


class _Nothing:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_nothing = _Nothing()


def on_device(device: torch.device):
    """``torch.cuda.device(device)``, which costs a few microseconds a call, only where it is not current already."""
    return _nothing if device.index == torch.cuda.current_device() else torch.cuda.device(device)


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def current_stream(device: torch.device) -> int:
    """The current stream's handle, without building a Stream object around it where torch offers that."""
    if _raw_stream is not None and device.index is not None:
        return _raw_stream(device.index)
    return torch.cuda.current_stream(device).cuda_stream
