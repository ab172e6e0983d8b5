"""Drop-in for the reference's ``mixed_cache_ops`` torch extension
(additional_designs/mixed_cache_kernels/mixed_cache.cu:233-237): same three
function names, same positional arguments, in-place on the caller's tensors,
enqueued on the current CUDA stream, returning ``None``.

Unlike the reference launchers (mixed_cache.cu:137,167 use the legacy default
stream) every op here runs on the current torch stream, and bf16 is accepted
next to fp32 / fp16.
"""
from __future__ import annotations

import torch

from . import _native as N


def _idx(t: torch.Tensor, name: str) -> torch.Tensor:
    if t.dtype != torch.int64:
        raise RuntimeError(f"{name} must be an int64 tensor (got {t.dtype})")
    return t if t.is_contiguous() else t.contiguous()


def _rows(t: torch.Tensor, name: str):
    """A 2-D (or [T, H, D]) tensor whose rows are contiguous; returns the row stride."""
    if t.dim() < 2:
        raise RuntimeError(f"{name} must have at least 2 dimensions")
    inner = t[0]
    if t.shape[0] > 0 and not inner.is_contiguous():
        raise RuntimeError(f"{name}: rows must be contiguous")
    return t.stride(0)


def hidden_to_cache(hidden: torch.Tensor, paged_cache: torch.Tensor, slot_mapping: torch.Tensor,
                    src_idx: torch.Tensor, target_slot_idx: torch.Tensor) -> None:
    """``paged_cache`` row ``slot_mapping[target_slot_idx[i]]`` := ``hidden[src_idx[i]]``
    (mixed_cache.cu:119-147).  ``paged_cache`` is the layer's ``[2, NB, BS, H, D]``
    tensor, addressed as flat rows of ``paged_cache.stride(2)`` elements."""
    dev = N.require_cuda(hidden, paged_cache, slot_mapping, src_idx, target_slot_idx)
    if hidden.dtype != paged_cache.dtype:
        raise RuntimeError("hidden_to_cache: hidden and paged_cache dtypes differ")
    n = src_idx.size(0)
    with N.on_device(dev):
        N.check(N.lib().aps_hidden_to_cache(
            N.ptr(hidden), N.ptr(paged_cache), N.ptr(_idx(slot_mapping, "slot_mapping")),
            N.ptr(_idx(src_idx, "src_idx")), N.ptr(_idx(target_slot_idx, "target_slot_idx")),
            n, hidden.size(1), _rows(hidden, "hidden"), paged_cache.stride(2),
            N.dtype_enum(hidden), N.current_stream(dev)))


def cache_to_hidden(hidden: torch.Tensor, paged_cache: torch.Tensor, slot_mapping: torch.Tensor,
                    dst_idx: torch.Tensor) -> None:
    """``hidden[t] := paged_cache`` row ``slot_mapping[t]`` for ``t`` in ``dst_idx``
    (mixed_cache.cu:150-176)."""
    dev = N.require_cuda(hidden, paged_cache, slot_mapping, dst_idx)
    if hidden.dtype != paged_cache.dtype:
        raise RuntimeError("cache_to_hidden: hidden and paged_cache dtypes differ")
    with N.on_device(dev):
        N.check(N.lib().aps_cache_to_hidden(
            N.ptr(hidden), N.ptr(paged_cache), N.ptr(_idx(slot_mapping, "slot_mapping")),
            N.ptr(_idx(dst_idx, "dst_idx")), dst_idx.size(0), hidden.size(1),
            _rows(hidden, "hidden"), paged_cache.stride(2), N.dtype_enum(hidden),
            N.current_stream(dev)))


def gather_hidden_rows(hidden_states: torch.Tensor, paged_cache: torch.Tensor, slot_mapping: torch.Tensor,
                       new_rows: torch.Tensor, cached_rows: torch.Tensor, rows: int) -> torch.Tensor:
    """The decode batch's gathered input (aptserve_opt.py:112-121): ``rows`` zero rows, ``hidden_states`` written at ``new_rows``, then
    ``cache_to_hidden`` at ``cached_rows``.  In one pass where the rows are wide and aligned as a layer's are; the three
    operations one after the other otherwise (other index types, shapes that broadcast, gradients or transforms).  The one
    pass leaves out indices outside the rows, ``attention.raise_on_device_status`` then raises; the indexed write
    stops the process's GPU context at them."""
    if _gathers(hidden_states, paged_cache, slot_mapping, new_rows, cached_rows, rows):
        dev = N.require_cuda(hidden_states, paged_cache, slot_mapping, new_rows, cached_rows)
        out = torch.empty(rows, hidden_states.shape[1], device=dev, dtype=hidden_states.dtype)
        sources = torch.empty(rows, device=dev, dtype=torch.int64)
        with N.on_device(dev):
            status = N.lib().aps_gather_hidden_rows(
                out.data_ptr(), hidden_states.data_ptr(), paged_cache.data_ptr(), slot_mapping.data_ptr(), new_rows.data_ptr(),
                new_rows.shape[0], cached_rows.data_ptr(), cached_rows.shape[0], rows, out.shape[1], out.shape[1],
                hidden_states.stride(0), paged_cache.stride(2), sources.data_ptr(), N.dtype_enum(hidden_states), N.current_stream(dev))
        if status != N.APS_ERR_UNSUPPORTED:
            N.check(status)
            return out
    out = torch.zeros(rows, hidden_states.shape[1], device=hidden_states.device, dtype=hidden_states.dtype)
    out[new_rows] = hidden_states
    cache_to_hidden(out, paged_cache, slot_mapping, cached_rows)
    return out


def _gathers(hidden, cache, slots, new_rows, cached_rows, rows) -> bool:
    """Whether the one pass takes these tensors."""
    return (N.only_values(hidden, cache, slots, new_rows, cached_rows)
            and hidden.dim() == 2 and hidden.stride(1) == 1 and cache.dim() == 5 and hidden.dtype == cache.dtype
            and all(t.dim() == 1 and t.dtype == torch.int64 and t.is_contiguous() and t.device == hidden.device
                    for t in (slots, new_rows, cached_rows))
            and cache.device == hidden.device and hidden.is_cuda
            and new_rows.shape[0] == hidden.shape[0] and hidden.stride(0) >= hidden.shape[1]
            and slots.shape[0] == rows and rows > 0 and hidden.shape[0] > 0 and cached_rows.shape[0] > 0)


def mixed_kv_to_cache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor,
                      v_cache: torch.Tensor, shared_k_cache: torch.Tensor,
                      shared_v_cache: torch.Tensor, slot_mapping: torch.Tensor,
                      slot_mapping_shared: torch.Tensor, kv_cache_use_tot: torch.Tensor,
                      hidden_cache_use_tot: torch.Tensor) -> None:
    """Dual-destination K/V scatter of a hybrid decode batch (mixed_cache.cu:179-230).
    ``key`` / ``value``: ``[N_tot, H, D]``; caches ``[NB, BS, H, D]`` and
    ``[2 NB, BS, H, D]``."""
    dev = N.require_cuda(key, value, k_cache, v_cache, shared_k_cache, shared_v_cache,
                         slot_mapping, slot_mapping_shared, kv_cache_use_tot,
                         hidden_cache_use_tot)
    if k_cache.stride(0) != v_cache.stride(0):  # TORCH_CHECK at mixed_cache.cu:202
        raise RuntimeError("mixed_kv_to_cache: k_cache.stride(0) != v_cache.stride(0)")
    if shared_k_cache.stride(0) != shared_v_cache.stride(0):
        raise RuntimeError("mixed_kv_to_cache: shared cache strides differ")
    with N.on_device(dev):
        N.check(N.lib().aps_mixed_kv_to_cache(
            N.ptr(key), N.ptr(value), N.ptr(k_cache), N.ptr(v_cache), N.ptr(shared_k_cache),
            N.ptr(shared_v_cache), N.ptr(_idx(slot_mapping, "slot_mapping")),
            N.ptr(_idx(slot_mapping_shared, "slot_mapping_shared")),
            N.ptr(_idx(kv_cache_use_tot, "kv_cache_use_tot")),
            N.ptr(_idx(hidden_cache_use_tot, "hidden_cache_use_tot")),
            kv_cache_use_tot.size(0), slot_mapping_shared.size(0), key.size(1), key.size(2),
            k_cache.size(1), _rows(key, "key"), _rows(value, "value"), k_cache.stride(0),
            shared_k_cache.stride(0), N.dtype_enum(key), N.current_stream(dev)))
