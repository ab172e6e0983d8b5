"""Decode-batch index tensors expanded on the device.

The reference's model runner builds ``slot_mapping``, ``slot_mapping_shared`` and the
index lists of a decode batch with a Python loop over every cached position of every
hidden-cached request and copies them to the GPU each step
(additional_designs/worker/aptserve_model_runner.py:515-564, 613-648).  Here the host
only ships the two block tables, the sequence lengths and the cache types;
``aps_expand_decode_lists`` (plain lists) or ``aps_expand_decode_metadata`` (tables padded on
the host, from rows of any other kind) writes the eight tensors on the device, bit-identical
to ``metadata.build_decode_metadata``.

``python -m apt_serve_b200.device_metadata`` times both constructions on configuration 2.
"""
from __future__ import annotations

import ctypes
from typing import List, Sequence

import numpy as np
import torch

from . import _native as N
from .metadata import DecodeMetadata, _pad_tables


def expand_decode_metadata(seq_lens: Sequence[int], use_hidden: Sequence[bool],
                           block_tables: Sequence[Sequence[int]],
                           block_tables_4_shared: Sequence[Sequence[int]], block_size: int,
                           device) -> DecodeMetadata:
    """Same arguments and result as ``metadata.build_decode_metadata``, with the tensors
    created on ``device`` by the expansion kernels.  Host work is O(number of blocks):
    reading the two block tables (plain lists natively and unpadded, at one moment).  Nothing waits for the device: one
    copy from pinned memory and one launch (two for padded tables) on the current stream.  The tensors are sections of three
    allocations (what came from the host, the tables, the indices).
    A request with more tokens than its private table has room for, or its shared one if it is hidden-cached, is refused
    (``ValueError``; ``build_decode_metadata`` stops at it with an index error)."""
    dev = torch.device(device)
    b = len(seq_lens)
    read = _read_lists(seq_lens, use_hidden, block_tables, block_tables_4_shared, b, block_size)
    if read is None:
        lens, types, counts = _measure(seq_lens, use_hidden, block_tables, b)
    else:
        lens, counts, (n_own, n_shared, too_long), packed = read
    n_h, n_hid_tok, width, least, most = counts
    if b and least < 1:
        # the kernels count a length below 1 as 1; the host counts must agree with them
        raise ValueError("expand_decode_metadata: every sequence length must be >= 1 "
                         "(it includes the token being decoded)")
    if len(block_tables) != b:
        raise ValueError(f"expand_decode_metadata: {len(block_tables)} block tables for {b} sequences")
    if read is None:
        too_long = _first_too_long(lens, types, block_tables, block_tables_4_shared, block_size)
    if too_long >= 0:
        # its positions would be those of block 0, which is another request's, or not written at all
        raise ValueError(f"expand_decode_metadata: request {too_long} has {lens[too_long]} tokens and no table for all of them "
                         f"(blocks of {block_size})")
    if dev.type == "cuda" and torch.cuda.is_current_stream_capturing():
        # the graph would read the staging buffer again on every replay, long after it has been given back
        raise RuntimeError("expand_decode_metadata: not during stream capture (the tables come from host memory)")
    n_kv = b - n_h
    n_tot = n_hid_tok + n_kv
    lib = N.lib()
    index_sizes = (n_tot, n_hid_tok, n_hid_tok, n_kv, b, n_tot - b, n_h, n_h)   # the eight index tensors
    if read is not None:
        # the lists' entries one behind the other; the GPU pads them into the three tables
        host = torch.empty(len(packed) // 4, dtype=torch.int32, pin_memory=dev.type == "cuda")
        ctypes.memmove(host.data_ptr(), packed, len(packed))
        rows, d_lens, d_type, lists = host.to(dev, non_blocking=True).split((2 * n_kv, b, b, 2 * (b + 1) + n_own + n_shared))
        kv_rows = rows.view(torch.int64)
        starts, own = lists.data_ptr(), lists.data_ptr() + 8 * (b + 1)
        tables = torch.empty(3, b, width, dtype=torch.int32, device=dev)
        priv, ref = tables[0], tables[2]
        parts = torch.empty(sum(index_sizes), dtype=torch.int64, device=dev).split(index_sizes)
        with N.on_device(dev):
            N.check(lib.aps_expand_decode_lists(
                own, starts, own + 4 * n_own, starts + 4 * (b + 1), d_lens.data_ptr(), d_type.data_ptr(), b, width, block_size,
                tables.data_ptr(), *(t.data_ptr() for t in parts), n_tot, n_hid_tok, N.current_stream(dev)))
    else:
        # everything the device gets, in one buffer and one copy: the K/V-cached rows, three tables (private, shared, and
        # the reference's: shared for hidden requests, private otherwise), lengths and types; sections of 128 bytes
        cuts = _cuts((2 * n_kv, b * width, b * width, b * width, b, b), 32)
        host = torch.empty(sum(cuts), dtype=torch.int32, pin_memory=dev.type == "cuda")
        _fill_host(host, cuts, block_tables, block_tables_4_shared, lens, types, width, n_h)
        rows, priv, shared, ref, d_lens, d_type = host.to(dev, non_blocking=True).split(cuts)[::2]
        priv, shared, ref = priv.view(b, width), shared.view(b, width), ref.view(b, width)
        kv_rows = rows.view(torch.int64)
        cuts = _cuts((*index_sizes, (lib.aps_decode_metadata_scratch_bytes(b) + 7) // 8), 16)   # and the kernels' scratch
        parts = torch.empty(sum(cuts), dtype=torch.int64, device=dev).split(cuts)[::2]
        with N.on_device(dev):
            N.check(lib.aps_expand_decode_metadata(
                N.ptr(priv), N.ptr(shared), N.ptr(d_lens), N.ptr(d_type), b, width, block_size,
                *(t.data_ptr() for t in parts[:8]), n_tot, n_hid_tok, None, N.ptr(parts[8]), parts[8].numel() * 8,
                N.current_stream(dev)))
    names = ("slot_mapping", "slot_mapping_shared", "hidden_cache_use_tot", "kv_cache_use_tot",
             "hidden_holder_upd", "hidden_holder_pull", "hidden_cache_store_tot", "hidden_cache_use_input")
    return DecodeMetadata(
        block_tables=ref, seq_lens_tensor=d_lens, seq_lens=lens.tolist(),
        num_hidden_cache_tokens=n_h, num_tot_tokens=n_tot, num_decode_tokens=b,
        max_decode_seq_len=most, private_block_tables=priv,
        cache_type=d_type, kv_request_rows=kv_rows, **dict(zip(names, parts)))


def _read_lists(seq_lens, use_hidden, tables, shared_tables, b, block_size):
    """Lengths and counts as ``_measure`` has them, (the entries of the private and of the shared tables, what
    ``_first_too_long`` says), and the batch as ``aps_read_decode_lists`` lays it out; None unless everything is plain lists that the
    host library reads and shared tables fit the private ones' width."""
    lib = N.host_lib()
    if lib is None or not b:
        return None
    counts = np.empty(8, dtype=np.int64)
    packed = lib.aps_read_decode_lists(seq_lens, use_hidden, tables, shared_tables, b, block_size, counts.ctypes.data)
    if packed is None:
        return None
    n_h, tokens, width, least, most, *entries = counts.tolist()
    return np.frombuffer(packed, np.int32, b, 8 * (b - n_h)), (n_h, tokens, max(1, width), least, most), entries, packed


def _first_too_long(lens, types, tables, shared_tables, block_size):
    """The first request with more tokens than its private table, or its shared one if it is hidden-cached, has room for; -1 if none has."""
    lib, b = N.host_lib(), len(lens)
    if lib is not None:
        r = lib.aps_first_too_long(tables, shared_tables, lens.ctypes.data, types.ctypes.data, b, block_size)
        if r != -2:
            return r
    needed = (-(-lens.astype(np.int64) // block_size)).tolist()
    for r, (n, hidden, own) in enumerate(zip(needed, types.tolist(), tables)):
        if n > len(own) or (hidden and (r >= len(shared_tables) or n > len(shared_tables[r]))):
            return r
    return -1


def _cuts(sizes, pitch):
    """Sizes to split a buffer by: each section and then what pads it to a multiple of ``pitch``."""
    return [n for size in sizes for n in (size, -size % pitch)]


def _measure(seq_lens, use_hidden, tables, b):
    """Lengths and types as int32 arrays, and (hidden-cached requests, their tokens, the widest table or 1, the shortest length,
    the longest): natively for plain lists where the host library has been built (lists that come here are those whose shared
    tables ``_read_lists`` does not take)."""
    lib = N.host_lib()
    if lib is not None and b:
        both = np.empty((2, b), dtype=np.int32)
        counts = np.empty(5, dtype=np.int64)
        at = both.ctypes.data
        if lib.aps_measure_decode_batch(seq_lens, use_hidden, tables, b, at, at + 4 * b, counts.ctypes.data) == 0:
            n_h, tokens, width, least, most = counts.tolist()
            return both[0], both[1], (n_h, tokens, max(1, width), least, most)
    lens = [int(s) for s in seq_lens]
    least, most = min(lens, default=0), max(lens, default=0)
    hid = np.asarray(list(use_hidden), dtype=bool)
    lens = np.asarray(lens, dtype=np.int32)
    width = max(1, max(map(len, tables))) if len(tables) == b else 1
    return lens, hid.astype(np.int32), (int(np.count_nonzero(hid)), int(lens[hid].sum(dtype=np.int64)), width, least, most)


def _fill_host(host, cuts, tables, shared_tables, lens, types, width, n_hidden):
    """The sections of the buffer that goes to the device: natively where the rows are plain, whatever the lengths came as (256 requests
    46 us, otherwise 76)."""
    lib, b = N.host_lib(), len(lens)
    if lib is not None and lib.aps_pack_decode_batch(tables, shared_tables, lens.ctypes.data, types.ctypes.data, b, width,
                                                     n_hidden, host.data_ptr()) == 0:
        return
    rows, priv, shared, ref, h_lens, h_type = (t.numpy() for t in host.split(cuts)[::2])
    pack_tables(tables, shared_tables, types != 0, priv.reshape(b, width), shared.reshape(b, width), ref.reshape(b, width))
    rows.view(np.int64)[:] = np.flatnonzero(types == 0)
    h_lens[:] = lens
    h_type[:] = types


def pack_tables(tables, shared_tables, hid, priv, shared, ref):
    """Pads the tables into three contiguous int32 arrays ``[sequences, width]``: private, shared (zero for K/V-cached requests)
    and the reference's (the one that the request's type selects).  Natively for lists of lists or tuples of plain
    integers where the host library has been built, by numpy otherwise."""
    lib = N.host_lib()
    if lib is None or lib.aps_pack_block_tables(tables, shared_tables, hid.ctypes.data, len(hid), priv.shape[1],
                                                priv.ctypes.data, shared.ctypes.data, ref.ctypes.data) != 0:
        _pack_tables(tables, shared_tables, hid, priv, shared, ref)


def _pack_tables(tables, shared_tables, hid, priv, shared, ref):
    """``aps_pack_block_tables`` for rows of any kind numpy takes."""
    priv[:] = _pad_tables(tables)
    shared[:] = 0
    for r, t in enumerate(shared_tables):
        if hid[r]:
            shared[r, :len(t)] = t
    ref[:] = np.where(hid[:, None], shared, priv)


def _time_both(config: int = 2, repeats: int = 5):
    import time
    from .metadata import BlockPool, blocks_needed, build_decode_metadata
    from .workloads import draw_decode_batch
    lens, hid = draw_decode_batch(config)
    rng = np.random.default_rng(0)
    pool = BlockPool(blocks_needed(lens, hid, 16) + 8, rng)
    tables = [pool.table_for(s, 16, h) for s, h in zip(lens, hid)]
    shared = [pool.shared_table_for(s, 16) if h else [] for s, h in zip(lens, hid)]
    dev = torch.device("cuda")
    for _ in range(2):
        expand_decode_metadata(lens, hid, tables, shared, 16, dev)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(repeats):
        m = expand_decode_metadata(lens, hid, tables, shared, 16, dev)
    torch.cuda.synchronize()
    t_dev = (time.perf_counter() - t0) / repeats
    t0 = time.perf_counter()
    for _ in range(repeats):
        h = build_decode_metadata(lens, hid, tables, shared, 16).to(dev)
    torch.cuda.synchronize()
    t_host = (time.perf_counter() - t0) / repeats
    # the reference's own construction: a Python loop appending two slots per cached position
    t0 = time.perf_counter()
    sm, sms = [], []
    for r, (s, u) in enumerate(zip(lens, hid)):
        if u:
            for j in range(s):
                sms.append(shared[r][j // 16] * 16 + j % 16)
                sm.append(tables[r][j // 16] * 16 + j % 16)
        else:
            sm.append(tables[r][(s - 1) // 16] * 16 + (s - 1) % 16)
    torch.tensor(sm, dtype=torch.long, device=dev); torch.tensor(sms, dtype=torch.long, device=dev)
    torch.cuda.synchronize()
    t_loop = time.perf_counter() - t0
    same = all(torch.equal(getattr(m, f), getattr(h, f)) for f in (
        "slot_mapping", "slot_mapping_shared", "hidden_cache_use_tot", "kv_cache_use_tot",
        "hidden_holder_upd", "hidden_holder_pull", "hidden_cache_store_tot", "hidden_cache_use_input"))
    bytes_dev = sum(v.numel() * v.element_size() for v in (m.private_block_tables, m.block_tables,
                                                           m.seq_lens_tensor, m.cache_type))
    print(f"config {config}: {len(lens)} requests, N_tot={m.num_tot_tokens}; identical={same}; "
          f"device expansion {t_dev * 1e3:.3f} ms per step ({bytes_dev} bytes host->device), "
          f"numpy construction + copy {t_host * 1e3:.3f} ms ({h.tensor_bytes()} bytes), "
          f"per-position Python loop (slot lists only) + copy {t_loop * 1e3:.1f} ms")


if __name__ == "__main__":
    _time_both()
