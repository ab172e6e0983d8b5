"""Device-side expansion of the decode index tensors: bit-identical to the host
construction (which restates the reference's model runner)."""
import numpy as np
import pytest
import torch

from apt_serve_b200.device_metadata import expand_decode_metadata
from apt_serve_b200.metadata import BlockPool, blocks_needed, build_decode_metadata
from apt_serve_b200.workloads import draw_decode_batch

pytestmark = pytest.mark.gpu

FIELDS = ("slot_mapping", "slot_mapping_shared", "hidden_cache_use_tot", "kv_cache_use_tot",
          "hidden_holder_upd", "hidden_holder_pull", "hidden_cache_store_tot",
          "hidden_cache_use_input", "block_tables", "seq_lens_tensor", "private_block_tables",
          "cache_type", "kv_request_rows")


def batch(lens, hid, seed=0, bs=16):
    rng = np.random.default_rng(seed)
    pool = BlockPool(blocks_needed(lens, hid, bs) + 5, rng)
    tables = [pool.table_for(s, bs, h) for s, h in zip(lens, hid)]
    shared = [pool.shared_table_for(s, bs) if h else [] for s, h in zip(lens, hid)]
    return tables, shared


def check(lens, hid, bs=16, seed=0):
    tables, shared = batch(lens, hid, seed, bs)
    host = build_decode_metadata(lens, hid, tables, shared, bs)
    dev = expand_decode_metadata(lens, hid, tables, shared, bs, "cuda")
    torch.cuda.synchronize()
    for f in FIELDS:
        a, b = getattr(dev, f).cpu(), getattr(host, f)
        assert a.dtype == b.dtype and torch.equal(a, b), f
    assert dev.num_tot_tokens == host.num_tot_tokens
    assert dev.num_hidden_cache_tokens == host.num_hidden_cache_tokens


def test_worked_example():
    check([3, 5], [True, False])


@pytest.mark.parametrize("lens,hid", [
    ([1, 1, 1], [True, False, True]),
    ([16, 17, 2048, 5], [True, True, True, True]),      # no K/V request
    ([40, 700, 33], [False, False, False]),             # no hidden request
    ([129, 1, 64, 300, 16, 15], [False, True, False, True, True, False]),
])
def test_edge_batches(lens, hid):
    check(lens, hid)


def test_block_size_32_and_many_requests():
    rng = np.random.default_rng(5)
    lens = rng.integers(1, 400, size=1500).tolist()    # more requests than scan threads
    hid = (rng.random(1500) < 0.4).tolist()
    check(lens, hid, bs=32, seed=5)


def test_config2_and_config4_batches():
    for cfg in (2, 4):
        lens, hid = draw_decode_batch(cfg)
        check(lens, hid, seed=cfg)


def test_counts_that_disagree_with_the_device_side_batch_write_nothing():
    """The caller sizes (and may NULL) the outputs from its own counts.  When the device-side
    cache types / lengths disagree with them the kernels must not store anything: every
    output keeps its sentinel, and the counts word shows what the device saw.  Two cases:
    all-hidden counts with a K/V row on the device (kv_cache_use_tot is NULL), and a
    sequence length of 0, which the device counts as 1."""
    from apt_serve_b200 import _native as N
    dev = torch.device("cuda")
    bs, width = 16, 4
    cases = [
        # (device-side lens, device-side cache types, claimed N_tot, claimed N_h)
        ([20, 7, 33], [1, 0, 1], 60, 60),     # claim: all three hidden
        ([20, 0, 33], [1, 1, 1], 53, 53),     # claim: host counted the empty request as 0 tokens
    ]
    for lens, ctype, n_tot, n_hid in cases:
        b = len(lens)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
        tables = torch.arange(b * width, dtype=torch.int32, device=dev).view(b, width)
        sent = -7
        full = lambda n: torch.full((max(n, 1),), sent, dtype=torch.int64, device=dev)
        out = {"slot_mapping": full(n_tot), "slot_mapping_shared": full(n_hid), "use_tot": full(n_hid),
               "upd": full(b), "pull": full(n_tot - b), "store": full(b), "use_input": full(b)}
        counts = torch.zeros(4, dtype=torch.int64, device=dev)
        scratch = torch.empty(N.lib().aps_decode_metadata_scratch_bytes(b) // 4, dtype=torch.int32, device=dev)
        st = N.lib().aps_expand_decode_metadata(
            N.ptr(tables), N.ptr(tables), N.ptr(i32(lens)), N.ptr(i32(ctype)), b, width, bs,
            N.ptr(out["slot_mapping"]), N.ptr(out["slot_mapping_shared"]), N.ptr(out["use_tot"]),
            None,                                   # kv_cache_use_tot: empty for an all-hidden claim
            N.ptr(out["upd"]), N.ptr(out["pull"]), N.ptr(out["store"]), N.ptr(out["use_input"]),
            n_tot, n_hid, N.ptr(counts), N.ptr(scratch), scratch.numel() * 4, N.current_stream(dev))
        assert st == N.APS_OK
        torch.cuda.synchronize()
        for name, t in out.items():
            assert bool((t == sent).all()), f"{name} was written despite the mismatch"
        seen = counts.tolist()
        assert seen[0] != n_tot or seen[1] != n_hid


@pytest.mark.parametrize("lens,ctype,n_tot,n_hid", [([20, 7, 33], [1, 0, 1], 60, 60), ([20, 0, 33], [1, 1, 1], 53, 53), ([20, 7, 33], [1, 0, 1], 54, 53)])
def test_lists_whose_counts_disagree_leave_the_indices_alone(lens, ctype, n_tot, n_hid):
    """The same for the lists that the GPU pads: the index tensors keep their sentinel (unless the counts agree, the last case), the
    tables are written."""
    from apt_serve_b200 import _native as N
    b, bs, width, sent = 3, 16, 4, -7
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    own, shared = [[1, 2], [3], [4, 5, 6]], [[7, 8], [], [9, 10, 11]]
    starts = lambda rows: i32([0, *np.cumsum([len(t) for t in rows]).tolist()])
    given = i32(sum(own, [])), starts(own), i32(sum(shared, [])), starts(shared), i32(lens), i32(ctype)
    tables = torch.full((3, b, width), sent, dtype=torch.int32, device="cuda")
    n_kv = n_tot - n_hid
    out = [torch.full((max(n, 1),), sent, dtype=torch.int64, device="cuda") for n in (n_tot, n_hid, n_hid, n_kv, b, n_tot - b, b, b)]
    N.check(N.lib().aps_expand_decode_lists(*(t.data_ptr() for t in given), b, width, bs, tables.data_ptr(),
                                            *(None if i == 3 and n_kv == 0 else t.data_ptr() for i, t in enumerate(out)), n_tot, n_hid,
                                            N.current_stream(tables.device)))
    agree = n_kv == 1
    assert all(bool((t == sent).all()) != agree for t in out)
    pad = lambda t: t + [0] * (width - len(t))
    used = [s if h else [] for s, h in zip(shared, ctype)]
    assert tables.tolist() == [[pad(t) for t in own], [pad(t) for t in used], [pad(s if h else t) for t, s, h in zip(own, used, ctype)]]


def test_zero_length_is_refused_on_the_host():
    with pytest.raises(ValueError, match=">= 1"):
        expand_decode_metadata([5, 0], [True, False], [[0], [1]], [[2], []], 16, "cuda")


def test_expansion_during_capture_is_refused():
    """A replay would copy from a staging buffer that is no longer this call's."""
    tables, shared = batch([40, 7], [True, False])
    expand_decode_metadata([40, 7], [True, False], tables, shared, 16, "cuda")
    x, g = torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        with pytest.raises(RuntimeError, match="capture"):
            expand_decode_metadata([40, 7], [True, False], tables, shared, 16, "cuda")
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    check([40, 7], [True, False])


@pytest.mark.parametrize("bs", [16, 32])
@pytest.mark.parametrize("lens,hid", [
    ([1], [True]),
    ([16, 17, 2048, 5], [True, True, True, True]),
    ([129, 1, 64, 300, 16, 15], [False, True, False, True, True, False]),
    ([int(x) for x in np.random.default_rng(3).integers(1, 2100, size=300)], [i % 3 == 0 for i in range(300)]),
])
def test_derived_tables_equal_the_tensor_form(lens, hid, bs):
    """The one-launch derivation against the same thing as tensor operations, in every form it accepts."""
    from dataclasses import replace
    from apt_serve_b200.metadata import _derive_with_tensor_ops, derive_private_block_tables
    tables, shared = batch(lens, hid, 1, bs)
    m = build_decode_metadata(lens, hid, tables, shared, bs).to("cuda")
    wide = torch.full((len(lens), m.block_tables.shape[1] + 3), 7, dtype=torch.int32, device="cuda")
    wide[:, :-3] = m.block_tables
    forms = [m,
             replace(m, block_tables=wide[:, :-3]),                                   # rows with a stride of their own
             replace(m, hidden_cache_use_input=m.hidden_cache_use_input.flip(0) - len(lens)),   # any order, from the end
             replace(m, seq_lens_tensor=m.seq_lens_tensor.long())]                    # a type the kernel does not take
    for f in forms:
        got, want = derive_private_block_tables(f, bs), _derive_with_tensor_ops(f, bs)
        for a, b in zip(got, want):
            assert a.dtype == b.dtype and torch.equal(a, b)


def test_derived_tables_bound_their_indices():
    """A claim that points outside slot_mapping: nothing is read there, the request is taken out of the step, the status
    says so once."""
    import ctypes
    from apt_serve_b200 import _native as N
    lib, host = N.lib(), ctypes.c_int(0)
    i32 = dict(dtype=torch.int32, device="cuda")
    i64 = dict(dtype=torch.int64, device="cuda")
    none = -2 ** 31
    for upd, rows, want, types in [([39, 40], [0], [[-1] * 4, [4, 5, 6, 7]], [none, 0]),
                                   ([31, 40], [0, 2], [[-1] * 4] * 2, [none] * 2),
                                   ([31, 40], [-3], [[-1] * 4] * 2, [none] * 2)]:
        tables, ctype = torch.full((2, 4), -5, **i32), torch.full((2,), -5, **i32)
        bt, lens = torch.arange(8, **i32).view(2, 4), torch.tensor([40, 7], **i32)
        slots, upd, rows = torch.arange(32, 64, **i64), torch.tensor(upd, **i64), torch.tensor(rows, **i64)
        stream = N.current_stream(tables.device)
        N.check(lib.aps_derive_private_tables(N.ptr(tables), N.ptr(ctype), N.ptr(bt), N.ptr(slots), 32, N.ptr(upd),
                                              N.ptr(rows), rows.numel(), N.ptr(lens), 2, 4, 4, 16, stream))
        for status in (2, 0):
            N.check(lib.aps_cache_ops_status(ctypes.addressof(host), stream))
            assert host.value == status
        assert tables.tolist() == want and ctype.tolist() == types


# direct path (fp16, fp32), re-projection on the tensor cores (few requests) and on the CUDA cores (three heads)
@pytest.mark.parametrize("heads,d,e,dtype", [(8, 128, 1024, torch.float16), (12, 64, 768, torch.float32),
                                             (2, 128, 256, torch.float16), (3, 64, 192, torch.float16)])
@pytest.mark.parametrize("fault", ["run", "slot", "list"])
def test_a_step_on_bad_metadata_touches_no_other_request(heads, d, e, dtype, fault):
    from apt_serve_b200 import attention as A
    from apt_serve_b200.metadata import derive_private_block_tables
    from apt_serve_b200.workloads import LayerShape, make_decode_workload
    from dataclasses import replace
    w = make_decode_workload(LayerShape("t", heads, d, e, dtype), [300, 40, 129, 33, 260], [True, False, True, True, False],
                             seed=5, device="cuda")
    two_caches = w.hidden_cache.data_ptr() != w.kv_cache.data_ptr()

    def step(meta):
        tables, types = derive_private_block_tables(meta, 16)
        return A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache,
                                   *w.kv_weights(), tables, meta.seq_lens_tensor, types, w.scale)

    before = w.kv_cache.clone(), w.hidden_cache.clone()
    want = step(w.meta)
    A.raise_on_device_status()
    rows = w.hidden_cache.reshape(-1, e)
    bad = 2
    at = w.block_tables[bad][-1] * 16 + (w.seq_lens[bad] - 1) % 16   # its new row
    rows[at] = before[1].reshape(-1, e)[at]
    after = w.kv_cache.clone(), w.hidden_cache.clone()
    w.kv_cache.copy_(before[0])
    if two_caches:
        w.hidden_cache.copy_(before[1])
    m = w.meta
    if fault == "run":
        m = replace(m, hidden_holder_upd=m.hidden_holder_upd + torch.tensor([0, 0, 5000, 0, 0], device="cuda"))
    elif fault == "slot":
        slots = m.slot_mapping.clone()
        slots[m.hidden_holder_upd[bad] - 128] = -1
        m = replace(m, slot_mapping=slots)
    else:
        m = replace(m, hidden_cache_use_input=torch.tensor([0, 3, 17], device="cuda"))
        after = before
    out = step(m)
    with pytest.raises(RuntimeError, match="outside its tensors"):
        A.raise_on_device_status()
    A.raise_on_device_status()   # said once
    assert torch.equal(w.kv_cache, after[0]) and torch.equal(w.hidden_cache, after[1])
    good = [] if fault == "list" else [0, 1, 3, 4]
    assert not out[[r for r in range(5) if r not in good]].any()
    if good:
        tol = 1e-4 if dtype == torch.float32 else 4e-3
        assert torch.allclose(out[good].float(), want[good].float(), rtol=tol, atol=tol)


# tables as lists that the GPU pads and tables padded on the host; rows with spare blocks, tuples, a wide table of a K/V-cached
# request, more requests than there are CTAs (two, then four for each)
@pytest.mark.parametrize("kind", ["plain", "spare blocks", "tuples", "one wide", "many", "very many"])
def test_lists_and_padded_tables_agree(kind, monkeypatch):
    from apt_serve_b200 import device_metadata as DM
    rng = np.random.default_rng(5)
    lens = [int(x) for x in rng.integers(1, 40 if "many" in kind else 600, size={"many": 1400, "very many": 4001}.get(kind, 23))]
    hid = [bool(i % 3) for i in range(len(lens))]
    make = lambda s: [int(x) for x in rng.integers(0, 2 ** 20, size=-(-s // 16))]
    tables, shared = [make(s) for s in lens], [make(s) if h else [] for s, h in zip(lens, hid)]
    if kind == "spare blocks":
        tables = [t + make(16 * (r % 4)) for r, t in enumerate(tables)]
        shared = [t + make(16 * (r % 3)) if t else t for r, t in enumerate(shared)]
        tables[4] = tables[4] + make(900)
    elif kind == "tuples":
        tables, shared = [tuple(t) for t in tables], [tuple(t) for t in shared]
    elif kind == "one wide":
        tables[3] = make(5000)
    with monkeypatch.context() as m:
        m.setattr(DM, "_fill_host", None)   # not by padded tables
        got = expand_decode_metadata(lens, hid, tables, shared, 16, "cuda")
    monkeypatch.setattr(DM, "_read_lists", lambda *a: None)
    want = expand_decode_metadata(lens, hid, tables, shared, 16, "cuda")
    for name, value in vars(want).items():
        other = getattr(got, name)
        assert torch.equal(value, other) if isinstance(value, torch.Tensor) else value == other, name


def test_lists_that_are_not_plain_take_the_general_path():
    lens, hid = [20, 40, 7], [True, False, True]
    tables, shared = [[1, 2], [3, 4, 5], [6]], [[7, 8], [], [9]]
    want = expand_decode_metadata(lens, hid, tables, shared, 16, "cuda")
    for other in ([np.int64(1), 2], np.array([1, 2], dtype=np.int32)):
        got = expand_decode_metadata(lens, hid, [other] + tables[1:], shared, 16, "cuda")
        for name, value in vars(want).items():
            assert torch.equal(value, getattr(got, name)) if isinstance(value, torch.Tensor) else value == getattr(got, name), name
    with pytest.raises(ValueError):   # a shared table wider than the widest private one
        expand_decode_metadata(lens, hid, tables, [[7, 8, 9, 10], [], [9]], 16, "cuda")
    with pytest.raises((ValueError, OverflowError)):
        expand_decode_metadata(lens, hid, tables, [[7, 2 ** 31], [], [9]], 16, "cuda")
