"""What the host side of a K/V-only decode step hands to the native calls, recorded in place of the library (no GPU)."""
import pytest
import torch

from apt_serve_b200 import _native as N
from apt_serve_b200 import attention as A
from apt_serve_b200 import ops

HEADS, D, BLOCK = 4, 64, 16
WIDTH = HEADS * D


class Recorder:
    """Stands in for the library: records the calls, answers APS_OK."""

    def __init__(self):
        self.calls = []

    def aps_attention_workspace_bytes(self, *a):
        return 1 << 20

    def __getattr__(self, name):
        return lambda *a: self.calls.append((name, a)) or 0


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(N, "lib", lambda: rec)
    monkeypatch.setattr(N, "require_cuda", lambda *t: torch.device("cpu"))
    monkeypatch.setattr(N, "on_device", lambda dev: N._nothing)
    monkeypatch.setattr(N, "current_stream", lambda dev: 0)
    return rec


def batch(n, slots=None, table_rows=None, lens=None):
    """Metadata of a decode batch, and its query, key and value rows."""
    none = torch.zeros(0, dtype=torch.int64)
    meta = A.FlashAttentionMetadata(
        num_prefills=0, num_prefill_tokens=0, num_decode_tokens=n, num_hidden_cache_tokens=0, num_tot_tokens=n,
        slot_mapping=torch.arange(n if slots is None else slots), slot_mapping_shared=none, hidden_cache_use_tot=none,
        kv_cache_use_tot=torch.arange(n), hidden_cache_use_input=none, hidden_cache_store_tot=none, hidden_holder_upd=torch.arange(n),
        hidden_holder_pull=none, seq_lens=[5] * n, seq_lens_tensor=torch.full((n if lens is None else lens,), 5, dtype=torch.int32),
        max_query_len=1, max_prefill_seq_len=0, max_decode_seq_len=5, query_start_loc=None, seq_start_loc=None,
        context_lens_tensor=None, block_tables=torch.zeros(n if table_rows is None else table_rows, 2, dtype=torch.int32),
        use_cuda_graph=False)
    return meta, [torch.randn(n, WIDTH).half() for _ in range(3)]


def impl_and_cache():
    return A.FlashAttentionImpl(HEADS, D, D ** -0.5, HEADS, None, None, "auto"), torch.zeros(2, 8, BLOCK, HEADS, D, dtype=torch.half)


def one_row(kind):
    """A row of WIDTH elements whose first stride is not WIDTH."""
    if kind == "of a buffer with an odd pitch":
        return torch.randn(3, WIDTH + 1).half()[:1, :WIDTH]
    if kind == "a transposed column":
        return torch.randn(WIDTH, 1).half().t()
    return torch.randn(WIDTH).half().as_strided((1, WIDTH), (0, 1))


@pytest.mark.parametrize("kind", ["of a buffer with an odd pitch", "a transposed column", "stride 0"])
def test_a_single_row_has_the_stride_of_a_row(lib, kind):
    impl, cache = impl_and_cache()
    meta, _ = batch(1)
    q, k, v = (one_row(kind) for _ in range(3))
    out = impl.forward(q, k, v, cache, None, meta)
    (name, a), = lib.calls
    assert name == "aps_plain_decode_step"
    assert a[15:19] == (WIDTH,) * 4   # of query, key, value and output
    assert out.shape == (1, WIDTH) and out.stride() == (WIDTH, 1)


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("slots", [2, 3, 5])
def test_no_slot_without_a_row(lib, monkeypatch, general, slots):
    """A padded slot mapping names rows of key and value that do not exist."""
    impl, cache = impl_and_cache()
    if general:
        monkeypatch.setattr(impl, "_plain_decode", lambda *a: None)
    meta, (q, k, v) = batch(3, slots=slots)
    impl.forward(q, k, v, cache, None, meta)
    name, a = lib.calls[0]
    assert (name, a[5 + 2 * (not general)]) == (("aps_reshape_and_cache", min(slots, 3)) if general else
                                                ("aps_plain_decode_step", min(slots, 3)))


@pytest.mark.parametrize("what", [dict(table_rows=2), dict(lens=2)])
def test_tables_and_lengths_of_fewer_requests_are_refused(lib, what):
    impl, cache = impl_and_cache()
    meta, (q, k, v) = batch(3, **what)
    assert impl._plain_decode(q, k, v, cache, meta) is None
    with pytest.raises(RuntimeError, match="for 3 requests"):
        impl.forward(q, k, v, cache, None, meta)
    assert not any("attention" in name or "plain" in name for name, _ in lib.calls)


def test_tables_and_lengths_of_more_requests_are_taken(lib):
    impl, cache = impl_and_cache()
    meta, (q, k, v) = batch(3, table_rows=5, lens=4)
    impl.forward(q, k, v, cache, None, meta)
    assert [name for name, _ in lib.calls] == ["aps_plain_decode_step"]
