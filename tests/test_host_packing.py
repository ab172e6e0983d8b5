"""The host side of expand_decode_metadata: the native reading of the lists gives what numpy gives."""
import contextlib
import ctypes
import threading

import numpy as np
import pytest
import torch

from apt_serve_b200 import _native as N
from apt_serve_b200 import device_metadata as DM


def both(monkeypatch, lens, hid, tables, shared):
    """(measured, buffer) with the host library and without it."""
    got = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(N, "host_lib", lambda: None)
        b = len(lens)
        m_lens, types, counts = DM._measure(lens, hid, tables, b)
        n_h, width = counts[0], counts[2]
        cuts = DM._cuts((2 * (b - n_h), b * width, b * width, b * width, b, b), 32)
        host = torch.full((sum(cuts),), -1, dtype=torch.int32)
        DM._fill_host(host, cuts, tables, shared, m_lens, types, width, n_h)
        got.append((m_lens.tolist(), types.tolist(), counts, [t.tolist() for t in host.split(cuts)[::2]]))
    return got


@pytest.mark.parametrize("kind", ["mixed", "all hidden", "none hidden", "tuples", "one", "numpy integers", "numpy booleans"])
def test_native_and_numpy_agree(monkeypatch, kind):
    if N.host_lib() is None:
        pytest.skip("the host library has not been built")
    rng = np.random.default_rng(3)
    lens = [17] if kind == "one" else [1, 16, 17, 300, 5]
    b = len(lens)
    hid = [True] * b if kind == "all hidden" else [False] * b if kind == "none hidden" else [i % 2 == 0 for i in range(b)]
    make = lambda s: [int(x) for x in rng.integers(0, 2 ** 31 - 1, size=-(-s // 16))]
    tables, shared = [make(s) for s in lens], [make(s) if h else [] for s, h in zip(lens, hid)]
    if kind == "tuples":
        tables, shared = [tuple(t) for t in tables], [tuple(t) for t in shared]
    if kind == "numpy integers":
        lens, tables = [np.int64(s) for s in lens], [[np.int32(x) for x in t] for t in tables]
    if kind == "numpy booleans":
        hid = [np.bool_(h) for h in hid]
    native, plain = both(monkeypatch, lens, hid, tables, shared)
    assert native == plain
    assert native[2] == (sum(map(bool, hid)), sum(int(s) for s, h in zip(lens, hid) if h), max(map(len, tables)), min(lens), max(lens))


@pytest.mark.parametrize("tables,shared", [([[1], [2 ** 31]], [[1], []]), ([[1], ["x"]], [[1], []]), ([[1], [2]], [[1, 2, 3], []])])
def test_what_numpy_refuses_is_refused(tables, shared):
    lens, types, counts = DM._measure([1, 2], [True, False], tables, 2)
    cuts = DM._cuts((2, 2 * counts[2], 2 * counts[2], 2 * counts[2], 2, 2), 32)
    with pytest.raises((ValueError, OverflowError)):
        DM._fill_host(torch.zeros(sum(cuts), dtype=torch.int32), cuts, tables, shared, lens, types, counts[2], 1)


def unpacked(lens, hid, tables, shared, changes=False):
    """What the native reading lays out one behind the other, as lists: K/V-cached rows, lengths, types, and the rows of both tables."""
    read = DM._read_lists(lens, hid, tables, shared, len(lens), 16)
    if read is None:
        return None
    m_lens, counts, (n_own, n_shared, too_long), packed = read
    if not changes:
        assert too_long == DM._first_too_long(m_lens, np.array(hid), tables, shared, 16)
    b, n_kv = len(m_lens), len(m_lens) - counts[0]
    rows = np.frombuffer(packed, np.int64, n_kv)
    words = np.frombuffer(packed, np.int32)[2 * n_kv:]
    got_lens, types, own_at, shared_at, own, extra = np.split(words, np.cumsum([b, b, b + 1, b + 1, n_own]))
    assert m_lens.tolist() == got_lens.tolist() and len(extra) == n_shared
    cut = lambda at, entries: [entries[x:y].tolist() for x, y in zip(at, at[1:])]
    assert own_at[0] == shared_at[0] == 0 and own_at[-1] == n_own and shared_at[-1] == n_shared
    return rows.tolist(), got_lens.tolist(), types.tolist(), cut(own_at, own), cut(shared_at, extra), counts


needs_host_library = pytest.mark.skipif(N.host_lib() is None, reason="the host library has not been built")


@needs_host_library
@pytest.mark.parametrize("hid", [[True, False, True, False], [True] * 4, [False] * 4])
@pytest.mark.parametrize("row", [list, tuple])
def test_lists_are_read_as_they_are(hid, row):
    lens, tables = [33, 1, 16, 5], [row([1, 2, 3]), row([4]), row([2 ** 30, 2 ** 31 - 1]), row([])]
    shared = [row([7, 8]) if h else "not looked at" for h in hid]
    got = unpacked(lens, hid, tables, shared)
    counts = (sum(hid), sum(s for s, h in zip(lens, hid) if h), 3, 1, 33)
    assert got == ([r for r in range(4) if not hid[r]], lens, [int(h) for h in hid], [list(t) for t in tables],
                   [[7, 8] if h else [] for h in hid], counts)


@needs_host_library
@pytest.mark.parametrize("lens,hid,tables,shared", [
    ([1, 2], [True, False], [[1], [2 ** 31]], [[1], []]), ([1, 2], [True, False], [[1], ["x"]], [[1], []]),
    ([1, 2], [True, False], [[1], [2]], [[1, 2, 3], []]), ([1, 2], [True, False], [[1], [2]], [[1]]),
    ([1, 2], [True, 0], [[1], [2]], [[1], []]), ([1, np.int64(2)], [True, False], [[1], [2]], [[1], []]),
    ((1, 2), [True, False], [[1], [2]], [[1], []]), ([1, 2], [True, False], [[1], np.array([2])], [[1], []]),
    ([1, 2], [True, False], [[1], [2]], [None, []]), ([1, True], [True, False], [[1], [2]], [[1], []]),
])
def test_what_is_not_plain_is_left_to_numpy(lens, hid, tables, shared):
    assert DM._read_lists(lens, hid, tables, shared, 2, 16) is None


@needs_host_library
def test_tables_that_change_while_they_are_read():
    """Another thread lengthens, shortens and replaces rows: what is read is the lists of one moment, never a size of one and
    entries of another."""
    b = 64
    row = lambda r, n: [1000 * r + i for i in range(n)]
    tables, shared = [row(r, 40) for r in range(b)], [row(r, 30) for r in range(b)]
    stop = threading.Event()

    def change():
        rng = np.random.default_rng(1)
        while not stop.is_set():
            r, n = int(rng.integers(b)), int(rng.integers(1, 200))
            which = tables if n & 1 else shared
            if n % 3 == 0:
                which[r] = row(r, n)
            elif n % 3 == 1:
                which[r].append(1000 * r + len(which[r])) if len(which[r]) < 400 else which[r].clear()
            else:
                del which[r][len(which[r]) // 2:]

    other = threading.Thread(target=change)
    other.start()
    read = 0
    try:
        for _ in range(3000):
            got = unpacked([5] * b, [r % 2 == 0 for r in range(b)], tables, shared, changes=True)
            if got is None:   # a shared table wider than all private ones
                continue
            read += 1
            for r in range(b):
                assert got[3][r] == row(r, len(got[3][r]))
                assert got[4][r] == (row(r, len(got[4][r])) if r % 2 == 0 else [])
            assert got[5][2] == max(1, max(map(len, got[3])))
    finally:
        stop.set()
        other.join()
    assert read > 0


@needs_host_library
def test_a_table_that_grows_during_the_call_stays_inside_the_buffer(monkeypatch):
    """The staging buffer's allocation gives the interpreter lock away; here it lengthens a table itself, as another thread may."""
    tables, shared = [[1, 2], [3, 4, 5]], [[7, 8], []]
    guard, real, buffers, called = 64, torch.empty, [], []

    def empty(*size, pin_memory=False, **kw):
        if buffers or len(size) != 1:
            return real(*size, **kw)
        tables[1].extend(range(100, 120))
        buffers.append(torch.full((size[0] + guard,), -99, **kw))
        return buffers[0][:size[0]]

    class Library:
        def aps_expand_decode_lists(self, entries, starts, *rest):
            at = np.frombuffer(ctypes.string_at(starts, 12), np.int32).tolist()
            called.append([np.frombuffer(ctypes.string_at(entries + 4 * x, 4 * (y - x)), np.int32).tolist() for x, y in zip(at, at[1:])])
            return N.APS_OK

    monkeypatch.setattr(DM.torch, "empty", empty)
    monkeypatch.setattr(N, "lib", Library)
    monkeypatch.setattr(N, "current_stream", lambda dev: 0)
    monkeypatch.setattr(N, "on_device", lambda dev: contextlib.nullcontext())
    DM.expand_decode_metadata([20, 40], [True, False], tables, shared, 16, "cpu")
    assert (buffers[0][-guard:] == -99).all()
    assert called == [[[1, 2], [3, 4, 5]]]


# one token more than there is room for: in the private table of either kind of request, in the shared one, in an empty or missing
# one; rows that numpy reads as well as plain ones.  Refused before anything is launched or copied.
@pytest.mark.parametrize("lens,hid,tables,shared,which", [
    ([100], [True], [[1]], [[2]], 0), ([16, 17], [False, False], [[1], [2]], [[], []], 1),
    ([16, 33], [False, True], [[1], [2, 3]], [[], [4, 5, 6]], 1), ([33], [True], [[1, 2, 3]], [[4, 5]], 0),
    ([1, 1], [True, False], [[1], []], [[2], []], 1), ([5, 33, 40], [True, True, False], [[1], [2, 3], [4]], [[1], [2, 3], []], 1),
    ([1, 1], [False, True], [[1], [2]], [[]], 1),
])
@pytest.mark.parametrize("rows", ["plain", "numpy rows", "numpy lengths", "no library"])
def test_requests_longer_than_their_tables_are_refused(monkeypatch, lens, hid, tables, shared, which, rows):
    if rows == "numpy rows":
        tables = [np.array(t, dtype=np.int32) for t in tables]
    elif rows == "numpy lengths":
        lens = [np.int64(s) for s in lens]
    elif rows == "no library":
        monkeypatch.setattr(N, "host_lib", lambda: None)
    monkeypatch.setattr(N, "lib", None)
    with pytest.raises(ValueError, match=f"request {which} has {lens[which]} tokens"):
        DM.expand_decode_metadata(lens, hid, tables, shared, 16, "cpu")
    from apt_serve_b200.metadata import build_decode_metadata
    with pytest.raises(IndexError):
        build_decode_metadata(lens, hid, tables, shared, 16)
