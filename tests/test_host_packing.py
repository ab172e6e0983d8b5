"""The host side of expand_decode_metadata: the native reading of the lists gives what numpy gives."""
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
