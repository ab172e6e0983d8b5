"""The gathered input of a decode batch in one pass against the three operations it stands for, bit for bit."""
import pytest
import torch

from apt_serve_b200 import attention as A
from apt_serve_b200 import mixed_cache_ops as M

pytestmark = pytest.mark.gpu


def three(hidden, cache, slots, new_rows, cached, rows):
    out = torch.zeros(rows, hidden.shape[1], device=hidden.device, dtype=hidden.dtype)
    out[new_rows] = hidden
    M.cache_to_hidden(out, cache, slots, cached)
    return out


# rows of one piece and of two (more than 16 KB), too short for the one pass, not aligned; more rows than a CTA and than all CTAs of the
# map's kernels have threads; rows that nothing is written to, rows of both kinds, slots of -1, indices from the end
@pytest.mark.parametrize("e,dtype,rows,n_new,one_pass", [
    (256, torch.float16, 3, 1, True), (5120, torch.float16, 700, 12, True), (9216, torch.bfloat16, 65, 5, True),
    (768, torch.float32, 2500, 40, True), (256, torch.bfloat16, 310000, 700, True),
    (128, torch.float16, 90, 7, False), (260, torch.float16, 90, 7, False),
])
@pytest.mark.parametrize("strided", [False, True])
def test_gather_is_the_three_operations(e, dtype, rows, n_new, one_pass, strided, monkeypatch):
    g = torch.Generator().manual_seed(rows)
    blocks = rows // 16 + 2
    cache = torch.randn(2, blocks, 16, 1, e, generator=g).to("cuda", dtype)
    hidden = torch.randn(n_new, 2 * e if strided else e, generator=g).to("cuda", dtype)[:, :e]
    order = torch.randperm(rows, generator=g)
    new_rows = order[:n_new].clone()
    new_rows[0] -= rows
    cached = order[n_new // 2: rows - rows // 5] if rows > 3 else order[1:2]
    slots = torch.randperm(2 * blocks * 16, generator=g)[:rows]
    slots[cached[::7]] = -1
    new_rows, cached, slots = new_rows.cuda(), cached.contiguous().cuda(), slots.cuda()
    want = three(hidden, cache, slots, new_rows, cached, rows)
    if one_pass:
        monkeypatch.setattr(M, "cache_to_hidden", None)   # not by the three operations
    got = M.gather_hidden_rows(hidden, cache, slots, new_rows, cached, rows)
    assert torch.equal(got, want)


def test_gather_keeps_graphs_and_other_indices():
    cache = torch.randn(2, 4, 16, 1, 256, device="cuda", dtype=torch.float16)
    hidden = torch.randn(2, 256, device="cuda", dtype=torch.float16)
    slots, cached = torch.arange(8, device="cuda"), torch.tensor([0, 1, 2, 4, 5], device="cuda")
    want = three(hidden, cache, slots, torch.tensor([3, 7], device="cuda"), cached, 8)
    at = torch.tensor([3, 7], dtype=torch.int32, device="cuda")
    mask = torch.zeros(8, dtype=torch.bool, device="cuda")
    mask[3] = mask[7] = True
    for rows in (at, mask):
        assert torch.equal(M.gather_hidden_rows(hidden, cache, slots, rows, cached, 8), want)
    leaf = hidden.clone().requires_grad_()
    assert M.gather_hidden_rows(leaf, cache, slots, at.long(), cached, 8).requires_grad


@pytest.mark.parametrize("new,cached", [([3, 8], [0, 1]), ([3, -9], [0, 1]), ([3, 7], [0, 8]), ([3, 7], [-1, 0])])
def test_indices_outside_the_rows_are_left_out_and_reported(new, cached):
    cache = torch.randn(2, 4, 16, 1, 256, device="cuda", dtype=torch.float16)
    hidden, slots = torch.randn(2, 256, device="cuda", dtype=torch.float16), torch.arange(8, device="cuda")
    index = lambda rows: torch.tensor(rows, device="cuda")
    A.raise_on_device_status()
    got = M.gather_hidden_rows(hidden, cache, slots, index(new), index(cached), 8)
    with pytest.raises(RuntimeError, match="outside its tensors"):
        A.raise_on_device_status()
    A.raise_on_device_status()   # said once
    inside = [i for i, t in enumerate(new) if -8 <= t < 8]
    assert torch.equal(got, three(hidden[inside], cache, slots, index([new[i] for i in inside]), index([t for t in cached if 0 <= t < 8]), 8))
