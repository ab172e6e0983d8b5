"""The fp32 layer-step with the projections moved to the query and the output (csrc/hidden_fp32.cu), at the sizes
where its chunks, groups and column ranges end, against the same attention in 64 bits and against the
re-projecting kernel: its distance from the former may not exceed the latter's.

Tolerance: an output is a few sums of E, D and T rounded terms, errors of independent sign of 2^-24 each, and the
scores' errors enter the weights multiplied by at most a few: 16 x 2^-24 x sqrt(E + T) of the rows' root mean square."""
import numpy as np
import pytest
import torch

from oracle import hybrid_cache_oracle as O
from apt_serve_b200 import _native as N
from apt_serve_b200 import attention as A
from apt_serve_b200.workloads import LayerShape, make_decode_workload

pytestmark = pytest.mark.gpu


def reference64(w, r):
    """Request r (hidden-cached, its new row written) in 64 bits."""
    m, s, h, d = w.meta, w.seq_lens[r], w.heads, w.shape.head_dim
    bs = w.shape.block_size
    t = torch.arange(s)
    rows = m.private_block_tables[r].cpu().long()[t // bs] * bs + t % bs
    x = O.flat_rows(w.hidden_cache.cpu())[rows].double()
    wk, bk, wv, bv = (y.cpu().double() for y in w.kv_weights())
    k, v = (x @ wk.T + bk).view(s, h, d), (x @ wv.T + bv).view(s, h, d)
    q = w.query[r].cpu().double().view(h, d)
    p = torch.softmax(torch.einsum("hd,thd->ht", q, k) * w.scale, dim=1)
    return torch.einsum("ht,thd->hd", p, v).reshape(-1)


def re_projected(w):
    """The same attention by the re-projecting kernel, which a call with the plain attention scratch takes."""
    m, d = w.meta, w.shape
    need = N.lib().aps_attention_workspace_bytes(len(w.seq_lens), m.private_block_tables.shape[1], d.block_size, w.heads, d.head_dim)
    return A.hybrid_decode_attention(w.query, w.kv_cache, w.hidden_cache, *w.kv_weights(), m.private_block_tables,
                                     m.seq_lens_tensor, m.cache_type, w.scale,
                                     workspace=torch.empty(need, dtype=torch.uint8, device="cuda"))


# (heads, head size, hidden, block size, lengths, every how many requests one is K/V-cached)
CASES = {
    "edges of chunks": (12, 64, 768, 16, (1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 129, 300), 0),
    "mixed": (12, 64, 768, 16, (230, 1, 64, 300, 16, 15, 700, 2), 3),
    "heads not a multiple of four, ragged columns": (5, 128, 260, 16, (90, 1, 300, 64), 0),
    "one head, fewer columns than a warp takes": (1, 32, 36, 32, (70, 5), 0),
    "one long request": (3, 64, 1028, 16, (2500,), 0),
    "larger blocks, wide rows": (6, 128, 2304, 64, (300, 17, 640, 1), 2),
}


@pytest.mark.parametrize("name", list(CASES))
def test_step_against_64_bits(name):
    heads, d, e, bs, lens, every = CASES[name]
    hidden = [not (every and i % every == 1) for i in range(len(lens))]
    w = make_decode_workload(LayerShape("t", heads, d, e, torch.float32, block_size=bs), list(lens), hidden, seed=3, device="cuda")
    m, weights = w.meta, w.kv_weights()
    args = (len(lens), m.private_block_tables.shape[1], bs, heads, d)
    assert (N.lib().aps_decode_layer_step_workspace_bytes(*args, e, N.DTYPE_ENUM[torch.float32])
            > N.lib().aps_attention_workspace_bytes(*args)), "this size does not take the path under test"
    step = lambda: A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, *weights,
                                       m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale)
    out = step()
    A.raise_on_device_status()
    assert torch.equal(out, step())
    old = re_projected(w)
    new_err = old_err = 0.0
    for r, u in enumerate(hidden):
        if not u:
            assert torch.equal(out[r], old[r])
            continue
        y = reference64(w, r)
        rms = float(y.pow(2).mean().sqrt())
        diff = (out[r].cpu().double() - y).abs()
        assert float(diff.max()) <= 16 * 2.0 ** -24 * (e + lens[r]) ** 0.5 * rms, (name, r, float(diff.max()) / rms)
        new_err += float(diff.pow(2).sum())
        old_err += float((old[r].cpu().double() - y).pow(2).sum())
    print(f"{name}: relative to the re-projecting kernel's {old_err ** 0.5:.2e}: {new_err ** 0.5:.2e}")
    assert new_err ** 0.5 <= 1.1 * old_err ** 0.5


def test_groups_and_chunks_of_a_wide_batch():
    """300 hidden-cached requests (two groups of the plan) whose tables allow so many tokens that the scratch takes
    longer chunks and fewer requests at a time."""
    rng = np.random.default_rng(0)
    lens = [int(x) for x in rng.integers(1, 130, size=300)]
    w = make_decode_workload(LayerShape("t", 8, 32, 512, torch.float32), lens, [i % 7 != 3 for i in range(300)], seed=4, device="cuda")
    m, weights = w.meta, w.kv_weights()
    wide = torch.zeros(300, 4096, dtype=torch.int32, device="cuda")
    wide[:, :m.private_block_tables.shape[1]] = m.private_block_tables
    outs = [A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, *weights, t,
                                m.seq_lens_tensor, m.cache_type, w.scale) for t in (m.private_block_tables, wide)]
    old = re_projected(w)
    rms = old.pow(2).mean(dim=1, keepdim=True).sqrt()
    for o in outs:
        assert bool(((o - old).abs() <= 32 * 2.0 ** -24 * 642 ** 0.5 * rms).all())


def test_rows_behind_the_sequence_are_not_read_into_it():
    w = make_decode_workload(LayerShape("t", 4, 64, 256, torch.float32), [21, 150, 40], [True] * 3, seed=6, device="cpu")
    rows = O.flat_rows(w.hidden_cache)
    for r, s in enumerate(w.seq_lens):
        last = w.block_tables[r][-1]
        rows[last * 16 + s % 16: last * 16 + 16] = float("nan")
    w = w.to("cuda")
    m = w.meta
    out = A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, *w.kv_weights(),
                              m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale)
    assert torch.isfinite(out).all()
