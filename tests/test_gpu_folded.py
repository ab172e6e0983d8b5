"""The layer-step's hidden path with the projections moved to the query and the output
(csrc/hidden_attention.cu) at the sizes where its tiles, stages, groups and splits end.

Tolerance of the hidden-cached requests' rows: the intermediates carry at least 22 bits (fp16: down to 2^-36), so what is left
is the rounding of the output, half a unit of its last place (u = 2^-11 of the value in fp16, 2^-8 in bf16),
and an eighth of that, relative to the rows' root mean square, for the sums and the oracle's own fp32.
K/V-cached requests: the 2e-2 of the other attention tests (their weights are rounded to the cache type)."""
import numpy as np
import pytest
import torch

from oracle import hybrid_cache_oracle as O
from apt_serve_b200 import _native as N
from apt_serve_b200 import attention as A
from apt_serve_b200.workloads import LayerShape, make_decode_workload

from helpers import assert_close

pytestmark = pytest.mark.gpu

HALF_ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def run_step(w):
    m = w.meta
    d = w.shape
    args = (len(w.seq_lens), m.private_block_tables.shape[1], d.block_size, w.heads, d.head_dim)
    assert (N.lib().aps_decode_layer_step_workspace_bytes(*args, d.hidden, N.DTYPE_ENUM[d.dtype])
            > N.lib().aps_attention_workspace_bytes(*args)), "this size does not take the path under test"
    wk, bk, wv, bv = w.kv_weights()
    out = A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache,
                              wk, bk, wv, bv, m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale)
    A.raise_on_device_status()
    return out


def check(w_cpu, what):
    w = w_cpu.to("cuda")
    out = run_step(w)
    again = run_step(w)
    assert torch.equal(out, again), f"{what}: two runs on the same inputs differ"
    ref = O.decode_layer_step(w_cpu.hidden_states, w_cpu.query, w_cpu.new_key, w_cpu.new_value, w_cpu.kv_cache,
                              w_cpu.hidden_cache, *w_cpu.kv_weights(), w_cpu.meta, w_cpu.scale)
    hid = [r for r, u in enumerate(w_cpu.use_hidden) if u]
    kv = [r for r, u in enumerate(w_cpu.use_hidden) if not u]
    if hid:
        x, y = out[hid].float().cpu(), ref[hid].float()
        u = HALF_ULP[w_cpu.shape.dtype]
        rms = y.pow(2).mean(dim=1, keepdim=True).sqrt()
        bad = ~((x - y).abs() <= u * y.abs() + u / 8 * rms)
        assert not bad.any(), (what, int(bad.sum()), float(((x - y).abs() / rms).max()))
    if kv:
        assert_close(out[kv], ref[kv], what)


F, B = torch.float16, torch.bfloat16
# (heads, head size, hidden, dtype, lengths, every how many requests one is K/V-cached)
CASES = {
    "edges of tiles and stages": (8, 128, 1024, F, (1, 15, 16, 17, 31, 32, 33, 255, 256, 257, 511, 512, 513, 529), 0),
    "the same in bf16, mixed": (8, 128, 1024, B, (1, 15, 16, 17, 31, 32, 33, 255, 256, 257, 511, 512, 513, 529), 4),
    "one long request": (40, 128, 512, F, (2048,), 0),
    "one token": (72, 128, 256, B, (1, 257), 0),
    "heads not a multiple of 16, wide rows": (9, 128, 9216, B, (300, 17, 640, 1, 256, 120, 900), 3),
    "two heads per row tile": (5, 64, 384, F, (300, 17, 640, 1, 256, 120, 900), 3),
    "four heads per row tile": (33, 32, 256, B, (300, 17, 640, 1, 256, 120, 900), 0),
    "a narrow hidden size": (12, 64, 128, F, (700, 5, 90, 1, 64), 0),
    "fewer projection rows than a tile": (1, 64, 128, F, (700, 5, 90), 0),
    "wide accumulators": (160, 32, 128, F, (70, 260, 5, 90), 0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_step_against_the_oracle(name):
    heads, d, e, dtype, lens, every = CASES[name]
    hidden = [not (every and i % every == 1) for i in range(len(lens))]
    w = make_decode_workload(LayerShape("t", heads, d, e, dtype), list(lens), hidden, seed=len(lens), device="cpu")
    check(w, name)


@pytest.mark.parametrize("n_hidden", [256, 257, 600])
def test_groups_of_hidden_requests(n_hidden):
    rng = np.random.default_rng(n_hidden)
    lens = [int(x) for x in rng.integers(1, 60, size=n_hidden + 20)]
    hidden = [True] * n_hidden + [False] * 20
    order = rng.permutation(len(lens))
    w = make_decode_workload(LayerShape("t", 4, 64, 256, F), [lens[i] for i in order], [hidden[i] for i in order],
                             seed=2, device="cpu")
    check(w, f"{n_hidden} hidden requests")


def test_larger_cache_blocks_and_garbage_behind_the_sequences():
    lens = [21, 150, 40, 511, 256, 33, 1030]
    w = make_decode_workload(LayerShape("t", 8, 128, 1024, F, block_size=32), lens, [True] * len(lens), seed=6, device="cpu")
    rows = O.flat_rows(w.hidden_cache)
    for r, s in enumerate(lens):
        if s % 32:
            last = w.block_tables[r][-1]
            rows[last * 32 + s % 32: last * 32 + 32] = float("nan")
    check(w, "garbage tail")


def test_small_and_large_queries_keep_their_bits():
    """The folded query is normalised per request and head: queries of very different sizes.  (Rows and weights: below.)"""
    w = make_decode_workload(LayerShape("t", 8, 128, 1024, F), [300] * 12, [True] * 12, seed=8, device="cpu")
    for r, s in enumerate((1e-6, 1e-4, 1e-2, 1.0, 8.0, 30.0, 1e-6, 1e-4, 1e-2, 1.0, 8.0, 0.0)):
        w.query[r] *= s
    check(w, "query sizes")


@pytest.mark.parametrize("dtype", [F, B, torch.float32])
def test_unaligned_weights_are_re_projected(dtype):
    """Head counts that do not fill a tile take weights of any alignment and row stride, as the CUDA-core kernel always has."""
    w = make_decode_workload(LayerShape("t", 5, 64, 384, dtype), [300, 17, 640, 1], [True, True, False, True], seed=3, device="cuda")
    m, (wk, bk, wv, bv) = w.meta, w.kv_weights()
    wide = torch.zeros(2, wk.shape[0], wk.shape[1] + 3, dtype=dtype, device="cuda")[:, :, 1:-2]
    wide[0], wide[1] = wk, wv
    assert wide[0].data_ptr() % 16 and wide.stride(1) % 4
    step = lambda k, v: A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, k,
                                            bk, v, bv, m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale)
    want, got = step(wk, wv), step(wide[0], wide[1])
    A.raise_on_device_status()
    u = {F: 2.0 ** -10, B: 2.0 ** -7, torch.float32: 1e-5}[dtype]   # both roundings of the output
    assert torch.allclose(got.float(), want.float(), rtol=u, atol=u * float(want.float().pow(2).mean().sqrt()))


def attention64(w, r):
    """Hidden-cached request r (its new row written) in 64 bits."""
    m, s, h, d, bs = w.meta, w.seq_lens[r], w.heads, w.shape.head_dim, w.shape.block_size
    t = torch.arange(s)
    rows = m.private_block_tables[r].cpu().long()[t // bs] * bs + t % bs
    x = O.flat_rows(w.hidden_cache.cpu())[rows].double()
    wk, bk, wv, bv = (y.cpu().double() for y in w.kv_weights())
    k, v = (x @ wk.T + bk).view(s, h, d), (x @ wv.T + bv).view(s, h, d)
    p = torch.softmax(torch.einsum("hd,thd->ht", w.query[r].cpu().double().view(h, d), k) * w.scale, dim=1)
    return torch.einsum("ht,thd->hd", p, v).reshape(-1)


# (heads, head size, hidden): one instruction per step for both terms of the folded query, and one for each
@pytest.mark.parametrize("heads,d,e", [(8, 128, 1024), (160, 32, 128)])
@pytest.mark.parametrize("rows,w_k", [(1.0, 0.02), (0.1, 0.02), (1e-2, 0.02), (1e-3, 0.02), (1.0, 1e-3), (1.0, 1e-4), (1e-4, "large")])
def test_rows_and_weights_of_any_size_keep_their_bits(rows, w_k, heads, d, e):
    """fp16 has few exponents: cached rows N(0, rows) against W_v of N(0, 1), W_k from N(0, 1e-4) up to entries whose
    folded queries (2 sum |W_k| over a head's rows) pass the largest fp16.  The bound is that of the oracle's
    cases, and half the spacing of the subnormal numbers for an output among them."""
    w = make_decode_workload(LayerShape("t", heads, d, e, F), [300, 17, 600, 1], [True] * 4, seed=9, device="cpu")
    hd = heads * d
    w.kv_cache.mul_(rows)
    if w.hidden_cache.data_ptr() != w.kv_cache.data_ptr():
        w.hidden_cache.mul_(rows)
    w.hidden_states.mul_(rows)
    w.qkv_weight[2 * hd:].mul_(50.0)
    w.qkv_bias.zero_()
    if w_k == "large":
        w.query.abs_().clamp_(max=0.4).add_(1.5)
        w.qkv_weight[hd:2 * hd].add_(1.0).mul_(51200.0 / d)
        assert float((w.query[0, :d].double() @ w.qkv_weight[hd:hd + d].double()).min()) > 65504
    else:
        w.qkv_weight[hd:2 * hd].mul_(w_k / 0.02)
    w = w.to("cuda")
    out = run_step(w).cpu().double()
    for r in range(4):
        y = attention64(w, r)
        bad = ~((out[r] - y).abs() <= 2.0 ** -11 * y.abs() + 2.0 ** -14 * y.pow(2).mean().sqrt() + 2.0 ** -25)
        assert not bad.any(), (r, int(bad.sum()), float(((out[r] - y).abs() / y.pow(2).mean().sqrt()).max()))


# Distance from 64 bits before the output's rounding, relative to the outputs' root mean square, that the re-projecting kernel
# shows on the same requests: about 6e-6 for 5120 columns, 3e-6 for 2048 (both types).
@pytest.mark.parametrize("heads,d,e,dtype,most", [(40, 128, 5120, F, 6.2e-6), (40, 128, 5120, B, 6.2e-6),
                                                  (32, 64, 2048, F, 3.2e-6), (32, 64, 2048, B, 3.2e-6)])
@pytest.mark.parametrize("others", [0, 120])
def test_sums_keep_their_bits_over_long_sequences(heads, d, e, dtype, most, others):
    """A value bias that cancels one request's output leaves what it lost before its rounding to be seen."""
    w = make_decode_workload(LayerShape("t", heads, d, e, dtype), [2048, 700] + [40] * others, [True] * (2 + others),
                             seed=4, device="cuda")
    hd = heads * d
    w.qkv_weight[hd:2 * hd].mul_(0.05)   # weights of similar size: every token counts
    w.qkv_bias.zero_()
    run_step(w)
    for r in range(2):
        y = attention64(w, r).cuda()
        w.qkv_bias[2 * hd:] = (-y).to(dtype)
        lost = run_step(w)[r].double() - (y + w.qkv_bias[2 * hd:].double())
        w.qkv_bias.zero_()
        assert float(lost.pow(2).mean().sqrt() / y.pow(2).mean().sqrt()) <= most


def _step_into(w, out, ws):
    m, (wk, bk, wv, bv) = w.meta, w.kv_weights()
    return A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, wk, bk, wv,
                               bv, m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale, out=out, workspace=ws)


def _chain_workloads():
    lens = [300, 17, 640, 1, 256, 120, 900, 33]
    return [make_decode_workload(LayerShape("t", 8, d, 1024, t), [x + 3 * i for x in lens], h, seed=30 + i, device="cuda")
            for i, (d, t, h) in enumerate([(128, F, [True, False] * 4), (64, B, [True] * 8), (128, B, [False, True] * 4),
                                           (64, F, [True, True, False, False] * 2)])]


def test_steps_that_follow_each_other_on_one_scratch():
    """The launches of a step overlap; steps of different shapes, enqueued without a wait between them on one
    scratch, with the step's inputs written just before it, give what each gives alone."""
    ws = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    ws_kv = A.attention_workspace(ws.device, 8, 64, 16, 8, 128)
    cases = _chain_workloads()
    want = []
    for w in cases:
        want.append((_step_into(w, torch.empty_like(w.query), ws), A.paged_decode_attention(
            w.query, w.kv_cache[0], w.kv_cache[1], w.meta.private_block_tables % w.kv_cache.shape[1], w.meta.seq_lens_tensor,
            w.scale, workspace=ws_kv)))
        torch.cuda.synchronize()
    live = [w.query.clone() for w in cases]
    for _ in range(20):
        got = []
        for w, q in zip(cases, live):
            w.query.zero_()
            out = torch.full_like(w.query, float("nan"))
            w.query.copy_(q)
            got.append((_step_into(w, out, ws), A.paged_decode_attention(
                w.query, w.kv_cache[0], w.kv_cache[1], w.meta.private_block_tables % w.kv_cache.shape[1],
                w.meta.seq_lens_tensor, w.scale, workspace=ws)))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_chained_step_replays_from_a_cuda_graph():
    ws = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    for w in _chain_workloads()[:2]:
        want = _step_into(w, torch.empty_like(w.query), ws).clone()
        torch.cuda.synchronize()
        out, g = torch.empty_like(w.query), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            _step_into(w, out, ws)
            _step_into(w, out, ws)
        for _ in range(3):
            out.zero_()
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("dtype", [F, B])
@pytest.mark.parametrize("n_hidden", [100, 150])
def test_wide_slices_of_the_weighted_sums(n_hidden, dtype):
    """Enough requests for slices of three (the last one of two) and of four 128-column blocks in fp16, of two in bf16."""
    rng = np.random.default_rng(n_hidden)
    lens = [int(x) for x in rng.integers(1, 100, size=n_hidden)]
    w = make_decode_workload(LayerShape("t", 5, 128, 1024, dtype), lens, [True] * n_hidden, seed=3, device="cpu")
    check(w, f"{n_hidden} requests")
