"""Branches of the layer-step's kernels that depend on how much work a batch is (csrc/hidden_attention.cu, csrc/paged_attention.cu),
against the oracle with the tolerances of test_gpu_folded.py."""
import pytest
import torch

from oracle import hybrid_cache_oracle as O
from apt_serve_b200 import attention as A
from apt_serve_b200.workloads import LayerShape, make_decode_workload

from helpers import assert_close
from test_gpu_folded import check

pytestmark = pytest.mark.gpu
F, B = torch.float16, torch.bfloat16
NONE = -2 ** 31   # cache type of a request without usable tables


def workload(heads, d, e, dtype, lens, hidden, device="cpu"):
    return make_decode_workload(LayerShape("t", heads, d, e, dtype), lens, hidden, seed=len(lens) + heads, device=device)


# softmax: single heads (few units) and pairs of heads, the last one alone; more tokens than a CTA's registers hold (2048)
@pytest.mark.parametrize("heads,dtype,lens", [
    (5, F, (4200, 3, 2049)), (5, B, (4200, 3, 2049)),
    (33, F, (2049, 17, 600, 1, 255, 256, 257, 16, 90, 4100, 31, 32)), (48, B, (2049, 17, 600, 1, 255, 256, 257, 16)),
])
def test_softmax_units(heads, dtype, lens):
    check(workload(heads, 64, 128, dtype, list(lens), [True] * len(lens)), f"{heads} heads, {len(lens)} requests")


def slice_of_the_sums(heads, e, dtype, n, sms=148):
    """Column blocks per item of the weighted sums that the plan gives n hidden-cached requests (csrc/hidden_attention.cu)."""
    terms, np_, steps = 2 if dtype == F else 3, -(-heads // 16) * 16, -(-e // 128)
    turns = lambda s: 4 if 5 * s * np_ <= 256 else 2 if 3 * s * np_ <= 256 else 1
    fits = lambda s: terms * np_ <= 256 and (terms - 1 + turns(s)) * s * np_ <= 256
    most = next(s for s in (4, 3, 2, 1) if s == 1 or 2 * s * np_ <= 256)
    if fits(1) and (fits(2) or 4 * np_ > 256):
        most = next(s for s in range(most, 0, -1) if all(map(fits, range(2, s + 1))))
    return next(s for s in range(min(most, steps), 0, -1) if s == 1 or n * -(-steps // s) >= 2 * sms)


# weighted sums: terms in one instruction or one for each, one, two and four turns of accumulators, stages of two and four cache blocks;
# lengths around a round of turns and a stage.  slices: column blocks per item in fp16 and in bf16 (one to four, stacked in bf16 at most two),
# the last one narrower; 3 in fp16 with 16 padded heads has stages of two blocks and four turns
@pytest.mark.parametrize("dtype", [F, B])
@pytest.mark.parametrize("heads,d,e,n,slices", [
    (16, 64, 384, 0, (1, 1)), (20, 64, 384, 0, (1, 1)), (48, 32, 384, 0, (1, 1)), (64, 32, 384, 0, (1, 1)), (72, 64, 256, 0, (1, 1)),
    (100, 32, 256, 0, (1, 1)), (128, 32, 256, 0, (1, 1)), (3, 64, 1152, 150, (4, 2)), (20, 32, 1152, 150, (4, 2)), (40, 32, 1152, 100, (2, 2)),
    (40, 32, 640, 150, (2, 2)), (9, 64, 1280, 59, (3, 2)), (20, 32, 1280, 59, (3, 2)),
])
def test_columns_of_the_weighted_sums(heads, d, e, n, slices, dtype):
    lens = [1, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 66, 80, 81, 96, 97, 127, 128, 129, 300]
    lens = lens + [1 + 37 * i % 90 for i in range(n)]
    assert slice_of_the_sums(heads, e, dtype, len(lens), torch.cuda.get_device_properties(0).multi_processor_count) == slices[dtype == B]
    w = workload(heads, d, e, dtype, lens, [True] * len(lens))
    rows = O.flat_rows(w.hidden_cache)   # what lies behind the sequences must not be seen
    for r, s in enumerate(lens):
        if s % 16:
            last = w.block_tables[r][-1]
            rows[last * 16 + s % 16: last * 16 + 16] = float("nan")
    check(w, f"{heads} heads, {len(lens)} requests")


# fold: one turn and several turns of 16 requests per epilogue warp, a second chunk of 128; it finds the requests by itself,
# those past 256 in the plan
@pytest.mark.parametrize("n,every", [(16, 1), (17, 1), (33, 2), (129, 1), (400, 3), (450, 1), (600, 2)])
@pytest.mark.parametrize("dtype", [F, B])
def test_fold_finds_its_requests(n, every, dtype):
    lens = [1 + 7 * i % 61 for i in range(n - 1)] + [450]
    check(workload(3, 128, 256, dtype, lens, [i % every == 0 for i in range(n)]), f"{n} requests, one in {every} hidden-cached")


def test_requests_without_tables_are_left_out():
    lens = [40, 17, 900, 1, 129, 64, 33, 200]
    w = workload(4, 128, 512, F, lens, [True, False] * 4, device="cuda")
    m, (wk, bk, wv, bv) = w.meta, w.kv_weights()

    def step(types, kv):
        out = torch.full_like(w.query, float("nan"))
        return A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, kv, kv, wk, bk, wv, bv,
                                   m.private_block_tables, m.seq_lens_tensor, types, w.scale, out=out)
    kv_all, kv_some = w.kv_cache.clone(), w.kv_cache.clone()
    want = step(m.cache_type, kv_all)
    types = m.cache_type.clone()
    types[2] = types[5] = NONE
    got = step(types, kv_some)
    assert torch.equal(got[[1, 3, 7]], want[[1, 3, 7]])   # K/V-cached
    # hidden-cached: another batch is cut into other pieces; both within check()'s bound of the oracle
    x, y = got[[0, 4, 6]].float(), want[[0, 4, 6]].float()
    rms = y.pow(2).mean(dim=1, keepdim=True).sqrt()
    assert ((x - y).abs() <= 2 * (2.0 ** -11 * y.abs() + 2.0 ** -14 * rms)).all()
    assert not got[[2, 5]].any()
    rows = kv_some.reshape(2, -1, 4 * 128)
    slot = int(m.private_block_tables[5][63 // 16]) * 16 + 63 % 16   # request 5 is K/V-cached: its new rows are not written
    assert torch.equal(rows[:, slot], w.kv_cache.reshape(2, -1, 4 * 128)[:, slot])


# new-token rows: a row shorter than a warp's 2 KB, one of several, K/V rows and layer-input rows of different lengths
@pytest.mark.parametrize("heads,d,e,dtype", [(1, 64, 128, F), (3, 128, 1152, B), (2, 64, 2560, F), (9, 128, 9216, B)])
def test_new_rows_are_written(heads, d, e, dtype):
    lens, hidden = [1, 16, 17, 40, 33, 128], [True, False, False, True, False, True]
    full = e % d == 0 and heads * d != e
    w = make_decode_workload(LayerShape("t", e // d if full else heads, d, e, dtype), lens, hidden, seed=7, device="cuda",
                             **({"tp_rank": 0, "tp_size": (e // d) // heads} if full else {}))
    m, (wk, bk, wv, bv) = w.meta, w.kv_weights()
    kv, hid = w.kv_cache.clone(), w.hidden_cache.clone()
    alias = w.hidden_cache.data_ptr() == w.kv_cache.data_ptr()
    A.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache, w.hidden_cache, wk, bk, wv, bv,
                        m.private_block_tables, m.seq_lens_tensor, m.cache_type, w.scale)
    width = w.new_key.reshape(len(lens), -1).shape[1]
    if alias:
        hid = kv
    flat, planes = hid.view(-1, e), kv.view(2, -1, width)
    for r, (s, u) in enumerate(zip(lens, hidden)):
        slot = int(m.private_block_tables[r][(s - 1) // 16]) * 16 + (s - 1) % 16
        if u:
            flat[slot] = w.hidden_states[r]
        else:
            planes[0, slot], planes[1, slot] = w.new_key.reshape(len(lens), -1)[r], w.new_value.reshape(len(lens), -1)[r]
    assert torch.equal(w.hidden_cache, hid) and torch.equal(w.kv_cache, kv)


# K/V path: units shared by four warps (CUDA cores, few of them) or not; units from a warp's place, from the counter, and from
# the counter without a look at the plan's total (long block tables); tolerances of test_gpu_attention.py
@pytest.mark.parametrize("heads,d,dtype,lens", [
    (3, 64, torch.float32, [1, 31, 32, 33, 127, 128, 129, 300]), (12, 64, torch.float32, [300] * 20 + [7] * 20),
    (2, 128, torch.float32, [96, 97, 513]), (2, 256, F, [96, 97, 513]), (2, 32, B, [33, 640]),
    (5, 64, F, [1, 90, 128, 129]), (40, 128, F, [130] * 40), (40, 64, B, [40] * 60 + [1300]), (40, 128, F, [40] * 60 + [1300]),
])
def test_kv_units(heads, d, dtype, lens):
    w = make_decode_workload(LayerShape("t", heads, d, heads * d, dtype), lens, [False] * len(lens), seed=len(lens))
    ref = O.paged_decode_attention(w.query, w.kv_cache[0], w.kv_cache[1], w.meta.block_tables, w.meta.seq_lens_tensor, w.scale)
    g = w.to("cuda")
    args = (g.query, g.kv_cache[0], g.kv_cache[1], g.meta.block_tables, g.meta.seq_lens_tensor, g.scale)
    out = A.paged_decode_attention(*args)
    assert torch.equal(out, A.paged_decode_attention(*args))
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert_close(out, ref, f"{len(lens)} requests of {heads} heads", tol, tol)


# scores of -infinity: such tokens have no weight, wherever the work of a request is cut (fp32: four warps per K/V unit, a quarter
# of its 128 tokens each; chunks of 32 cached rows); tolerances of test_gpu_attention.py
@pytest.mark.parametrize("first,last", [(32, 64), (0, 32), (96, 128), (0, 128), (40, 300)])
def test_scores_of_minus_infinity(first, last):
    w = make_decode_workload(LayerShape("t", 3, 64, 192, torch.float32), [300], [False], seed=4)
    m, q = w.meta, w.query.view(1, 3, 64)
    q[..., 0] = 1.0
    if last == 300:   # all of them
        first = 0
    slots = torch.tensor([int(m.block_tables[0][t // 16]) * 16 + t % 16 for t in range(300)])
    key, value = (w.kv_cache[i].reshape(-1, 3, 64)[slots].double() for i in (0, 1))
    key[first:last, :, 0] = float("-inf")
    w.kv_cache[0].view(-1, 3, 64)[slots] = key.float()
    p = torch.softmax(torch.einsum("hd,thd->ht", q[0].double(), key) * w.scale, dim=1)
    ref = torch.einsum("ht,thd->hd", p, value).reshape(1, 192)
    g = w.to("cuda")
    out = A.paged_decode_attention(g.query, g.kv_cache[0], g.kv_cache[1], g.meta.block_tables, g.meta.seq_lens_tensor, g.scale)
    if last == 300:
        assert torch.isnan(out).all() and torch.isnan(ref).all()
    else:
        assert_close(out, ref, f"tokens {first} to {last}", 1e-4, 1e-4)


@pytest.mark.parametrize("first,last", [(32, 64), (0, 32), (96, 128), (0, 128), (0, 300)])
def test_scores_of_minus_infinity_of_cached_rows(first, last):
    e = 64
    w = make_decode_workload(LayerShape("t", 1, 64, e, torch.float32), [300], [True], seed=4)
    m, (wk, bk, wv, bv) = w.meta, w.kv_weights()
    w.query.mul_(100.0)
    slots = torch.tensor([int(m.private_block_tables[0][t // 16]) * 16 + t % 16 for t in range(300)])
    x = w.hidden_cache.reshape(-1, e)[slots]
    qt = wk.double().t() @ w.query[0].double() * w.scale   # scores are x . qt
    col = int(qt.abs().argmax())
    x[first:last] = 0.0
    x[first:last, col] = -3e38 * float(qt[col].sign())
    w.hidden_cache.view(-1, e)[slots] = x
    x = x.double()
    assert float(qt[col].abs()) > 1.2   # the product is out of fp32's range
    s = x @ qt
    s[first:last] = float("-inf")
    p = torch.softmax(s, dim=0)
    ref = (p @ torch.where(p[:, None] > 0, x, torch.zeros_like(x))) @ wv.double().t() + (0 if bv is None else bv.double())
    g = w.to("cuda")
    wk, bk, wv, bv = g.kv_weights()
    out = A.hybrid_decode_attention(g.query, g.kv_cache, g.hidden_cache, wk, bk, wv, bv, g.meta.private_block_tables,
                                    g.meta.seq_lens_tensor, g.meta.cache_type, g.scale)
    if last == 300:   # all of them
        assert torch.isnan(out).all() and torch.isnan(ref).all()
    else:
        assert_close(out, ref[None], f"tokens {first} to {last}", 1e-4, 1e-4)
