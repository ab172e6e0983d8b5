"""aps_prefill_attention against causal attention of every prompt in fp64.

Tolerance: the weights and the output are rounded to the inputs' type (u: half a unit of the last place, relative), the sums
are fp32: |x - y| <= u |y| + u sum_k p_k |v_k|, half of the latter again for the products' and exponentials' own rounding.  fp16
below its normal range: 2^-25 for the output and for every weight, times the |v_k| of the keys the row sees."""
import pytest
import torch

from apt_serve_b200 import _native as N
from apt_serve_b200 import attention as A

pytestmark = pytest.mark.gpu
F, B = torch.float16, torch.bfloat16
U = {F: 2.0 ** -11, B: 2.0 ** -8}


def prompts(lens, heads, d, dtype, seed=0, spread=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = torch.randn(sum(lens), 3 * heads * d, generator=g, device="cuda").mul_(spread).to(dtype)
    q, k, v = (t.view(-1, heads, d) for t in qkv.chunk(3, dim=1))   # row strides of the projection
    bounds = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    return q, k, v, bounds


def reference(q, k, v, lens, scale):
    out, size, least = (torch.empty(q.shape, dtype=torch.double, device="cuda") for _ in range(3))
    a = 0
    for n in lens:
        s = torch.einsum("qhd,khd->hqk", q[a:a + n].double(), k[a:a + n].double()) * scale
        p = torch.softmax(s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), float("-inf")), dim=2)
        out[a:a + n] = torch.einsum("hqk,khd->qhd", p, v[a:a + n].double())
        size[a:a + n] = torch.einsum("hqk,khd->qhd", p, v[a:a + n].double().abs())
        least[a:a + n] = 2.0 ** -25 * (1 + v[a:a + n].double().abs().cumsum(0)) if q.dtype == F else 0.0
        a += n
    return out, size, least


def attend(q, k, v, bounds, lens, scale):
    assert A._prefill_supported(q, k, v, bounds, scale), "this size does not take the kernel under test"
    return A._varlen_prefill_attention(q, k, v, bounds, max(lens), scale)


@pytest.mark.parametrize("dtype", [F, B])
@pytest.mark.parametrize("heads,d,lens,spread", [
    (2, 128, [1, 127, 128, 129, 255, 256, 257, 2, 640], 1.0), (3, 64, [1, 127, 128, 129, 255, 256, 257, 2, 640], 1.0),
    (1, 128, [2048], 1.0), (5, 64, [700, 33], 3.0), (2, 128, [300] * 20, 4.0),
])
def test_against_fp64(heads, d, lens, spread, dtype):
    scale = d ** -0.5
    q, k, v, bounds = prompts(lens, heads, d, dtype, spread=spread)
    out = attend(q, k, v, bounds, lens, scale)
    assert torch.equal(out, attend(q, k, v, bounds, lens, scale))
    ref, size, least = reference(q, k, v, lens, scale)
    bad = ~((out.double() - ref).abs() <= U[dtype] * (ref.abs() + 1.5 * size) + least)
    assert not bad.any(), (int(bad.sum()), float(((out.double() - ref).abs() / size).max() / U[dtype]))


def test_growing_scores_move_the_maximum():
    """Scores that grow by more than 2^8 per tile: what has been accumulated is rescaled."""
    lens, d = [900], 128
    q, k, v, bounds = prompts(lens, 2, d, F, seed=1)
    k *= torch.linspace(0.0, 4.0, 900, device="cuda").view(-1, 1, 1).half()
    q.copy_(k * 0.5 + q * 0.1)
    out = attend(q, k, v, bounds, lens, d ** -0.5)
    ref, size, least = reference(q, k, v, lens, d ** -0.5)
    assert ((out.double() - ref).abs() <= U[F] * (ref.abs() + 1.5 * size) + least).all()


def test_prompts_do_not_see_each_other():
    lens = [130, 40, 7]
    q, k, v, bounds = prompts(lens, 2, 64, F, seed=2)
    want = attend(q, k, v, bounds, lens, 0.125)
    k[170:], v[170:] = float("nan"), float("inf")
    got = attend(q, k, v, bounds, lens, 0.125)
    assert torch.equal(got[:170], want[:170]) and torch.isfinite(got[:170]).all()


def test_what_it_does_not_take_goes_to_the_library():
    q, k, v, bounds = prompts([40, 9], 2, 32, F, seed=3)
    assert not A._prefill_supported(q, k, v, bounds, 0.2)
    out = A._varlen_prefill_attention(q, k, v, bounds, 40, 0.2)
    ref, size, least = reference(q, k, v, [40, 9], 0.2)
    assert ((out.double() - ref).abs() <= U[F] * (ref.abs() + 4 * size) + least).all()


def test_prompts_of_no_tokens():
    lens = [0, 40, 0, 0, 130, 0]
    q, k, v, bounds = prompts(lens, 2, 64, F, seed=4)
    want = attend(q, k, v, torch.tensor([0, 40, 170], device="cuda", dtype=torch.int32), [40, 130], 0.125)
    assert torch.equal(attend(q, k, v, bounds, lens, 0.125), want)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("which", ["query", "key", "value"])
@pytest.mark.parametrize("where", [3, 130, 255, 399])
def test_nan_inside_a_prompt(which, where, d):
    """A row is not finite where it attends to the bad row, and at most in the bad row's 128 query rows before it (weights of
    zero there, times the bad value); the rows of other prompts and of earlier query tiles are as they were."""
    lens = [400, 70]
    q, k, v, bounds = prompts(lens, 2, d, B, seed=5)
    want = attend(q, k, v, bounds, lens, d ** -0.5)
    {"query": q, "key": k, "value": v}[which][where, :, 5] = float("nan")
    got = attend(q, k, v, bounds, lens, d ** -0.5)
    same = [t for t in range(470) if t < where // 128 * 128 or t >= 400 or (which == "query" and t != where)]
    assert torch.equal(got[same], want[same])
    bad = got[where if which == "query" else slice(where, 400)]
    assert torch.isnan(bad[..., 5] if which == "value" else bad).all()


def test_gradients_flow_where_they_are_wanted():
    lens = [70, 33]
    q, k, v, bounds = prompts(lens, 2, 64, B, seed=6)
    plain = attend(q, k, v, bounds, lens, 0.125)
    assert not plain.requires_grad
    q, k, v = (t.detach().clone().requires_grad_() for t in (q, k, v))
    out = A._varlen_prefill_attention(q, k, v, bounds, max(lens), 0.125)
    g = torch.randn(out.shape, generator=torch.Generator(device="cuda").manual_seed(7), device="cuda").to(B)
    got = torch.autograd.grad(out, (q, k, v), g)
    qd, kd, vd = (t.detach().double().requires_grad_() for t in (q, k, v))
    rows = []
    for a, n in ((0, 70), (70, 33)):
        s = torch.einsum("qhd,khd->hqk", qd[a:a + n], kd[a:a + n]) * 0.125
        p = torch.softmax(s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), float("-inf")), dim=2)
        rows.append(torch.einsum("hqk,khd->qhd", p, vd[a:a + n]))
    want = torch.autograd.grad(torch.cat(rows), (qd, kd, vd), g.double())
    for x, y in zip(got, want):   # sums of products of factors rounded to bf16: a few units of 2^-8 in the 2-norm
        assert float((x.double() - y).norm() / y.norm()) < 4 * U[B]
    with torch.no_grad():
        assert torch.equal(A._varlen_prefill_attention(q, k, v, bounds, max(lens), 0.125), plain)


@pytest.mark.parametrize("scale", [0.0, -0.125, 1e-40, float("inf"), float("nan")])
def test_scales_it_is_wrong_for_go_to_the_library(scale):
    q, k, v, bounds = prompts([40, 9], 2, 64, F, seed=8)
    assert A._prefill_supported(q, k, v, bounds, 0.125) and not A._prefill_supported(q, k, v, bounds, scale)
    assert A._varlen_prefill_attention(q, k, v, bounds, 40, scale).shape == q.shape


def test_a_wait_that_runs_out_is_reported():
    A.raise_on_device_status()
    N.check(N.lib().aps_selftest_prefill_wait(200000, N.current_stream(torch.device("cuda", 0))))
    with pytest.raises(RuntimeError, match="status 3"):
        A.raise_on_device_status()
    A.raise_on_device_status()   # said once
    q, k, v, bounds = prompts([40], 2, 64, F)
    attend(q, k, v, bounds, [40], 0.125)
    A.raise_on_device_status()
