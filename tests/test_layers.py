"""The output projection on the CPU: which biases it takes, with and without a reduction."""
import pytest
import torch
import torch.nn.functional as F

from apt_serve_b200.layers import RowParallelLinear


@pytest.mark.parametrize("w_type,b_type,shape", [
    (torch.bfloat16, torch.bfloat16, (24,)), (torch.float32, torch.float32, (24,)), (torch.float16, torch.float32, (24,)),
    (torch.bfloat16, torch.float32, (24,)), (torch.float32, torch.bfloat16, (24,)), (torch.bfloat16, torch.bfloat16, (1, 24)),
    (torch.float32, torch.float32, (1,)), (torch.float32, torch.float32, ()), (torch.float32, torch.float32, (5, 24)),
])
def test_bias_of_any_type_that_can_be_added(w_type, b_type, shape):
    torch.manual_seed(0)
    w, x, b = torch.randn(24, 16, dtype=w_type), torch.randn(5, 16, dtype=w_type), torch.randn(shape, dtype=b_type)
    out, extra = RowParallelLinear(w, b)(x)
    want = F.linear(x, w) + b
    assert extra is None and out.dtype == want.dtype and out.shape == want.shape
    exact = x.double() @ w.double().T + b.double()
    eps = max(torch.finfo(t).eps for t in (w_type, b_type))   # two roundings of the sum at most
    assert ((out.double() - exact).abs() <= eps * (exact.abs() + (x.double() @ w.double().T).abs()) + 1e-6).all()


def test_no_bias():
    w, x = torch.randn(24, 16), torch.randn(5, 16)
    assert torch.equal(RowParallelLinear(w, None)(x)[0], F.linear(x, w))
