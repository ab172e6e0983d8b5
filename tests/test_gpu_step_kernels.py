"""Branches of the layer-step's kernels that depend on how much work a batch is (csrc/hidden_attention.cu, csrc/paged_attention.cu),
against the oracle with the tolerances of test_gpu_folded.py."""
import pytest
import torch

from apt_serve_b200.workloads import LayerShape, make_decode_workload

from test_gpu_folded import check

pytestmark = pytest.mark.gpu
F, B = torch.float16, torch.bfloat16


def workload(heads, d, e, dtype, lens, hidden, device="cpu"):
    return make_decode_workload(LayerShape("t", heads, d, e, dtype), lens, hidden, seed=len(lens) + heads, device=device)


# softmax: single heads (few units) and pairs of heads, the last one alone; more tokens than a CTA's registers hold (2048)
@pytest.mark.parametrize("heads,dtype,lens", [
    (5, F, (4200, 3, 2049)), (5, B, (4200, 3, 2049)),
    (33, F, (2049, 17, 600, 1, 255, 256, 257, 16, 90, 4100, 31, 32)), (48, B, (2049, 17, 600, 1, 255, 256, 257, 16)),
])
def test_softmax_units(heads, dtype, lens):
    check(workload(heads, 64, 128, dtype, list(lens), [True] * len(lens)), f"{heads} heads, {len(lens)} requests")
