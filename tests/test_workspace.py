"""The scratch handed out per device: what a call gets depends on what it asks for, not on the calls before it (no GPU)."""
import torch

from apt_serve_b200 import _native as N
from apt_serve_b200 import attention as A

CPU = torch.device("cpu")
SHAPE = (64, 40, 16, 40, 128)


def test_scratch_size_does_not_depend_on_earlier_calls(monkeypatch):
    """A layer-step re-projects or attends directly by the size of its scratch: an attention-sized one must not have
    grown with someone else's layer-step."""
    monkeypatch.setattr(A, "_workspaces", {})
    plain = N.lib().aps_attention_workspace_bytes(*SHAPE)
    step = N.lib().aps_decode_layer_step_workspace_bytes(*SHAPE, 5120, N.DTYPE_ENUM[torch.float16])
    assert 1 << 20 < plain < step
    assert A.attention_workspace(CPU, *SHAPE).numel() == plain
    big = A.layer_step_workspace(CPU, *SHAPE, 5120, torch.float16)
    assert big.numel() == step
    again = A.attention_workspace(CPU, *SHAPE)
    assert again.numel() == plain and again.data_ptr() == big.data_ptr()
    assert A.attention_workspace(CPU, 1, 1, 16, 1, 32).numel() == 1 << 20
    assert A.layer_step_workspace(CPU, *SHAPE, 5120, torch.float16).data_ptr() == big.data_ptr()


def test_scratch_of_a_few_requests_is_small():
    """The projected outputs and the partial scores are sized for the batch, not for a full group of requests."""
    size = lambda b, blocks, t: N.lib().aps_decode_layer_step_workspace_bytes(b, blocks, 16, 40, 128, 5120, N.DTYPE_ENUM[t])
    one = size(1, 39, torch.float16)
    # 16 requests' folded queries in two terms, seven ranges of projected outputs, partial scores of 3 tiles and 51 pieces,
    # 39 blocks of weights, the plan and some rounding
    assert one < 16 * (2 * 40 * 5120 * 2 + 7 * 5120 * 4) + (3 + 51) * 40 * 1024 + 39 * 2 * 48 * 32 + (1 << 18)
    assert size(8, 39, torch.float16) < 2 * one and size(256, 128, torch.float16) > 10 * one
    small = N.lib().aps_decode_layer_step_workspace_bytes(1, 39, 16, 12, 64, 768, N.DTYPE_ENUM[torch.float32])
    assert small < 4 << 20
