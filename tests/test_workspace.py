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
