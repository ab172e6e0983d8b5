"""FlashAttentionImpl.forward on a batch of decode tokens without hidden-cached requests: the short way to the two native
calls gives what the general one gives, and takes no argument that the general one refuses."""
import pytest
import torch

from apt_serve_b200 import attention as A
from apt_serve_b200.workloads import LayerShape, make_decode_workload

pytestmark = pytest.mark.gpu


def setup(dtype=torch.float16, heads=4, d=64, lens=(5, 40, 129, 16, 1)):
    w = make_decode_workload(LayerShape("t", heads, d, heads * d, dtype), list(lens), [False] * len(lens), seed=9, device="cuda")
    impl = A.FlashAttentionImpl(heads, d, w.scale, heads, None, None, "auto")
    return w, impl, A.FlashAttentionMetadata.from_decode(w.meta)


def forward(impl, w, meta, q, k, v, general, monkeypatch):
    cache = w.kv_cache.clone()
    with monkeypatch.context() as m:
        if general:
            m.setattr(impl, "_plain_decode", lambda *a: None)
        return impl.forward(q, k, v, cache, None, meta), cache


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strided", ["no", "columns of one projection", "rows of no multiple of 16 bytes", "a slot left out"])
def test_equals_the_general_path(monkeypatch, dtype, strided):
    w, impl, meta = setup(dtype)
    q, k, v = w.query, w.new_key, w.new_value
    n = q.shape[0]
    q, k, v = q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)
    if strided == "columns of one projection":
        q, k, v = torch.cat([q, k, v], dim=1).chunk(3, dim=1)
    elif strided == "rows of no multiple of 16 bytes":
        k, v = (torch.nn.functional.pad(t, (0, 1))[:, :-1] for t in (k, v))
    elif strided == "a slot left out":
        meta.slot_mapping[2] = -1
    assert impl._plain_decode(q, k, v, w.kv_cache.clone(), meta) is not None
    short, general = (forward(impl, w, meta, q, k, v, g, monkeypatch) for g in (False, True))
    assert torch.equal(short[0], general[0]) and torch.equal(short[1], general[1])
    assert short[0].shape == general[0].shape and short[0].stride() == general[0].stride()


@pytest.mark.parametrize("pitch", [4 * 64, 4 * 64 + 1, 1, 0])
def test_a_single_row_of_any_stride(monkeypatch, pitch):
    w, impl, meta = setup(lens=(40,))
    q, k, v = (t.reshape(-1).as_strided((1, 4 * 64), (pitch, 1)) for t in (w.query, w.new_key, w.new_value))
    assert impl._plain_decode(q, k, v, w.kv_cache.clone(), meta) is not None
    short, general = (forward(impl, w, meta, q, k, v, g, monkeypatch) for g in (False, True))
    assert torch.equal(short[0], general[0]) and torch.equal(short[1], general[1])
    assert short[0].stride() == general[0].stride()


@pytest.mark.parametrize("what", ["slots", "dtype", "rows", "lengths"])
def test_refuses_what_the_general_path_refuses(monkeypatch, what):
    w, impl, meta = setup()
    q, k, v = (t.reshape(t.shape[0], -1) for t in (w.query, w.new_key, w.new_value))
    if what == "slots":
        meta.slot_mapping = meta.slot_mapping.int()
    elif what == "dtype":
        k = k.float()
    elif what == "rows":
        k = k[:-1]
    else:
        meta.seq_lens_tensor = meta.seq_lens_tensor.long()
    errors = []
    for general in (False, True):
        with pytest.raises((RuntimeError, AssertionError, ValueError)) as e:
            forward(impl, w, meta, q, k, v, general, monkeypatch)
        errors.append(e.type)
    assert errors[0] is errors[1]
