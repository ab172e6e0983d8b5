"""The work that a serving engine has this package do, as timed cases.

A case names one call of the hybrid-cache path with its sizes; ``prepare`` makes what the engine
holds when it makes the call (a layer's caches, its weights, the step's inputs, the index tensors of
the batch), ``run`` makes the call.  Kinds of call:

  step      ``attention.decode_layer_step``: one decode layer between the projections and o_proj
  layer     ``layers.OPTAttention`` on a decode batch, from the model runner's unchanged metadata
            (Q / K / V projections, the step, o_proj)
  backend   ``FlashAttentionImpl.forward`` on a decode batch without hidden-cached requests
            (cache write of the new tokens + paged attention)
  prompt    ``layers.OPTAttention`` on packed prompts, some of them hidden-designated
  store     the cache writes of a prefill batch and its copy-on-write block copies
            (``ops.prefill_cache_write``, ``FlashAttentionBackend.copy_blocks``)
  copy      copy-on-write block copies over the layers of a model
  literal   ``layers.OPTAttention(fused=False)``: the reference's own op sequence, op by op
  indices   ``device_metadata.expand_decode_metadata``: host block tables to device index tensors

Sequence lengths and cache types belong to the case (drawn from its ``mix`` number), values to the
seed: the same case with another seed is the same work on other numbers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from apt_serve_b200 import attention, device_metadata, ops
from apt_serve_b200.layers import OPTAttention
from apt_serve_b200.metadata import BlockPool, blocks_needed
from apt_serve_b200.workloads import LayerShape, make_decode_workload

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
# model -> heads, head size, hidden size
MODELS = {"opt-125m": (12, 64, 768), "opt-1.3b": (32, 64, 2048), "opt-13b": (40, 128, 5120),
          "opt-66b": (72, 128, 9216)}
BLOCK = 16


def _case(kind, model, dtype, batch, median, hidden, mix, tp=1, layers=1):
    return {"kind": kind, "model": model, "dtype": dtype, "batch": batch, "median": median,
            "hidden": hidden, "mix": mix, "tp": tp, "layers": layers}


def listed():
    def named(name, *a, **kw):
        return dict(_case(*a, **kw), name=name)
    return [
        # a full OPT-13B serving batch, half of the requests hidden-cached: the headline workload
        named("step 13b b256", "step", "opt-13b", "fp16", 256, 700, 0.5, 1002),
        # one rank of eight of an OPT-66B layer: few heads, wide rows, a hidden cache of its own
        named("step 66b tp8 b128", "step", "opt-66b", "bf16", 128, 900, 0.4, 1004, tp=8),
        # a small model's batch, 64-element heads, most of the requests hidden-cached
        named("step 1.3b b48", "step", "opt-1.3b", "bf16", 48, 450, 0.7, 21),
        # the CPU-sized configuration in fp32
        named("step 125m fp32 b8", "step", "opt-125m", "fp32", 8, 230, 0.5, 1001),
        # a server with a single user: latency of one hidden-cached request
        named("step 13b b1", "step", "opt-13b", "fp16", 1, 611, 1.0, 5),
        # a whole attention layer at long contexts, all hidden-cached (cache pressure)
        named("layer 13b b24 long", "layer", "opt-13b", "fp16", 24, 1800, 1.0, 1005),
        # plain K/V serving (no memory pressure): what every step is until the scheduler changes types
        named("backend 13b b128", "backend", "opt-13b", "fp16", 128, 700, 0.0, 33),
        # a handful of short chats on a small model: launches and host work
        named("backend 1.3b b5", "backend", "opt-1.3b", "fp16", 5, 90, 0.0, 34),
        # new prompts, half of them hidden-designated
        named("prompt 13b b6", "prompt", "opt-13b", "fp16", 6, 500, 0.5, 41),
        # cache writes of 32 prompts and the copies of 5 % of the blocks
        named("store 13b b32", "store", "opt-13b", "fp16", 32, 900, 0.5, 1003),
        # the reference's own op sequence for an unmodified caller
        named("literal 13b b12", "literal", "opt-13b", "fp16", 12, 400, 0.5, 51),
        # index tensors of a decode batch from host block tables
        named("indices b256", "indices", "opt-13b", "fp16", 256, 700, 0.5, 1002),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["step"] * 6 + ["layer", "layer", "backend", "backend", "prompt", "store", "copy",
                                      "literal", "indices"])
    model = rng.choice(["opt-125m", "opt-1.3b", "opt-13b", "opt-13b", "opt-66b"])
    dtype = rng.choice(["fp16", "bf16"])
    tp = rng.choice([1, 2, 8]) if kind == "step" and model in ("opt-13b", "opt-66b") else 1
    if model == "opt-66b" and tp == 1:
        model = "opt-13b"
    if kind == "step" and model == "opt-125m" and rng.random() < 0.5:
        dtype = "fp32"
    if kind in ("layer", "prompt", "literal", "store", "backend") and model == "opt-66b":
        model = "opt-13b"
    most = {"step": 256, "layer": 128, "backend": 256, "prompt": 8, "store": 32, "copy": 96, "literal": 12,
            "indices": 256}[kind]
    c = _case(kind, model, dtype, log_int(1, most), log_int(40, 1500), 0.0 if kind == "backend" else
              rng.choice([0.2, 0.35, 0.5, 0.75, 1.0]), rng.randrange(10 ** 6), tp=tp,
              layers=log_int(2, 24) if kind == "copy" else 1)
    if kind == "literal" and c["hidden"] == 1.0:
        c["hidden"] = 0.5
    ceiling = max(work(x)["bytes"] for x in listed())
    while c["batch"] > 1 and work(c)["bytes"] > ceiling:
        c["batch"] = max(1, c["batch"] * 3 // 4)
    return c


# ---- sizes ------------------------------------------------------------------------------
def _lengths(case):
    """Sequence lengths (lognormal around the median, 1..2048) and cache types of the batch."""
    rng = np.random.default_rng(case["mix"])
    n = case["batch"]
    lens = np.clip(np.rint(rng.lognormal(math.log(case["median"]), 0.6, size=n)), 1, 2048).astype(int)
    if n == 1:
        lens[0] = min(2048, case["median"])
    k = int(math.ceil(n * case["hidden"]))
    hid = np.zeros(n, dtype=bool)
    hid[rng.permutation(n)[:k]] = True
    if case["kind"] == "literal" and n > 1:
        hid[0], hid[1] = True, False   # both kinds, as in a batch that takes this path
    return [int(x) for x in lens], [bool(x) for x in hid]


def _shape(case):
    h, d, e = MODELS[case["model"]]
    return LayerShape(case["model"], h, d, e, DTYPES[case["dtype"]], BLOCK)


def work(case):
    """Bytes and operations of one pass, each input read and each output written once."""
    lens, hid = _lengths(case)
    h_all, d, e = MODELS[case["model"]]
    h = h_all // case["tp"]
    hd, es, n = h * d, 4 if case["dtype"] == "fp32" else 2, case["batch"]
    t_h = sum(s for s, u in zip(lens, hid) if u)
    t_kv = sum(s for s, u in zip(lens, hid) if not u)
    n_h = sum(hid)
    n_kv = n - n_h
    kind = case["kind"]
    if kind in ("step", "backend", "layer"):
        # cached rows once, the K and V weights once when a request is hidden-cached, query and
        # output, the new token's rows read and written
        by = (t_kv * 2 * hd + t_h * e + (2 * hd * e if n_h else 0) + 2 * n * hd
              + 2 * (n_kv * 2 * hd + n_h * e)) * es
        # K/V attention; hidden rows: scores and weighted sums against the rows themselves plus the
        # two small contractions with W_k and W_v per request
        fl = 4.0 * t_kv * hd + 4.0 * t_h * h * e + 4.0 * n_h * hd * e
        if kind == "layer":
            by += (3 * hd * e + hd * e + 2 * n * e) * es - (2 * hd * e * es if n_h else 0)
            fl += 2.0 * n * e * hd * 2 + (2.0 * n_kv * e * 2 * hd)
        return {"bytes": float(by), "flops": fl}
    if kind == "prompt":
        t = t_h + t_kv
        by = (4 * hd * e + 2 * t * e + 3 * t * hd + t_kv * 2 * hd + t_h * e) * es
        return {"bytes": float(by), "flops": 2.0 * t * e * 4 * hd + 2.0 * hd * sum(s * s for s in lens)}
    if kind == "store":
        return {"bytes": float(2 * es * (t_kv * 2 * hd + t_h * e) + 2 * _n_copies(case) * 2 * BLOCK * hd * es), "flops": 0.0}
    if kind == "copy":
        return {"bytes": float(2 * case["layers"] * n * 2 * BLOCK * hd * es), "flops": 0.0}
    if kind == "literal":
        # gathered rows, their projection, both scatters, attention over the shared cache
        tot = t_h + n_kv
        by = (tot * e * 2 + 2 * hd * e * 2 + tot * 2 * hd * 2 + t_h * 2 * hd + 4 * n * hd) * es
        return {"bytes": float(by), "flops": 2.0 * tot * e * 2 * hd + 2.0 * n * e * 2 * hd}
    # indices: two block tables in, int64 index tensors out
    blocks = sum(-(-s // BLOCK) for s in lens)
    return {"bytes": float(8 * (t_h + n_kv) + 8 * 2 * t_h + 8 * (t_h + n_kv - n) + 8 * 2 * n + 4 * 2 * blocks),
            "flops": 0.0}


def _n_copies(case):
    lens, hid = _lengths(case)
    return max(1, blocks_needed(lens, hid, BLOCK) // 20)


def tolerance(case):
    if case["kind"] in ("store", "copy", "indices"):
        return "exact"
    # four times the distance of the path from itself in 64 bits: 2.1e-4 - 2.6e-4 in fp16 and 1.7e-3 - 1.8e-3
    # in bf16 (of which the rounding of the outputs alone is 2.1e-4 and 1.7e-3), 5e-7 in fp32 at short contexts
    # (twice that allowed for, the sums grow with the context)
    return {"fp16": {"rel": 1e-3}, "bf16": {"rel": 8e-3}, "fp32": {"rel": 4e-6}}[case["dtype"]]


# ---- inputs ------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    lens, hid = _lengths(case)
    shape = _shape(case)
    if kind in ("step", "layer", "backend", "literal"):
        w = make_decode_workload(shape, lens, hid, seed, "cuda", tp_rank=case["tp"] // 2, tp_size=case["tp"],
                                 with_shared_cache=kind == "literal")
        state = {"case": case, "w": w}
        if kind in ("layer", "literal"):
            state["layer"] = OPTAttention(shape.hidden, shape.num_heads, w.qkv_weight, w.qkv_bias, w.o_weight,
                                          w.o_bias, fused=kind == "layer")
            state["meta"] = attention.FlashAttentionMetadata.from_decode(w.meta)
        if kind == "backend":
            state["impl"] = attention.FlashAttentionImpl(shape.num_heads, shape.head_dim, w.scale,
                                                         shape.num_heads, None, None, "auto")
            state["meta"] = attention.FlashAttentionMetadata.from_decode(w.meta)
        return state
    if kind in ("prompt", "store"):
        w = make_decode_workload(shape, [1], [False], seed, "cuda", prefill=(lens, hid))
        p = w.prefill
        state = {"case": case, "w": w, "p": p}
        if kind == "prompt":
            state["layer"] = OPTAttention(shape.hidden, shape.num_heads, w.qkv_weight, w.qkv_bias, w.o_weight,
                                          w.o_bias)
            state["meta"] = attention.FlashAttentionMetadata.from_prefill(p.meta)
        else:
            # copy-on-write: blocks of the decode pool into fresh blocks of a second layer's cache
            n = _n_copies(case)
            g = torch.Generator(device="cuda").manual_seed(seed + 7)
            state["other"] = torch.randn(2, 2 * n, BLOCK, shape.num_heads, shape.head_dim, generator=g,
                                         device="cuda", dtype=shape.dtype)
            ids = np.random.default_rng(case["mix"]).permutation(2 * n)
            state["pairs"] = torch.from_numpy(np.stack([ids[:n], ids[n:]], axis=1).astype(np.int64)).cuda()
        return state
    if kind == "copy":
        n = case["batch"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        caches = [torch.randn(2, 2 * n + 3, BLOCK, shape.num_heads, shape.head_dim, generator=g, device="cuda",
                              dtype=shape.dtype) for _ in range(case["layers"])]
        ids = np.random.default_rng(case["mix"]).permutation(2 * n + 3)
        pairs = torch.from_numpy(np.stack([ids[:n], ids[n:2 * n]], axis=1).astype(np.int64)).cuda()
        return {"case": case, "caches": caches, "pairs": pairs}
    # indices: what the engine's scheduler hands over, lists on the host
    pool = BlockPool(blocks_needed(lens, hid, BLOCK) + 8, np.random.default_rng(seed))
    tables = [pool.table_for(s, BLOCK, u) for s, u in zip(lens, hid)]
    shared = [pool.shared_table_for(s, BLOCK) if u else [] for s, u in zip(lens, hid)]
    return {"case": case, "lens": lens, "hid": hid, "tables": tables, "shared": shared}


# ---- the calls ---------------------------------------------------------------------------
def run(state):
    kind = state["case"]["kind"]
    if kind == "step":
        w, m = state["w"], state["w"].meta
        wk, bk, wv, bv = w.kv_weights()
        out = attention.decode_layer_step(w.query, w.hidden_states, w.new_key, w.new_value, w.kv_cache,
                                          w.hidden_cache, wk, bk, wv, bv, m.private_block_tables,
                                          m.seq_lens_tensor, m.cache_type, w.scale)
        return [out, w.kv_cache] + ([] if w.hidden_cache is w.kv_cache else [w.hidden_cache])
    if kind == "layer":
        w = state["w"]
        return [state["layer"](w.hidden_states, w.kv_cache, None, state["meta"]), w.kv_cache]
    if kind == "literal":
        w = state["w"]
        return [state["layer"](w.hidden_states, w.kv_cache, w.shared_cache, state["meta"]), w.kv_cache,
                w.shared_cache]
    if kind == "backend":
        w = state["w"]
        return [state["impl"].forward(w.query, w.new_key, w.new_value, w.kv_cache, None, state["meta"]), w.kv_cache]
    if kind == "prompt":
        w = state["w"]
        return [state["layer"](state["p"].hidden_states, w.kv_cache, None, state["meta"]), w.kv_cache]
    if kind == "store":
        w, p = state["w"], state["p"]
        ops.prefill_cache_write(p.key, p.value, p.hidden_states, w.kv_cache, w.hidden_cache, p.meta.slot_mapping,
                                p.meta.kv_cache_use_tot, p.meta.hidden_cache_use_input)
        attention.FlashAttentionBackend.copy_blocks([state["other"]], state["pairs"])
        return [w.kv_cache, state["other"]]
    if kind == "copy":
        attention.FlashAttentionBackend.copy_blocks(state["caches"], state["pairs"])
        return state["caches"]
    m = device_metadata.expand_decode_metadata(state["lens"], state["hid"], state["tables"], state["shared"],
                                               BLOCK, "cuda")
    return [m.slot_mapping, m.slot_mapping_shared, m.hidden_cache_use_tot, m.kv_cache_use_tot, m.hidden_holder_upd,
            m.hidden_holder_pull, m.hidden_cache_store_tot, m.hidden_cache_use_input, m.block_tables,
            m.private_block_tables, m.seq_lens_tensor, m.cache_type]
