"""The work that a user of this package has it do, as cases that can be timed and compared.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

* ``step``     one decoding step of ``VQCodeCache.decode_step``: the token's K and V rows are encoded and appended, the
               query attends over the stored codes (``rotary``: the cache holds pre-rotary keys, as the Mistral adapter does);
* ``host``     the same step driven from pinned host buffers (``VQCodeCache.decode_step_host``);
* ``split``    a sequence-split step as it runs on one rank: attention over the token range gives a partial softmax
               state, the ranks' states (here one) are merged;
* ``prefill``  ``VQCodeCache.append`` of a whole prompt, with the quantised rows (which the adapter attends with) or without;
* ``train``    forward and backward of a codec module (``ClosedLoopUniformResidualVQ`` / ``ClosedLoopGroupedCQ``) on one
               layer: codes and rows out, then the gradients of the states and of the trainable V tables;
* ``rebuild``  rows from stored codes (``ops.decode``).

Layouts are (groups, stages, group width) of head_dim 128 with 256 words: ``gsrq2`` = (16, 2, 8) and ``full2`` =
(1, 2, 128) are the benchmark's, ``gsrq16`` = (1, 16, 128), ``cq16x8`` = (16, 1, 8) and ``cq32x4`` = (32, 1, 4) the deployed
ladders and grouped codebooks of the adapter.  8 KV heads throughout.
"""

from __future__ import annotations

import math

import torch

from tac_vq_kv_cache_b200 import ops
from tac_vq_kv_cache_b200.code_cache import VQCodeCache
from tac_vq_kv_cache_b200.jointkv.cq_tac import ClosedLoopGroupedCQ
from tac_vq_kv_cache_b200.jointkv.uniform_depth_tac import ClosedLoopUniformResidualVQ

HEADS, DIM, WORDS = 8, 128, 256
LAYOUTS = {"gsrq2": (16, 2, 8), "full2": (1, 2, 128), "gsrq16": (1, 16, 128), "cq16x8": (16, 1, 8), "cq32x4": (32, 1, 4)}
# spread of a stage's words: the benchmark's 0.5, 0.25 for grouped codebooks, 0.1 for full-width ones, and a shrinking ladder
SCALES = {"gsrq2": (0.5, 0.25), "full2": (0.1, 0.1), "gsrq16": tuple(0.09 * 0.9**s for s in range(16)), "cq16x8": (0.5,), "cq32x4": (0.5,)}
THETA = 1e6  # Mistral's rope base


def listed() -> list[dict]:
    return [
        # the smallest call: one user's chat a few hundred tokens long, where launches and host time are what counts
        {"name": "step-b1-777", "kind": "step", "layout": "gsrq2", "batch": 1, "tokens": 777, "q_heads": 32, "window": 0, "rotary": False},
        # the package's headline: batch 8 at 32k context, rows from the host and the result back to it
        {"name": "host-b8-32k", "kind": "host", "layout": "gsrq2", "batch": 8, "tokens": 32767, "q_heads": 32, "window": 0, "rotary": False},
        # the same serving batch under Mistral's sliding window; a length that ends inside a tile
        {"name": "step-b8-window4096", "kind": "step", "layout": "gsrq2", "batch": 8, "tokens": 30001, "q_heads": 32, "window": 4096, "rotary": False},
        # one very long sequence: the part of it that one of several ranks, or a single GPU, scans
        {"name": "split-b1-131k", "kind": "split", "layout": "gsrq2", "batch": 1, "tokens": 131071, "q_heads": 32, "window": 0, "rotary": False},
        # two additive full-width codebooks: one layer of the all-layer configuration
        {"name": "step-full2-b16-16k", "kind": "step", "layout": "full2", "batch": 16, "tokens": 16383, "q_heads": 32, "window": 0, "rotary": False},
        # codes of pre-rotary keys, as the adapter stores them, for a serving batch
        {"name": "step-rotary-b8-32k", "kind": "step", "layout": "gsrq2", "batch": 8, "tokens": 32767, "q_heads": 32, "window": 0, "rotary": True},
        # the adapter as it is deployed: depth-16 ladder, one sequence, rotary keys, window of 4096
        {"name": "step-ladder16-rotary-b1", "kind": "step", "layout": "gsrq16", "batch": 1, "tokens": 6143, "q_heads": 32, "window": 4096, "rotary": True},
        # prompt of a serving batch: K and V encoded, quantised rows wanted for the prompt's own attention
        {"name": "prefill-b4-8k", "kind": "prefill", "layout": "gsrq2", "batch": 4, "tokens": 8192, "recon": True, "dtype": "fp16"},
        # the largest: the whole context of one layer of the all-layer configuration, codes only
        {"name": "prefill-full2-b16-16k", "kind": "prefill", "layout": "full2", "batch": 16, "tokens": 16384, "recon": False, "dtype": "fp16"},
        # one training step of the V tables of the deployed ladder, keys assigned in a whitened space
        {"name": "train-ladder16", "kind": "train", "layout": "gsrq16", "batch": 1, "tokens": 2048, "whitened": True, "dtype": "fp16"},
        # the same for grouped codebooks with selector whiteners; an odd length, fp32 states
        {"name": "train-cq32x4", "kind": "train", "layout": "cq32x4", "batch": 1, "tokens": 3001, "whitened": True, "dtype": "fp32"},
        # a cache handed back to ordinary attention: all rows of batch 8 at 32k context, fp16
        {"name": "rebuild-b8-32k", "kind": "rebuild", "layout": "gsrq2", "batch": 8, "tokens": 32768, "dtype": "fp16"},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng) -> dict:
    """One more case: any kind over its whole range of layouts, lengths, batches and options."""
    kind = rng.choice(("step", "step", "step", "host", "split", "prefill", "prefill", "train", "train", "rebuild"))
    if kind in ("step", "host", "split"):
        rotary = kind == "step" and rng.random() < 0.4
        layout = "gsrq2" if kind != "step" else rng.choice(("gsrq2", "gsrq2", "full2", "gsrq16", "cq16x8", "cq32x4"))
        # at most the listed 8 x 32k tokens a step; the deep ladder serves a few sequences at a time
        most = 262144 if layout != "gsrq16" else 16384 if rotary else 65536
        batch = 1 if kind == "split" else rng.choice((1, 2, 3, 4, 8, 16))
        tokens = _log_int(rng, 64, min(131072, most // batch))
        window = 4096 if kind != "split" and tokens > 4096 and rng.random() < 0.4 else 0
        q_heads = rng.choice((32, 32, 16, 8))
        return {"kind": kind, "layout": layout, "batch": batch, "tokens": tokens, "q_heads": q_heads, "window": window, "rotary": rotary}
    batch = rng.choice((1, 1, 2, 3, 4, 8))
    if kind == "prefill":
        layout = rng.choice(tuple(LAYOUTS))
        most = {"gsrq16": 16384, "full2": 262144}.get(layout, 65536)
        tokens = _log_int(rng, 16, min(32768, most // batch))
        return {"kind": kind, "layout": layout, "batch": batch, "tokens": tokens, "recon": rng.random() < 0.5, "dtype": rng.choice(("fp16", "fp16", "fp32"))}
    if kind == "train":
        layout = rng.choice(("gsrq16", "gsrq16", "full2", "cq16x8", "cq32x4"))
        tokens = _log_int(rng, 128, 4096 // batch)
        return {"kind": kind, "layout": layout, "batch": batch, "tokens": tokens, "whitened": rng.random() < 0.6, "dtype": rng.choice(("fp16", "fp16", "fp32"))}
    layout = rng.choice(tuple(LAYOUTS))
    tokens = _log_int(rng, 16, min(131072, 262144 // batch))
    return {"kind": kind, "layout": layout, "batch": batch, "tokens": tokens, "dtype": rng.choice(("fp16", "fp16", "fp32"))}


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _tables(gen, layout: str) -> torch.Tensor:
    """fp32 masters [H,S,G,K,d]."""
    groups, stages, sub = LAYOUTS[layout]
    words = torch.randn(HEADS, stages, groups, WORDS, sub, device="cuda", generator=gen)
    return words * torch.tensor(SCALES[layout], device="cuda").view(1, stages, 1, 1, 1)


def _rows(gen, batch: int, tokens: int, dtype: torch.dtype, outliers: int = 0) -> torch.Tensor:
    """States [B,H,T,D], N(0,1); keys have a few channels per head that are eight times as large."""
    x = torch.randn(batch, HEADS, tokens, DIM, device="cuda", generator=gen)
    if outliers:
        for h in range(HEADS):
            x[:, h, :, torch.randperm(DIM, device="cuda", generator=gen)[:outliers]] *= 8.0
    return x.to(dtype)


def _filled_cache(gen, case: dict) -> VQCodeCache:
    """A cache in the middle of decoding: codes of `tokens` positions stored, room for the next one."""
    tokens = case["tokens"]
    cache = VQCodeCache(
        _tables(gen, case["layout"]), _tables(gen, case["layout"]), batch=case["batch"], max_tokens=tokens + 1,
        window=case["window"] or None, device="cuda", rope_theta=THETA if case["rotary"] else None,
    )
    for side in (cache.key, cache.value):
        side.random_(0, 256, generator=gen)
    cache.length = tokens
    return cache


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, layout, batch, tokens = case["kind"], case["layout"], case["batch"], case["tokens"]
    groups, stages, sub = LAYOUTS[layout]
    dtype = torch.float32 if case.get("dtype") == "fp32" else torch.float16
    state = {"case": case}
    if kind in ("step", "host", "split"):
        state["cache"] = _filled_cache(gen, case)
        query = (torch.randn(batch, case["q_heads"], DIM, device="cuda", generator=gen) / DIM**0.5).half()
        key, value = _rows(gen, batch, 1, torch.float16, 4), _rows(gen, batch, 1, torch.float16)
        if kind == "host":
            state["rows"] = torch.cat([query.flatten(), key.flatten(), value.flatten()]).cpu().pin_memory()
            state["out"] = torch.empty(batch, case["q_heads"], DIM, dtype=torch.float16).pin_memory()
        else:
            state.update(query=query, key=key, value=value)
    elif kind == "prefill":
        state["cache"] = VQCodeCache(_tables(gen, layout), _tables(gen, layout), batch=batch, max_tokens=tokens, device="cuda")
        state.update(key=_rows(gen, batch, tokens, dtype, 4), value=_rows(gen, batch, tokens, dtype))
    elif kind == "train":
        key_table, value_table = _tables(gen, layout), _tables(gen, layout)
        width = DIM if groups == 1 else sub
        whitener = torch.eye(width, device="cuda").expand(HEADS, groups, width, width)
        if case["whitened"]:
            whitener = whitener + 0.3 * torch.randn(HEADS, groups, width, width, device="cuda", generator=gen) / width**0.5
        if groups == 1:
            state["codec"] = ClosedLoopUniformResidualVQ(
                [key_table[:, :, 0]], [value_table[:, :, 0]], [whitener[:, 0] if case["whitened"] else None], depth=stages, dynamic_bpa=1.0
            )
        else:
            state["codec"] = ClosedLoopGroupedCQ([key_table[:, 0]], [value_table[:, 0]], [whitener], dynamic_bpa=1.0)
        state.update(key=_rows(gen, batch, tokens, dtype, 4).requires_grad_(), value=_rows(gen, batch, tokens, dtype).requires_grad_())
        state.update(key_grad=_rows(gen, batch, tokens, dtype), value_grad=_rows(gen, batch, tokens, dtype))
    else:
        state["codes"] = torch.empty(batch, HEADS, tokens, stages, groups, dtype=torch.uint8, device="cuda").random_(0, 256, generator=gen)
        state.update(tables=ops.deployed_tables(_tables(gen, layout)), dtype=dtype)
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------


def run(state: dict):
    kind, case = state["case"]["kind"], state["case"]
    cache = state.get("cache")
    if kind == "step":
        cache.length = case["tokens"]  # the same position every time
        out = cache.decode_step(state["query"], state["key"], state["value"])
        return {"out": out, "key_codes": cache.key, "value_codes": cache.value}
    if kind == "host":
        cache.length = case["tokens"]
        out = cache.decode_step_host(state["rows"], state["out"], case["q_heads"], direct=True)
        return {"out": out, "key_codes": cache.key, "value_codes": cache.value}
    if kind == "split":
        _, partial = cache.attend(state["query"], want_state=True)
        return ops.attn_combine(partial[None])[0]  # the merge over the ranks' states, here of one
    if kind == "prefill":
        cache.reset()
        rows = cache.append(state["key"], state["value"], want_recon=case["recon"])
        return {"rows": rows, "key_codes": cache.key, "value_codes": cache.value}
    if kind == "train":
        codec = state["codec"]
        got = codec(0, state["key"], state["value"])
        grads = torch.autograd.grad(
            (got.key, got.value), (state["key"], state["value"], codec.value_tables[0]), (state["key_grad"], state["value_grad"])
        )
        return {"rows": (got.key, got.value), "codes": (got.key_indices, got.value_indices), "grads": grads}
    return ops.decode(state["codes"], state["tables"], state["dtype"])


def work(case: dict) -> dict:
    groups, stages, sub = LAYOUTS[case["layout"]]
    kind, batch, tokens = case["kind"], case["batch"], case["tokens"]
    table_words = HEADS * stages * WORDS * DIM  # of one side
    if kind in ("step", "host", "split"):
        seen = min(tokens + (kind != "split"), case["window"] or tokens + 1)
        codes = 2 * batch * HEADS * seen * stages * groups
        small = 2 * batch * (2 * case["q_heads"] + 2 * HEADS) * DIM
        return {"bytes": codes + 2 * 2 * table_words + small, "flops": 4 * batch * case["q_heads"] * seen * DIM}
    wide = 4 if case["dtype"] == "fp32" else 2
    values = batch * HEADS * tokens * DIM
    codes = batch * HEADS * tokens * stages * groups
    distances = 2 * batch * HEADS * tokens * stages * WORDS * DIM
    if kind == "prefill":
        return {"bytes": 2 * (values * wide * (2 if case["recon"] else 1) + codes + 2 * table_words), "flops": 2 * distances}
    if kind == "train":
        # states in, rows out, their gradients in, the states' gradients out; fp32 masters in, V table gradient out
        return {"bytes": 2 * (4 * values * wide + codes) + 3 * 4 * table_words, "flops": 2 * distances}
    return {"bytes": values * wide + codes + 2 * table_words, "flops": values * stages}


def tolerance(case: dict):
    # Against fp64 attention over the stored codes the steps measure rel 2.0e-4 to 2.8e-4 and max 4.5e-4 to 8.2e-4 (most of
    # it the rounding of the fp16 result); codes are whole numbers and stay the same.
    if case["kind"] in ("step", "host", "split"):
        return {"rel": 1.2e-3, "max": 4e-3, "differ": 0.0}
    # The table gradient is a sum of fp32 rows: rel 1e-7 and max 1.3e-6 against fp64 and between two runs.
    if case["kind"] == "train":
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
    return "exact"
