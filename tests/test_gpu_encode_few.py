"""GPU parity of the few-row encode of wide groups (decode steps): a block per (side, head, group) and one, two or four rows.

Row counts on both sides of every split (rows per block, the last block's missing rows), table rings that are and are not
recycled (more than three stages), small codebooks, one so small that the kernel does not take it, and the decode step that
encodes both sides at once.  Codes and rows are bit-exact with the C oracle.
"""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from tests.util import make_states, make_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "batch,tokens,sub,groups,stages,words,dtype",
    [
        (1, 1, 128, 1, 16, 256, torch.float16),
        (8, 1, 128, 1, 2, 256, torch.float16),
        (9, 1, 128, 1, 3, 201, torch.float32),
        (1, 16, 128, 1, 18, 256, torch.float16),
        (17, 1, 64, 2, 2, 33, torch.float16),
        (4, 8, 32, 4, 2, 256, torch.float32),
        (2, 5, 64, 2, 1, 7, torch.float16),   # 28 words in all: not this kernel's
        (2, 5, 64, 2, 16, 7, torch.float16),
        (1, 3, 32, 4, 33, 96, torch.float16),
    ],
)
def test_few_rows_of_wide_groups_are_bit_exact(device, batch, tokens, sub, groups, stages, words, dtype):
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(sub + batch)
    tables = make_tables(gen, 2, stages, groups, sub, [0.1 * 0.9**s for s in range(stages)])[:, :, :, :words].contiguous()
    states = make_states(gen, (batch, 2, tokens, 128), dtype)
    cache = torch.full((batch, 2, tokens + 3, stages, groups), 0xEE, dtype=torch.uint8, device=device)
    want, want_recon = C.encode(states, tables)
    codes, recon = ops.encode(states.to(device), tables.to(device), codes=cache, t0=2)
    assert torch.equal(codes[:, :, 2 : 2 + tokens].cpu(), want)
    assert torch.equal(recon.cpu(), want_recon)
    assert bool((codes[:, :, :2] == 0xEE).all()) and bool((codes[:, :, 2 + tokens :] == 0xEE).all())
    norms = ops.table_sqnorm(tables.to(device))
    again, _ = ops.encode(states.to(device), tables.to(device), table_sqnorm=norms, want_recon=False)
    assert torch.equal(again.cpu(), want)
    assert ops.encode_tensor_memory_timeouts(device) == 0


@pytest.mark.parametrize("rope", [None, 1e6])
@pytest.mark.parametrize("batch,groups,stages,sub", [(3, 1, 2, 128), (1, 1, 16, 128), (2, 2, 2, 64), (2, 32, 1, 4)])
def test_decode_step_appends_the_codes_and_attends_like_the_separate_calls(device, rope, batch, groups, stages, sub):
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(stages)
    tables = [make_tables(gen, 2, stages, groups, sub, [0.1 * 0.9**s for s in range(stages)]) for _ in range(2)]
    caches = [VQCodeCache(*tables, batch=batch, max_tokens=80, window=48, device=device, rope_theta=rope) for _ in range(2)]
    prompt = [make_states(gen, (batch, 2, 70, 128)) for _ in range(2)]
    for cache in caches:
        cache.append(*(p.to(device) for p in prompt))
    for step in range(3):
        query = (torch.randn(batch, 8, 128, generator=gen) / 128**0.5).half().to(device)
        new = [make_states(gen, (batch, 2, 1, 128)) for _ in range(2)]
        out = caches[0].decode_step(query, *(n.to(device) for n in new))
        caches[1].append(*(n.to(device) for n in new))
        assert torch.equal(out, caches[1].attend(query))
        for side, table, row in (("key", tables[0], new[0]), ("value", tables[1], new[1])):
            want, _ = C.encode(row, table, want_recon=False)
            assert torch.equal(getattr(caches[0], side)[:, :, 70 + step : 71 + step].cpu(), want)
    assert torch.equal(caches[0].key, caches[1].key) and torch.equal(caches[0].value, caches[1].value)


@pytest.mark.parametrize("scale", [1.0, 1e-3, 3e4])
@pytest.mark.parametrize("rows,sub,groups", [(1, 128, 1), (13, 64, 2), (32, 32, 4)])
def test_ties_and_extreme_scales_are_left_to_the_exact_chain(device, rows, sub, groups, scale):
    """Every word stored twice (all rows tie), rows that are words, rows half way between two words; magnitudes near
    fp16's ends.  The lowest index wins, as in a sequential scan."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(rows)
    tables = make_tables(gen, 2, 2, groups, sub, [0.2, 0.1]).float() * scale
    tables[:, :, :, 1::2] = tables[:, :, :, 0::2]
    tables = tables.clamp(-60000, 60000).half()
    pick = torch.randint(0, 256, (2, rows, 2, groups), generator=gen)
    first = tables[:, 0].float()  # [H,G,K,d]
    states = torch.stack([torch.stack([
        torch.cat([(first[h, g, pick[h, r, 0, g]] + (first[h, g, pick[h, r, 1, g]] if r % 2 else first[h, g, pick[h, r, 0, g]])) / 2 for g in range(groups)])
        for r in range(rows)]) for h in range(2)])[None].half()
    want, want_recon = C.encode(states, tables)
    codes, recon = ops.encode(states.to(device), tables.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)


def test_rows_of_a_wide_cache_feed_the_next_step_of_a_narrow_one(device):
    """The quantised rows of a few-row encode are a later launch's input on the same stream: all of them are there when it reads them."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(5)
    wide_tables = [make_tables(gen, 8, 16, 1, 128, [0.1 * 0.9**s for s in range(16)]) for _ in range(2)]
    narrow_tables = [make_tables(gen, 8, 2, 16, 8) for _ in range(2)]
    wide = VQCodeCache(*wide_tables, batch=1, max_tokens=12, device=device)
    narrow = VQCodeCache(*narrow_tables, batch=1, max_tokens=12, device=device)
    query = (torch.randn(1, 32, 128, generator=gen) / 128**0.5).half().to(device)
    states = [[make_states(gen, (1, 8, 1, 128)).to(device) for _ in range(2)] for _ in range(12)]
    rows = []
    for key, value in states:
        rows.append(wide.append(key, value, want_recon=True))
        narrow.decode_step(query, *rows[-1])
    for t, (key, value) in enumerate(states):
        for got, codes, table, deep, x in zip(rows[t], (narrow.key, narrow.value), narrow_tables, wide_tables, (key, value)):
            want_row = C.encode(x.cpu(), deep)[1]
            assert torch.equal(got.cpu(), want_row)
            assert torch.equal(codes[:, :, t : t + 1].cpu(), C.encode(want_row, table, want_recon=False)[0])
