"""GPU parity of attention over codes of pre-rotary keys (the reference's decode branch with its
rotary step), through the C ABI.

Fixture ``rotary.npz``: that branch restated with transformers' Mistral rotary functions on the rebuilt
fp16 window and fp16 SDPA.  Oracle: the same with fp32 sums.  Tolerance (fp16 output): relative L2
error <= 2e-3 and max abs error <= 2e-3 of the largest reference magnitude.
"""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from oracle import jointkv_oracle as O
from tests.util import make_states, make_tables, max_rel, rel_l2

pytestmark = pytest.mark.gpu
TOL = 2e-3


def _ops():
    from tac_vq_kv_cache_b200 import ops

    return ops


def _check(out, want):
    assert rel_l2(out, want) <= TOL, (rel_l2(out, want), max_rel(out, want))
    assert max_rel(out, want) <= TOL, (rel_l2(out, want), max_rel(out, want))


@pytest.mark.parametrize("theta,dim,first", [(1000000.0, 128, 0), (10000.0, 128, 0), (10000.0, 64, 5), (500000.0, 256, 0)])
def test_rope_table_matches_the_reference_arithmetic(device, theta, dim, first):
    ops = _ops()
    tokens = 4099
    table = ops.rope_table(tokens, dim, theta, device, first_position=first).cpu()
    cos, sin = O.rotary_table(tokens, dim, theta, first)
    # fp32 cos/sin of two libraries may differ in the last place; after the cast to fp16 that is at most
    # one fp16 step on a vanishing share of the entries
    for got, want in ((table[:, 0], cos), (table[:, 1], sin)):
        differs = got != want
        assert float(differs.float().mean()) < 2e-3
        assert float((got.float() - want.float()).abs().max()) <= 2.0 ** -10


@pytest.mark.parametrize("case", ["gsrq", "cq"])
def test_rotary_attention_matches_the_reference_golden(golden, device, case):
    ops = _ops()
    g = golden("rotary.npz")
    q = g(f"{case}.q_rotated")
    dim = q.shape[-1]
    scaled = (q.float() / dim**0.5).half()
    kcodes, vcodes = g(f"{case}.kcodes"), g(f"{case}.vcodes")
    rope = ops.rope_table(kcodes.shape[2], dim, float(g(f"{case}.theta")), device)
    out, _ = ops.attn_decode(
        scaled.to(device), kcodes.to(device), vcodes.to(device), g(f"{case}.ktab").to(device), g(f"{case}.vtab").to(device),
        g(f"{case}.seq_start").to(device), g(f"{case}.seq_end").to(device), rope=rope,
    )
    _check(out.float().cpu(), g(f"{case}.out"))


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub,theta",
    [
        (2, 32, 8, 3000, 16, 2, 8, 1000000.0),   # benchmark geometry
        (1, 8, 8, 1500, 1, 2, 128, 10000.0),     # two full-width codebooks, no head sharing
        (2, 16, 2, 700, 32, 1, 4, 1000000.0),    # 8 query heads per KV head
        (1, 4, 2, 900, 8, 3, 8, 10000.0),        # head_dim 64
        (2, 8, 2, 5000, 32, 1, 4, 1000000.0),    # 32 groups of 4 in the two-pass kernel
        (2, 8, 4, 4500, 16, 1, 8, 10000.0),      # one-stage grouped CQ in the two-pass kernel
        (1, 8, 4, 9001, 16, 2, 8, 10000.0),      # benchmark layout, 2 query heads per KV head, several splits, ragged tail
        (2, 4, 4, 333, 16, 2, 8, 1000000.0),     # benchmark layout without head sharing, less than one block of tokens
    ],
)
def test_rotary_attention_matches_the_oracle(device, b, hq, hkv, t, groups, stages, sub, theta):
    ops = _ops()
    gen = torch.Generator().manual_seed(t)
    dim = groups * sub
    kcodes = torch.randint(0, 256, (b, hkv, t, stages, groups), generator=gen, dtype=torch.uint8)
    vcodes = torch.randint(0, 256, (b, hkv, t, stages, groups), generator=gen, dtype=torch.uint8)
    scales = [0.1] * stages if sub == 128 else None
    ktab = make_tables(gen, hkv, stages, groups, sub, scales)
    vtab = make_tables(gen, hkv, stages, groups, sub, scales)
    q = (torch.randn(b, hq, dim, generator=gen) / dim**0.5).half()
    start, end = [0, 123][:b], [t, t - 57][:b]
    want, m, l, acc = O.attention_over_codes(q, kcodes, vcodes, ktab, vtab, start, end, rope_theta=theta)
    rope = ops.rope_table(t, dim, theta, device)
    out, state = ops.attn_decode(
        q.to(device), kcodes.to(device), vcodes.to(device), ktab.to(device), vtab.to(device),
        torch.tensor(start, dtype=torch.int32, device=device), torch.tensor(end, dtype=torch.int32, device=device),
        rope=rope, want_state=True,
    )
    _check(out.float().cpu(), want)
    state = state.cpu()
    lse, want_lse = state[..., 0] + state[..., 1].log(), m + l.log()
    torch.testing.assert_close(lse, want_lse, rtol=0, atol=2e-3)
    _check(state[..., 2:] / state[..., 1:2], acc / l[..., None])


@pytest.mark.parametrize(
    "b,hq,hkv,t,ranges",
    [
        (3, 8, 2, 700, [(0, 700), (100, 333), (5, 5)]),                                   # one block's rows: whole, part, nothing
        (4, 4, 4, 2049, [(0, 1), (2048, 2049), (7, 1500), (1024, 1032)]),                 # ranges that hardly meet
        (5, 8, 4, 4100, [(0, 4100), (4, 4099), (4000, 4100), (300, 100), (0, 8)]),        # rows spread over two unequal groups
        (2, 8, 2, 6150, [(0, 6150), (3, 6149)]),                                          # more positions than one chunk of two rows
        (9, 2, 2, 31, [(0, 31)] * 8 + [(30, 31)]),                                        # less than a tile
    ],
)
def test_rotary_rows_of_a_batch_that_share_positions(device, b, hq, hkv, t, ranges):
    """Rows of one block stand at the same positions but see ranges of their own; a row that sees nothing gets zeros."""
    ops = _ops()
    gen = torch.Generator().manual_seed(b * t)
    kcodes, vcodes = (torch.randint(0, 256, (b, hkv, t, 2, 16), generator=gen, dtype=torch.uint8) for _ in range(2))
    ktab, vtab = make_tables(gen, hkv, 2, 16, 8), make_tables(gen, hkv, 2, 16, 8)
    q = (torch.randn(b, hq, 128, generator=gen) / 128**0.5).half()
    start, end = [r[0] for r in ranges], [r[1] for r in ranges]
    live = [i for i in range(b) if end[i] > start[i]]
    want, *_ = O.attention_over_codes(q[live], kcodes[live], vcodes[live], ktab, vtab, [start[i] for i in live], [end[i] for i in live], rope_theta=1e6)
    out, state = ops.attn_decode(
        q.to(device), kcodes.to(device), vcodes.to(device), ktab.to(device), vtab.to(device),
        torch.tensor(start, dtype=torch.int32, device=device), torch.tensor(end, dtype=torch.int32, device=device),
        rope=ops.rope_table(t, 128, 1e6, device), want_state=True,
    )
    out, state = out.float().cpu(), state.cpu()
    for i, row in enumerate(live):
        _check(out[row], want[i])
    for row in set(range(b)) - set(live):
        assert not out[row].any() and (state[row, :, 0] == -float("inf")).all() and not state[row, :, 1:].any()


@pytest.mark.parametrize(
    "b,hq,hkv,stages,t,ranges,peak",
    [
        (1, 4, 1, 16, 1, [(0, 1)], 1.0),                                                  # one token, one cluster
        (1, 8, 2, 4, 17, [(0, 17)], 1.0),                                                 # a tile and a token, four stages
        (2, 16, 4, 8, 511, [(3, 500), (10, 10)], 1.0),                                    # a row that sees nothing
        (1, 8, 8, 12, 4097, [(0, 4097)], 1.0),                                            # a token more than a cluster holds at a time
        (5, 8, 4, 16, 300, [(0, 300), (299, 300), (0, 1), (17, 250), (100, 164)], 1.0),   # more items than clusters, heads change inside one
        (1, 4, 2, 16, 3000, [(0, 3000)], 12.0),                                           # one token carries most of the weight
    ],
)
def test_rotary_attention_over_deep_ladders(device, b, hq, hkv, stages, t, ranges, peak):
    """Full-width ladders of 4 to 16 stages; ``peak``: by how much the first token's logit stands out."""
    ops = _ops()
    gen = torch.Generator().manual_seed(stages * t)
    kcodes, vcodes = (torch.randint(0, 256, (b, hkv, t, stages, 1), generator=gen, dtype=torch.uint8) for _ in range(2))
    scales = [0.3 * 0.85**s for s in range(stages)]
    ktab, vtab = make_tables(gen, hkv, stages, 1, 128, scales), make_tables(gen, hkv, stages, 1, 128, scales)
    q = (torch.randn(b, hq, 128, generator=gen) / 128**0.5).half()
    if peak > 1.0:  # queries along the first token's key, which stands at position 0: no rotation
        key = ktab[:, torch.arange(stages), 0, kcodes[0, :, 0, :, 0].long()][torch.arange(hkv), torch.arange(hkv)].float().sum(1)
        q = (peak * key / (key * key).sum(-1, keepdim=True)).half().repeat_interleave(hq // hkv, 0)[None].expand(b, -1, -1).contiguous()
    start, end = [r[0] for r in ranges], [r[1] for r in ranges]
    live = [i for i in range(b) if end[i] > start[i]]
    want, m, l, acc = O.attention_over_codes(q[live], kcodes[live], vcodes[live], ktab, vtab, [start[i] for i in live], [end[i] for i in live], rope_theta=1e6)
    out, state = ops.attn_decode(
        q.to(device), kcodes.to(device), vcodes.to(device), ktab.to(device), vtab.to(device),
        torch.tensor(start, dtype=torch.int32, device=device), torch.tensor(end, dtype=torch.int32, device=device),
        rope=ops.rope_table(t, 128, 1e6, device), want_state=True,
    )
    out, state = out.float().cpu(), state.cpu()
    for i, row in enumerate(live):
        _check(out[row], want[i])
    torch.testing.assert_close(state[live][..., 0] + state[live][..., 1].log(), m + l.log(), rtol=0, atol=2e-3)
    for row in set(range(b)) - set(live):
        assert not out[row].any() and (state[row, :, 0] == -float("inf")).all() and not state[row, :, 1:].any()


@pytest.mark.parametrize("stages,word", [(4, float("inf")), (16, float("inf")), (12, float("-inf"))])
def test_an_infinite_key_word_of_a_ladder_stays_with_its_token(device, stages, word):
    """A token whose score is -inf has no weight; the tokens beside it keep theirs."""
    ops = _ops()
    gen = torch.Generator().manual_seed(stages)
    kcodes, vcodes = (torch.randint(0, 255, (1, 2, 100, stages, 1), generator=gen, dtype=torch.uint8) for _ in range(2))
    ktab, vtab = (make_tables(gen, 2, stages, 1, 128, [0.3 * 0.85**s for s in range(stages)]) for _ in range(2))
    q = (torch.randn(1, 8, 128, generator=gen) / 128**0.5).half()
    q[:, :, [5, 69]] = -0.1 if word > 0 else 0.1  # at position 1 channel 5 and its partner both get words of that sign
    ktab[:, stages - 2, 0, 255, 5] = word
    kcodes[:, :, 1, stages - 2, 0] = 255
    want, *_ = O.attention_over_codes(q, kcodes, vcodes, ktab, vtab, rope_theta=1e6)
    assert bool(want.isfinite().all())
    out, _ = ops.attn_decode(*(x.to(device) for x in (q, kcodes, vcodes, ktab, vtab)), rope=ops.rope_table(100, 128, 1e6, device))
    _check(out.float().cpu(), want)

@pytest.mark.parametrize("stages", [4, 16])
@pytest.mark.parametrize("tokens,first,last", [(2, 1, 2), (3, 1, 2), (8, 7, 8), (9, 8, 9), (57, 56, 57), (800, 100, 200), (800, 95, 205), (4500, 1, 4500), (9000, 1, 9000)])
def test_infinite_scores_of_a_whole_share_of_a_ladder_weigh_nothing(device, stages, tokens, first, last):
    """Tokens first..last score -inf: all that one of eight blocks adds up the scores of, or a whole split.  That is so for one head of
    four; the others score +inf there, which is NaN, and no other head's result is."""
    ops = _ops()
    gen = torch.Generator().manual_seed(stages + tokens)
    kcodes, vcodes = (torch.randint(0, 255, (1, 1, tokens, stages, 1), generator=gen, dtype=torch.uint8) for _ in range(2))
    ktab, vtab = (make_tables(gen, 1, stages, 1, 128, [0.3 * 0.85**s for s in range(stages)]) for _ in range(2))
    q = (torch.randn(1, 4, 128, generator=gen) / 128**0.5).half()
    q[:, :, [63, 127]] = 0.1
    q[:, 2, [63, 127]] = -0.1  # from position 1 on channel 63 and its partner both get words of the same sign
    ktab[:, 1, 0, 255, 63] = float("inf")
    kcodes[:, :, first:last, 1, 0] = 255
    arguments = [x.to(device) for x in (q, kcodes, vcodes, ktab, vtab)]
    rope = ops.rope_table(tokens, 128, 1e6, device)
    want, *_ = O.attention_over_codes(q, kcodes, vcodes, ktab, vtab, rope_theta=1e6)
    assert bool(want[:, 2].isfinite().all()) and bool(want[:, [0, 1, 3]].isnan().all())
    out, state = ops.attn_decode(*arguments, rope=rope, want_state=True)
    _check(out[:, 2].float().cpu(), want[:, 2])
    assert bool(out[:, [0, 1, 3]].isnan().all()) and bool(state[:, 2].isfinite().all())
    # a range of nothing but such tokens has no result, as it has none in softmax
    start, end = (torch.tensor([x], dtype=torch.int32, device=device) for x in (first, last))
    out, _ = ops.attn_decode(*arguments, seq_start=start, seq_end=end, rope=rope)
    assert bool(out.isnan().all())


@pytest.mark.parametrize("b,hq,hkv,stages,t", [(1, 4, 1, 16, 4096), (2, 8, 4, 16, 700), (1, 2, 2, 8, 3000), (2, 8, 2, 4, 9000)])
def test_ladder_weights_have_the_precision_of_fp32(device, b, hq, hkv, stages, t):
    """The state against 64 bits, for logits over a range of about 30 and a rotary table that turns nothing: keys are the sums of their
    words in fp16, values the sums themselves.

    A weight is exp of an fp32 difference of at most 30 (2^-24 of it, 1.8e-6) by exp2 with two units in the last place (1.2e-7 each); the
    errors of different tokens are not alike, so a weighted mean has less than a single weight's.
    """
    ops = _ops()
    gen = torch.Generator().manual_seed(stages * t)
    ktab, vtab = (make_tables(gen, hkv, stages, 1, 128, [1.2 / stages] * stages) for _ in range(2))
    codes = [torch.randint(0, 256, (b, hkv, t, stages, 1), generator=gen, dtype=torch.uint8) for _ in range(2)]
    q = (6 * torch.randn(b, hq, 128, generator=gen) / 128**0.5).half()
    still = torch.zeros(t, 2, 64, dtype=torch.float16, device=device)
    still[:, 0] = 1.0
    _, state = ops.attn_decode(q.to(device), *(x.to(device) for x in (*codes, ktab, vtab)), rope=still, want_out=False, want_state=True)
    heads = torch.arange(hkv)[None, :, None]
    key, value = (sum(tab[:, s, 0].double()[heads, c[:, :, :, s, 0].long()] for s in range(stages)).repeat_interleave(hq // hkv, 1) for c, tab in zip(codes, (ktab, vtab)))
    score = torch.einsum("bhd,bhtd->bht", q.double(), key.half().double())
    state = state.cpu().double()
    assert rel_l2(state[..., 2:] / state[..., 1:2], torch.einsum("bht,bhtd->bhd", score.softmax(-1), value)) <= 1.5e-6
    torch.testing.assert_close(state[..., 0] + state[..., 1].log(), score.logsumexp(-1), rtol=0, atol=4e-6)

@pytest.mark.parametrize(
    "batch,heads,q_heads,groups,stages,sub,max_tokens,window,first,new",
    [
        (1, 8, 32, 1, 16, 128, 513, None, 295, 1),   # rows of odd length: every position's codes begin inside a sector in some head
        (1, 8, 32, 1, 16, 128, 4097, None, 4081, 1),
        (3, 8, 16, 1, 16, 128, 337, None, 310, 1),   # more items than clusters, heads change inside one
        (1, 2, 8, 1, 4, 128, 45, None, 0, 1),        # from the first token on: a new token alone in its tile
        (5, 3, 3, 1, 8, 128, 271, 100, 250, 1),      # the range moves against the tiles
        (2, 4, 16, 1, 12, 128, 303, None, 240, 3),   # several new tokens, across the end of a tile
        (1, 1, 4, 1, 16, 128, 1023, None, 500, 2),
        (3, 2, 8, 16, 2, 8, 333, None, 305, 1),
        (5, 2, 4, 16, 2, 8, 97, 40, 60, 2),
    ],
)
def test_a_step_sees_the_codes_of_its_own_token(device, batch, heads, q_heads, groups, stages, sub, max_tokens, window, first, new):
    """Attention starts before the new token's codes are written over others: whatever was there before must not be seen.  The new
    key carries most of the weight, and steps go over the edges of tiles, sectors and splits."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(max_tokens + stages)
    scales = [0.5 * 0.85**s for s in range(stages)] if groups == 1 else None
    tables = [make_tables(gen, heads, stages, groups, sub, scales) for _ in range(2)]
    cache = VQCodeCache(*tables, batch=batch, max_tokens=max_tokens, window=window, device=device, rope_theta=1e6)
    kept = [torch.randint(0, 256, cache.key.shape, generator=gen, dtype=torch.uint8) for _ in range(2)]
    cache.key.copy_(kept[0]), cache.value.copy_(kept[1])
    cache.length = first
    last = min(first + 34, max_tokens)
    for end in range(first + new, last + 1, new):
        rows = [make_states(gen, (batch, heads, new, 128)) for _ in range(2)]
        for store, table, row in zip(kept, tables, rows):
            C.encode(row, table, codes=store, t0=end - new, want_recon=False)
        key = O.reconstruct(kept[0][:, :, end - 1 : end], tables[0], torch.float16)
        key = O.apply_rotary_fp16(key, *O.rotary_table(1, 128, 1e6, end - 1)).float()[:, :, 0]
        query = (9.0 * key / (key * key).sum(-1, keepdim=True)).half().repeat_interleave(q_heads // heads, 1)
        out = cache.decode_step(query.to(device), *(row.to(device) for row in rows))
        start, stop = cache.visible()
        want, *_ = O.attention_over_codes(query, *kept, *tables, [start] * batch, [stop] * batch, rope_theta=1e6)
        assert torch.equal(cache.key.cpu(), kept[0]) and torch.equal(cache.value.cpu(), kept[1])
        _check(out.float().cpu(), want)

def test_code_cache_with_rope_follows_the_reference_decode_loop(device):
    """Prefill + three decode steps through VQCodeCache(rope_theta=...): codes of pre-rotary keys are
    appended in place, the query arrives rotated; compared with the oracle on the cache's own codes."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(77)
    b, hq, hkv, dim, theta = 1, 8, 2, 128, 1000000.0
    ktab = make_tables(gen, hkv, 2, 16, 8)
    vtab = make_tables(gen, hkv, 2, 16, 8)
    cache = VQCodeCache(ktab, vtab, batch=b, max_tokens=512, window=400, device=device, rope_theta=theta)
    cache.append(torch.randn(b, hkv, 380, dim, generator=gen).half().to(device), torch.randn(b, hkv, 380, dim, generator=gen).half().to(device))
    for _ in range(30):
        q = (torch.randn(b, hq, dim, generator=gen) / dim**0.5).half()
        k = torch.randn(b, hkv, 1, dim, generator=gen).half()
        v = torch.randn(b, hkv, 1, dim, generator=gen).half()
        out = cache.decode_step(q.to(device), k.to(device), v.to(device))
        start, end = cache.visible()
        want, *_ = O.attention_over_codes(q, cache.key.cpu(), cache.value.cpu(), ktab, vtab, [start], [end], rope_theta=theta)
        _check(out.float().cpu(), want)
    assert cache.length == 410 and cache.visible() == (10, 410)


def test_rotary_argument_errors(device):
    from tac_vq_kv_cache_b200 import _lib

    ops = _ops()
    with pytest.raises(_lib.TacvqError):
        ops.rope_table(16, 127, 10000.0, device)          # odd head_dim
    with pytest.raises(_lib.TacvqError):
        ops.rope_table(16, 128, -1.0, device)             # theta must be positive
    gen = torch.Generator().manual_seed(1)
    codes = torch.randint(0, 256, (1, 2, 64, 2, 16), generator=gen, dtype=torch.uint8).to(device)
    tab = make_tables(gen, 2, 2, 16, 8).to(device)
    q = torch.zeros(1, 8, 128, dtype=torch.float16, device=device)
    with pytest.raises(ValueError):
        ops.attn_decode(q, codes, codes, tab, tab, rope=torch.zeros(32, 2, 64, dtype=torch.float16, device=device))
