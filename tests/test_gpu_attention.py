"""GPU parity of decode-step attention over codes (through the C ABI).

Oracle: rebuild K and V from the codes as the reference does (fp32 stage sum,
one cast to fp16), repeat KV heads, softmax(q K^T) V over the visible range.
Tolerance (fp16 output): relative L2 error <= 2e-3 and max abs error <= 2e-3 of
the largest reference magnitude.
"""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from tests.util import make_tables, max_rel, rel_l2

pytestmark = pytest.mark.gpu
TOL = 2e-3


def _ops():
    from tac_vq_kv_cache_b200 import ops

    return ops


def _workload(seed, b, hq, hkv, t, groups, stages, sub, scales=None):
    gen = torch.Generator().manual_seed(seed)
    dim = groups * sub
    kcodes = torch.randint(0, 256, (b, hkv, t, stages, groups), generator=gen, dtype=torch.uint8)
    vcodes = torch.randint(0, 256, (b, hkv, t, stages, groups), generator=gen, dtype=torch.uint8)
    ktab = make_tables(gen, hkv, stages, groups, sub, scales)
    vtab = make_tables(gen, hkv, stages, groups, sub, scales)
    q = (torch.randn(b, hq, dim, generator=gen) / dim**0.5).half()
    return q, kcodes, vcodes, ktab, vtab


def _check(out, want):
    assert rel_l2(out, want) <= TOL, (rel_l2(out, want), max_rel(out, want))
    assert max_rel(out, want) <= TOL, (rel_l2(out, want), max_rel(out, want))


def _check_state(state, want):
    """(m, l, acc) is defined up to its reference m: compare log-sum-exp m + ln l and acc / l."""
    lse, want_lse = state[..., 0] + state[..., 1].log(), want[..., 0] + want[..., 1].log()
    torch.testing.assert_close(lse, want_lse, rtol=0, atol=2e-3)
    assert bool((state[..., 0] <= want[..., 0] + 2e-3).all())       # the reference never exceeds the maximum score
    assert bool((state[..., 0] >= want[..., 0] - 5.6).all())        # and stays within 8 octaves (8 ln 2) of it
    _check(state[..., 2:] / state[..., 1:2], want[..., 2:] / want[..., 1:2])


def _run(device, work, start=None, end=None, **kw):
    ops = _ops()
    dev = [x.to(device) for x in work]
    st = None if start is None else torch.tensor(start, dtype=torch.int32, device=device)
    en = None if end is None else torch.tensor(end, dtype=torch.int32, device=device)
    return ops.attn_decode(*dev, st, en, **kw)


@pytest.mark.parametrize("case", ["gsrq", "cq"])
def test_attention_matches_reference_golden(golden, device, case):
    g = golden("attention.npz")
    work = tuple(g(f"{case}.{n}") for n in ("q", "kcodes", "vcodes", "ktab", "vtab"))
    out, _ = _run(device, work, g(f"{case}.seq_start").tolist(), g(f"{case}.seq_end").tolist())
    _check(out, g(f"{case}.out"))


@pytest.mark.parametrize("tokens", [1, 2, 31, 32, 33, 255, 257, 1000, 4097])
def test_gsrq2_geometry_ragged_lengths(device, tokens):
    work = _workload(tokens, 2, 8, 2, tokens, 16, 2, 8)
    out, state = _run(device, work, want_state=True)
    want, want_state = C.attention(*work)
    _check(out, want)
    _check_state(state.cpu(), want_state)


def test_sliding_window_and_empty_rows(device):
    # 6144 stored tokens, the last 4096 visible (the reference's window), one row empty, one row partial
    work = _workload(5, 4, 8, 2, 6144, 16, 2, 8)
    start, end = [2048, 0, 100, 6000], [6144, 0, 4196, 6144]
    out, state = _run(device, work, start, end, want_state=True)
    want, want_state = C.attention(*work, start, end)
    _check(out, want)
    assert bool((out[1] == 0).all()) and bool((state[1, :, 1] == 0).all()) and bool(torch.isinf(state[1, :, 0]).all())


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub",
    [
        (2, 8, 2, 700, 1, 2, 128),   # two additive full-width codebooks
        (2, 8, 2, 1, 1, 2, 128),     # ... a single token
        (1, 32, 8, 5000, 1, 16, 128),  # the reference's own GSRQ layout at depth 16, 4 query heads per KV head
        (1, 8, 8, 300, 1, 16, 128),  # the reference's own GSRQ layout, depth 16, no query-head sharing
        (2, 4, 2, 500, 16, 1, 8),    # one-stage grouped CQ
        (1, 4, 1, 400, 32, 1, 4),    # 32 groups of 4
        (2, 16, 2, 333, 8, 2, 8),    # 8 query heads per KV head, head_dim 64
    ],
)
def test_other_geometries(device, b, hq, hkv, t, groups, stages, sub):
    work = _workload(9, b, hq, hkv, t, groups, stages, sub, [0.1] * stages if sub == 128 else None)
    out, _ = _run(device, work)
    want, _ = C.attention(*work)
    _check(out, want)


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub",
    [
        (8, 32, 8, 5000, 16, 1, 8),   # one-stage grouped CQ at the benchmark's head layout
        (2, 8, 2, 9000, 16, 1, 8),    # more than one block's worth of tokens per row
        (2, 8, 4, 1200, 8, 2, 16),    # 16-wide groups, two stages, 2 query heads per KV head
        (1, 4, 4, 800, 2, 2, 64),     # two 64-wide groups, no head sharing
        (3, 12, 3, 257, 4, 1, 32),    # odd batch, 32-wide groups
        (2, 16, 4, 6000, 32, 1, 4),   # 32 groups of 4 (a lane's eight channels are two whole words)
        (1, 2, 2, 300, 32, 1, 4),     # ... without head sharing
    ],
)
def test_grouped_codebooks_of_one_and_two_stages_at_head_dim_128(device, b, hq, hkv, t, groups, stages, sub):
    """The kernel for at most 32 slots: groups of every width, ragged ranges, an empty row."""
    work = _workload(31 + t, b, hq, hkv, t, groups, stages, sub, [0.2] * stages if sub >= 32 else None)
    start = [(7 * i) % 50 for i in range(b)]
    end = [t - (11 * i) % 40 for i in range(b)]
    if b > 2:
        end[1] = start[1]  # an empty row
    out, state = _run(device, work, start, end, want_state=True)
    want, want_state = C.attention(*work, start, end)
    _check(out, want)
    live = [i for i in range(b) if end[i] > start[i]]
    _check_state(state.cpu()[live], want_state[live])
    if len(live) < b:
        dead = [i for i in range(b) if i not in live]
        assert bool((out.cpu()[dead] == 0).all()) and bool((state.cpu()[dead][..., 1:] == 0).all())


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub,order",
    [
        (1, 4, 1, 33000, 1, 1, 128, "random"),   # one slot, eight copies of the tables; bins folded because they could overflow
        (1, 2, 2, 2047, 1, 3, 128, "rising"),    # slots that are no power of two, the reference score grows in every segment
        (2, 8, 2, 4099, 1, 5, 128, "falling"),   # a first token far above the rest: small weights
        (1, 4, 2, 5000, 2, 4, 64, "rising"),     # eight slots
        (2, 4, 1, 1025, 4, 3, 32, "random"),     # twelve
        (1, 8, 2, 513, 8, 3, 16, "falling"),     # 24: two heads a block
        (3, 4, 2, 9001, 16, 2, 8, "rising"),     # 32, two query heads per KV head
        (9, 4, 2, 700, 32, 1, 4, "falling"),     # 4-wide words, a row per block
        (2, 8, 2, 6000, 1, 16, 128, "falling"),
    ],
)
def test_tables_of_up_to_32_slots(device, b, hq, hkv, t, groups, stages, sub, order):
    """Every rounding of the slot count, rows that end inside a segment, and scores in an order that moves the softmax reference."""
    q, kcodes, vcodes, ktab, vtab = _workload(t + stages, b, hq, hkv, t, groups, stages, sub, [0.3 * 0.8**s for s in range(stages)] if sub >= 16 else None)
    if order != "random":
        q = q * 3  # logits over a range of about ten
        for row in range(b):
            for h in range(hkv):
                score = torch.zeros(t)
                for s in range(stages):
                    for g in range(groups):
                        score += (ktab[h, s, g].float() @ q[row, h * (hq // hkv), g * sub : (g + 1) * sub].float())[kcodes[row, h, :, s, g].long()]
                kcodes[row, h] = kcodes[row, h, score.argsort(descending=order == "falling")]
    start, end = [5 * i for i in range(b)], [t - 3 * i for i in range(b)]
    work = (q, kcodes, vcodes, ktab, vtab)
    out, state = _run(device, work, start, end, want_state=True)
    want, want_state = C.attention(*work, start, end)
    _check(out, want)
    _check_state(state.cpu(), want_state)


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub",
    [
        (2, 8, 2, 700, 16, 1, 8),
        (2, 16, 4, 9000, 16, 1, 8),
        (1, 4, 2, 2000, 32, 1, 4),
        (2, 4, 2, 5000, 16, 2, 8),
        (1, 8, 8, 3000, 16, 2, 8),
        (1, 4, 2, 16384, 1, 2, 128),
        (1, 8, 8, 8192, 1, 16, 128),
        (2, 8, 2, 5000, 8, 3, 16),
        (1, 4, 1, 3000, 1, 20, 128),
    ],
)
def test_weights_have_the_precision_of_fp32(device, b, hq, hkv, t, groups, stages, sub):
    """The state of attention without a rotary step against 64 bits, for logits over a range of about 30.

    A weight is exp of an fp32 difference of at most 30 (2^-24 of it, 1.8e-6) by exp2 with two units in the last place (1.2e-7 each); the
    errors of different tokens are not alike, so a weighted mean has less than a single weight's.
    """
    gen = torch.Generator().manual_seed(t + stages)
    scales = [0.5 * 0.8**s for s in range(stages)] if sub <= 16 else [0.6 / stages**0.5] * stages
    ktab, vtab = (make_tables(gen, hkv, stages, groups, sub, scales) for _ in range(2))
    codes = [torch.randint(0, 256, (b, hkv, t, stages, groups), generator=gen, dtype=torch.uint8) for _ in range(2)]
    q = (4 * torch.randn(b, hq, 128, generator=gen) / 128**0.5).half()
    _, state = _run(device, (q, *codes, ktab, vtab), want_out=False, want_state=True)
    heads, at = torch.arange(hkv)[None, :, None, None], torch.arange(groups)
    rows = [sum(tab.double()[heads, s, at, c[:, :, :, s].long()] for s in range(stages)).flatten(3).repeat_interleave(hq // hkv, 1) for c, tab in zip(codes, (ktab, vtab))]
    score = torch.einsum("bhd,bhtd->bht", q.double(), rows[0])
    weight = score.softmax(-1)
    state = state.cpu().double()
    assert rel_l2(state[..., 2:] / state[..., 1:2], torch.einsum("bht,bhtd->bhd", weight, rows[1])) <= 1.5e-6
    torch.testing.assert_close(state[..., 0] + state[..., 1].log(), score.logsumexp(-1), rtol=0, atol=4e-6)

@pytest.mark.parametrize("t", [40, 3000])  # one block a row and head, several
@pytest.mark.parametrize(
    "hq,hkv,groups,stages,sub,rotary",
    [
        (8, 2, 16, 2, 8, False),
        (4, 2, 16, 2, 8, False),
        (8, 2, 1, 2, 128, False),
        (8, 2, 1, 16, 128, False),
        (2, 2, 32, 1, 4, False),
        (8, 2, 8, 2, 8, False),     # head_dim 64
        (16, 2, 8, 1, 16, False),   # eight query heads per KV head
        (8, 2, 16, 2, 8, True),
        (8, 2, 1, 16, 128, True),
        (8, 2, 1, 2, 128, True),
        (8, 2, 1, 3, 128, True),
    ],
)
def test_a_query_that_is_not_a_number_spoils_its_own_rows_only(device, hq, hkv, groups, stages, sub, rotary, t):
    ops = _ops()
    q, kcodes, vcodes, ktab, vtab = _workload(t, 3, hq, hkv, t, groups, stages, sub, [0.3 * 0.8**s for s in range(stages)] if sub >= 16 else None)
    start, end = [0, 0, 5], [t, t - 3, 5]
    rope = ops.rope_table(t, groups * sub, 1e6, device) if rotary else None
    want, _ = _run(device, (q, kcodes, vcodes, ktab, vtab), start, end, rope=rope)
    q[0, hq - 1, 7] = float("nan")
    q[1, 0] = float("nan")
    q[2, 1, 0] = float("nan")
    out, state = _run(device, (q, kcodes, vcodes, ktab, vtab), start, end, rope=rope, want_state=True)
    bad = torch.zeros(3, hq, dtype=torch.bool)
    bad[0, hq - 1] = bad[1, 0] = True
    out, state = out.cpu(), state.cpu()
    assert bool(out[bad].isnan().all()) and bool(state[..., 1][bad].isnan().all())
    _check(out[:2][~bad[:2]], want.cpu()[:2][~bad[:2]])
    assert bool((out[2] == 0).all()) and bool((state[2, :, 1] == 0).all())  # a row that sees nothing has no use for its query

def test_partial_states_merge_to_the_whole(device):
    """Sequence split as ranks would do it: per-range states, then the log-sum-exp merge."""
    ops = _ops()
    work = _workload(13, 2, 8, 2, 3000, 16, 2, 8)
    whole, _ = _run(device, work)
    states = []
    for lo, hi in ((0, 1000), (1000, 1000), (1000, 2200), (2200, 3000)):  # one empty range
        _, st = _run(device, work, [lo, lo], [hi, hi], want_out=False, want_state=True)
        states.append(st)
    merged_out, merged_state = ops.attn_combine(torch.stack(states), want_state=True)
    want, want_state = C.attention(*work)
    _check(merged_out, want)
    _check(whole, want)
    _check_state(merged_state.cpu(), want_state)
    c_out, _ = C.merge(torch.stack(states).cpu())
    _check(merged_out, c_out)


@pytest.mark.parametrize("parts", [1, 2, 7, 8, 9, 17, 64, 65, 200])
@pytest.mark.parametrize("dim", [32, 128, 256])
def test_merges_of_few_and_many_parts(device, parts, dim):
    """Both ways to merge, at their border; parts without a token, a row without any, one part of a row that is not a number."""
    ops = _ops()
    gen = torch.Generator().manual_seed(parts + dim)
    states = torch.randn(parts, 2, 5, dim + 2, generator=gen)
    states[..., 0] *= 20
    states[..., 1] = states[..., 1].abs() + 0.1
    empty = torch.rand(parts, 2, 5, generator=gen) < 0.3
    empty[:, 1, 4] = True
    empty[0, 0, 0] = False
    states[empty] = 0.0
    states[..., 0][empty] = -float("inf")
    out, merged = ops.attn_combine(states.to(device), want_state=True)
    want, want_merged = C.merge(states)
    torch.testing.assert_close(out.cpu().float(), want.float(), rtol=2e-3, atol=2e-3)
    torch.testing.assert_close(merged.cpu(), want_merged, rtol=2e-5, atol=2e-5)
    assert bool((out[1, 4] == 0).all()) and float(merged[1, 4, 1]) == 0
    states[parts // 2, 0, 0, 1] = float("nan")
    states[parts // 2, 0, 0, 0] = -float("inf")
    out, merged = ops.attn_combine(states.to(device), want_state=True)
    assert bool(out[0, 0].isnan().all()) and bool(merged[0, 0, 1].isnan())
    assert not bool(out[0, 1:].isnan().any()) and not bool(out[1].isnan().any())


def test_benchmark_size_32k_context(device):
    """Full benchmark shape: batch 8, 32 query / 8 KV heads, 32768 tokens, 2x16 code bytes per token."""
    work = _workload(8601, 8, 32, 8, 32768, 16, 2, 8)
    out, _ = _run(device, work)
    want, _ = C.attention(*work)
    _check(out, want)
    again, _ = _run(device, work)
    assert torch.equal(out, again)  # deterministic


def test_full_width_codebooks_at_the_all_layer_configuration(device):
    """Two additive 256 x 128 codebooks at batch 16, 32 query / 8 KV heads, 16384 tokens: one layer of the
    all-layer configuration (every (row, head) pair is one block that writes its result itself)."""
    work = _workload(8604, 16, 32, 8, 16384, 1, 2, 128, [0.1, 0.1])
    out, state = _run(device, work, want_state=True)
    want, want_state = C.attention(*work)
    _check(out, want)
    _check_state(state.cpu(), want_state)
    again, _ = _run(device, work)
    assert torch.equal(out, again)


def test_full_width_codebooks_split_ranges_and_deep_ladders(device):
    """Few pairs (several blocks per pair, merged afterwards), a ragged window, and the reference's own depth-16 ladder."""
    work = _workload(8605, 2, 8, 2, 9000, 1, 2, 128, [0.1, 0.1])
    out, _ = _run(device, work, [100, 0], [9000, 8500])
    want, _ = C.attention(*work, [100, 0], [9000, 8500])
    _check(out, want)
    work = _workload(8606, 3, 12, 3, 2100, 1, 16, 128, [0.1 * 0.7**s for s in range(16)])
    out, _ = _run(device, work, [0, 5, 2100], [2100, 1999, 2100])  # the last row is empty
    want, _ = C.attention(*work, [0, 5, 2100], [2100, 1999, 2100])
    _check(out, want)
    assert bool((out[2] == 0).all())


def test_sliding_window_launch_of_the_benchmark(device):
    """The benchmark's own window case: batch 8, the last 4096 of 32768 stored tokens visible."""
    work = _workload(8607, 8, 32, 8, 32768, 16, 2, 8)
    start, end = [32768 - 4096] * 8, [32768] * 8
    out, _ = _run(device, work, start, end)
    want, _ = C.attention(*work, start, end)
    _check(out, want)


def test_attention_argument_errors(device):
    from tac_vq_kv_cache_b200 import _lib

    ops = _ops()
    work = [x.to(device) for x in _workload(1, 1, 4, 1, 64, 16, 2, 8)]
    with pytest.raises(_lib.TacvqError) as err:
        ops.attn_decode(*work, workspace=torch.empty(256, dtype=torch.uint8, device=device))
    assert err.value.status == -5
    with pytest.raises(ValueError):
        ops.attn_decode(work[0].float(), *work[1:])
    with pytest.raises(ValueError):
        ops.attn_decode(work[0][:, :3].contiguous(), *work[1:])  # 3 query heads over 1 KV head is fine? no: rep=3 unsupported


def test_very_large_batch_is_not_the_scans(device):
    """More than 1024 (row, head) pairs: the benchmark layout's scan steps aside (its per-pair tables would need > 64 MB)."""
    work = _workload(21, 300, 16, 4, 70, 16, 2, 8)
    out, _ = _run(device, work)
    want, _ = C.attention(*work)
    _check(out, want)


@pytest.mark.parametrize(
    "b,hq,hkv,t,groups,stages,sub,shift",
    [
        (2, 8, 2, 600, 1, 40, 128, 0),     # more than 32 slots
        (2, 16, 2, 600, 8, 2, 16, 0),      # eight query heads per KV head
        (2, 8, 2, 600, 16, 2, 8, 4),       # a query that does not start at a multiple of 16 bytes
        (3, 2, 2, 1500, 1, 2, 128, 1),
        (1, 2, 1, 900, 32, 2, 4, 0),       # 64 slots
    ],
)
def test_head_dim_128_calls_that_only_the_general_kernel_takes(device, b, hq, hkv, t, groups, stages, sub, shift):
    ops = _ops()
    q, *rest = _workload(t + stages, b, hq, hkv, t, groups, stages, sub, [0.5 / stages**0.5] * stages if sub >= 16 else None)
    start, end = [3 * i for i in range(b)], [t - 5 * i for i in range(b)]
    room = torch.zeros(q.numel() + shift, dtype=torch.float16, device=device)
    out, _ = ops.attn_decode(
        room[shift:].view(q.shape).copy_(q), *(x.to(device) for x in rest), torch.tensor(start, dtype=torch.int32, device=device), torch.tensor(end, dtype=torch.int32, device=device)
    )
    want, _ = C.attention(q, *rest, start, end)
    _check(out, want)
