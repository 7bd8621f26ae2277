"""GPU test of the preallocated code store: in-place append, the window rule and attention over it."""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from tests.util import make_states, make_tables, max_rel, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [96, None])
def test_prefill_then_decode_steps_match_the_oracle(device, window):
    """The visible range changes at every step - a sliding window of 96, or all stored tokens with the length
    crossing a 32-token tile edge at 128 - and the fused single call (fp16 and fp32 rows) alternates with the two-call route."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(8601)
    batch, heads, q_heads, dim = 2, 2, 8, 128
    ktab, vtab = make_tables(gen, heads, 2, 16, 8), make_tables(gen, heads, 2, 16, 8)
    cache = VQCodeCache(ktab.float(), vtab.float(), batch=batch, max_tokens=160, window=window, device=device)
    keys = make_states(gen, (batch, heads, 130, dim), outlier_channels=4)
    values = make_states(gen, (batch, heads, 130, dim))
    want_k, want_krec = C.encode(keys, ktab)
    want_v, _ = C.encode(values, vtab, want_recon=False)

    krec, vrec = cache.append(keys[:, :, :100].to(device), values[:, :, :100].to(device), want_recon=True)
    assert torch.equal(krec.cpu(), want_krec[:, :, :100])
    assert cache.length == 100 and cache.visible() == ((4, 100) if window else (0, 100))
    assert cache.payload_bytes() == 2 * batch * heads * 100 * 32
    for step in range(100, 130):  # token by token, as a decode loop does
        query = (torch.randn(batch, q_heads, dim, generator=gen) / dim**0.5).half()
        k_new, v_new = keys[:, :, step : step + 1].contiguous().to(device), values[:, :, step : step + 1].contiguous().to(device)
        if step % 2:  # both routes: two calls, or the fused single call
            cache.append(k_new, v_new)
            out = cache.attend(query.to(device))
        elif step % 4:  # fp32 rows (the same values) take the same route and give the same codes
            out = cache.decode_step(query.to(device), k_new.float(), v_new.float())
        else:
            out = cache.decode_step(query.to(device), k_new, v_new)
        start, end = cache.visible()
        assert (start, end) == ((step + 1 - window) if window else 0, step + 1)
        want, _ = C.attention(query, want_k[:, :, : step + 1].contiguous(), want_v[:, :, : step + 1].contiguous(), ktab, vtab,
                              [start] * batch, [end] * batch)
        assert rel_l2(out, want) <= 2e-3 and max_rel(out, want) <= 2e-3, (step, rel_l2(out, want))
    assert torch.equal(cache.key[:, :, :130].cpu(), want_k) and torch.equal(cache.value[:, :, :130].cpu(), want_v)
    with pytest.raises(ValueError):
        cache.append(keys[:, :, :40].to(device), values[:, :, :40].to(device))  # 130 + 40 > 160
    cache.reset()
    assert cache.length == 0 and cache.payload_bytes() == 0


@pytest.mark.parametrize("direct", [False, True, "rows"], ids=["copies", "result-in-place", "rows-and-result-in-place"])
def test_single_call_host_step_equals_the_device_step(device, direct):
    """tacvq_decode_step_host (rows from pinned host memory, result back to host, one call) gives the same
    codes and the same attention result as decode_step on device tensors, both with enqueued copies and with the
    kernels reading and writing the pinned buffers in place."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(8603)
    batch, heads, q_heads, dim = 2, 2, 8, 128
    ktab, vtab = make_tables(gen, heads, 2, 16, 8), make_tables(gen, heads, 2, 16, 8)
    a = VQCodeCache(ktab.float(), vtab.float(), batch=batch, max_tokens=96, window=64, device=device)
    b = VQCodeCache(ktab.float(), vtab.float(), batch=batch, max_tokens=96, window=64, device=device)
    keys, values = make_states(gen, (batch, heads, 90, dim)), make_states(gen, (batch, heads, 90, dim))
    a.append(keys[:, :, :60].to(device), values[:, :, :60].to(device))
    b.append(keys[:, :, :60].to(device), values[:, :, :60].to(device))
    nq, nkv = batch * q_heads * dim, batch * heads * dim
    host_rows = torch.empty(nq + 2 * nkv, dtype=torch.float16).pin_memory()
    host_out = torch.empty(batch, q_heads, dim, dtype=torch.float16).pin_memory()
    for step in range(60, 90):
        query = (torch.randn(batch, q_heads, dim, generator=gen) / dim**0.5).half()
        k_new, v_new = keys[:, :, step : step + 1].contiguous(), values[:, :, step : step + 1].contiguous()
        host_rows[:nq].copy_(query.reshape(-1))
        host_rows[nq : nq + nkv].copy_(k_new.reshape(-1))
        host_rows[nq + nkv :].copy_(v_new.reshape(-1))
        got = a.decode_step_host(host_rows, host_out, q_heads, direct=direct)
        want = b.decode_step(query.to(device), k_new.to(device), v_new.to(device))
        assert torch.equal(got, want.cpu()), step
    assert a.length == b.length == 90 and torch.equal(a.key, b.key) and torch.equal(a.value, b.value)
    with pytest.raises(ValueError):
        a.decode_step_host(host_rows[:-1], host_out, q_heads, direct=direct)


def _decoding_pair(gen, device, groups, stages, sub, rope, batch=2, heads=2, prompt=50):
    """A cache that is stepped and one that appends and attends, after the same prompt, and a source of step inputs."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    tables = [make_tables(gen, heads, stages, groups, sub, [0.1 * 0.9**s for s in range(stages)]) for _ in range(2)]
    pair = [VQCodeCache(*tables, batch=batch, max_tokens=80, window=32, device=device, rope_theta=rope) for _ in range(2)]
    rows = [make_states(gen, (batch, heads, prompt, groups * sub)).to(device) for _ in range(2)]
    for cache in pair:
        cache.append(*rows)

    def inputs():
        query = (torch.randn(batch, 8, groups * sub, generator=gen) / (groups * sub) ** 0.5).half().to(device)
        return query, *(make_states(gen, (batch, heads, 1, groups * sub)).to(device) for _ in range(2))

    return (*pair, inputs)


def _step_equals_append_and_attend(stepped, plain, query, key, value):
    out = stepped.decode_step(query, key, value)
    plain.append(key, value)
    want = plain.attend(query)
    assert rel_l2(out, want) <= 1e-3
    assert torch.equal(stepped.key, plain.key) and torch.equal(stepped.value, plain.value)
    assert rel_l2(stepped.attend(query), want) <= 1e-3  # and the range left on the device is the one that was seen


@pytest.mark.parametrize("rope", [None, 1e6])
@pytest.mark.parametrize(
    "batch,heads,q_heads,groups,stages,sub,tokens,window",
    [
        (4, 2, 8, 16, 2, 8, 5000, 700),
        (3, 2, 4, 16, 2, 8, 5000, None),
        (1, 2, 8, 1, 16, 128, 9000, 900),
        (5, 2, 8, 1, 2, 128, 4000, 600),
        (2, 4, 8, 16, 1, 8, 6000, 1500),
        (2, 2, 8, 2, 3, 64, 3000, 100),
    ],
)
def test_a_step_equals_append_and_attend_bit_for_bit(device, batch, heads, q_heads, groups, stages, sub, tokens, window, rope):
    """However little of the buffer is visible; also while it fills, and after a captured call of either kind."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(tokens + stages)
    tables = [make_tables(gen, heads, stages, groups, sub, [0.3 * 0.8**s for s in range(stages)] if sub >= 16 else None) for _ in range(2)]
    pair = [VQCodeCache(*tables, batch=batch, max_tokens=tokens, window=window, device=device, rope_theta=rope) for _ in range(2)]
    codes = [torch.randint(0, 256, pair[0].key.shape, generator=gen, dtype=torch.uint8) for _ in range(2)]
    for cache in pair:
        cache.key.copy_(codes[0]), cache.value.copy_(codes[1])
    for length in (1, 250, tokens // 2, tokens - 1):
        query = (2 * torch.randn(batch, q_heads, 128, generator=gen) / 128**0.5).half().to(device)
        rows = [make_states(gen, (batch, heads, 1, 128)).to(device) for _ in range(2)]
        for cache in pair:
            cache.length = length
        out = pair[0].decode_step(query, *rows)
        pair[1].append(*rows)
        want = pair[1].attend(query)
        assert torch.equal(out, want), (length, rel_l2(out, want))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = pair[1].attend(query)
        graph.replay()
        assert rel_l2(captured, want) <= 1e-3


@pytest.mark.parametrize("rope", [None, 1e6])
@pytest.mark.parametrize("groups,stages,sub,q_heads", [(16, 2, 8, 8), (16, 2, 8, 2), (1, 2, 128, 8), (1, 16, 128, 8), (16, 1, 8, 8), (32, 1, 4, 8), (2, 3, 64, 8)])
def test_three_steps_in_one_graph_equal_three_steps(device, groups, stages, sub, q_heads, rope):
    """A step's first launch may start before what computes its rows has ended, in a graph too: there behind a copy on another
    stream, a product and the step before.  The graph is replayed on other inputs, over codes that are not the new ones."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(groups + stages)
    batch, heads, tokens = 3, 2, 500
    tables = [make_tables(gen, heads, stages, groups, sub, [0.3 * 0.8**s for s in range(stages)] if sub >= 16 else None) for _ in range(2)]
    plain, captured = (VQCodeCache(*tables, batch=batch, max_tokens=tokens, window=300, device=device, rope_theta=rope) for _ in range(2))
    codes = [torch.randint(0, 256, plain.key.shape, generator=gen, dtype=torch.uint8).to(device) for _ in range(2)]
    turn = (torch.randn(128, 128, generator=gen) / 128**0.5).half().to(device)
    source = [torch.zeros(3, batch, n, 128, dtype=torch.float16, device=device) for n in (q_heads, heads, heads)]
    landed = [torch.zeros_like(x) for x in source]

    def three(cache):
        cache.key.copy_(codes[0]), cache.value.copy_(codes[1])
        cache.length = 400
        here, aside = torch.cuda.current_stream(), torch.cuda.Stream()
        aside.wait_stream(here)
        with torch.cuda.stream(aside):
            for to, x in zip(landed, source):
                to.copy_(x)
        here.wait_stream(aside)
        return [cache.decode_step(*(x[i] @ turn if j == 0 else (x[i] @ turn)[:, :, None] for j, x in enumerate(landed))) for i in range(3)]

    def renew():
        for x in source:
            x.copy_(torch.randn(x.shape, generator=gen) * (0.2 if x is source[0] else 1.0))

    renew()
    three(captured)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = three(captured)
    for _ in range(3):
        renew()
        want = three(plain)
        graph.replay()
        for i, (out, expected) in enumerate(zip(got, want)):
            assert torch.equal(out, expected), (i, rel_l2(out, expected))
        assert torch.equal(captured.key, plain.key) and torch.equal(captured.value, plain.value) and captured.length == plain.length == 403
        assert not torch.equal(plain.key[:, :, 400:403], codes[0][:, :, 400:403])


@pytest.mark.parametrize("rope", [None, 1e6])
@pytest.mark.parametrize("groups,stages,sub", [(16, 2, 8), (1, 2, 128)])
def test_a_step_uses_the_buffers_tables_and_window_that_the_cache_has_now(device, groups, stages, sub, rope):
    gen = torch.Generator().manual_seed(8611)
    stepped, plain, inputs = _decoding_pair(gen, device, groups, stages, sub, rope)
    _step_equals_append_and_attend(stepped, plain, *inputs())
    for cache in (stepped, plain):
        cache.window = 8
    _step_equals_append_and_attend(stepped, plain, *inputs())
    for cache in (stepped, plain):
        cache.window = None
    left = stepped.key
    before = left.clone()
    for cache in (stepped, plain):  # sequences change places, as in a beam search
        cache.key, cache.value = cache.key.flip(0).contiguous(), cache.value.flip(0).contiguous()
    _step_equals_append_and_attend(stepped, plain, *inputs())
    assert torch.equal(left, before)
    tables = [make_tables(gen, 2, stages, groups, sub, [0.2 * 0.9**s for s in range(stages)]).to(device) for _ in range(2)]
    for cache in (stepped, plain):  # tables after a training step
        cache.key_tables, cache.value_tables = tables[0].clone(), tables[1].clone()
    _step_equals_append_and_attend(stepped, plain, *inputs())
    length = stepped.length
    for name, wrong in (("key", stepped.key[:, :, :-1]), ("value", stepped.value.to(torch.int16)), ("key_tables", stepped.key_tables[:, :, :, :, : sub // 2]),
                        ("value_tables", stepped.value_tables.float())):
        kept = getattr(stepped, name)
        setattr(stepped, name, wrong)
        with pytest.raises(ValueError):
            stepped.decode_step(*inputs())
        setattr(stepped, name, kept)
    assert stepped.length == length


@pytest.mark.parametrize("duplicate", ["copy", "deepcopy", "pickle"])
@pytest.mark.parametrize("groups,stages,sub", [(16, 2, 8), (1, 2, 128)])
def test_a_copied_cache_steps_on_its_own_buffers(device, groups, stages, sub, duplicate):
    import copy
    import pickle

    gen = torch.Generator().manual_seed(8612)
    stepped, plain, inputs = _decoding_pair(gen, device, groups, stages, sub, None)
    _step_equals_append_and_attend(stepped, plain, *inputs())
    fork = {"copy": copy.copy, "deepcopy": copy.deepcopy, "pickle": lambda cache: pickle.loads(pickle.dumps(cache))}[duplicate](stepped)
    other = copy.deepcopy(plain)
    if duplicate == "copy":
        fork.key, fork.value = fork.key.clone(), fork.value.clone()
    for _ in range(2):  # the fork runs ahead; the original goes on from where it was
        _step_equals_append_and_attend(fork, other, *inputs())
    assert torch.equal(stepped.key, plain.key) and torch.equal(stepped.value, plain.value)
    query, _, _ = inputs()
    assert rel_l2(stepped.attend(query), plain.attend(query)) <= 1e-3
    _step_equals_append_and_attend(stepped, plain, *inputs())


def test_a_rotary_cache_takes_the_rows_that_append_takes(device):
    """Rows of a [B,T,H,D] projection seen as [B,H,T,D], rows and queries cut out of one fused buffer, K and V of different
    types, rows at odd addresses, no new token; results copied to another type, to strided memory and over the query."""
    gen = torch.Generator().manual_seed(8613)
    stepped, plain, inputs = _decoding_pair(gen, device, 1, 3, 128, 1e6)

    def projected(tokens):
        return make_states(gen, (2, tokens, 2, 128)).to(device).transpose(1, 2)

    fused = make_states(gen, (2, 1, 8 + 2 + 2, 128)).to(device) / 4  # heads of q, k, v side by side
    query, key, value = inputs()
    shifted = torch.empty(key.numel() + 1, dtype=key.dtype, device=device)[1:].view(key.shape).copy_(key)
    for case in (
        (query, projected(3), projected(3)),
        (fused[:, 0, :8], fused[:, :, 8:10].transpose(1, 2), fused[:, :, 10:].transpose(1, 2)),
        (query, key, value.float()),
        (query, shifted, shifted),
        (query, key[:, :, :0], value[:, :, :0]),
    ):
        _step_equals_append_and_attend(stepped, plain, *case)
    for cache in (stepped, plain):
        cache.key_tables = cache.key_tables.transpose(3, 4).contiguous().transpose(3, 4)
    _step_equals_append_and_attend(stepped, plain, query, key, value)
    wide = torch.zeros(2, 8, 256, dtype=torch.float16, device=device)
    for out in (torch.empty(2, 8, 128, device=device), wide[:, :, ::2], torch.empty_like(query), query.clone()):
        case = (out if out.dtype == torch.float16 and torch.equal(out, query) else query, key, value)
        before = case[0].clone()
        got = stepped.decode_step(*case, out=out)
        plain.append(key, value)
        assert got is out and torch.equal(got.half(), plain.attend(before))
    assert torch.equal(stepped.key, plain.key) and bool((wide[:, :, 1::2] == 0).all())


def test_a_host_step_uses_the_buffers_tables_and_window_that_the_cache_has_now(device):
    gen = torch.Generator().manual_seed(8614)
    stepped, plain, inputs = _decoding_pair(gen, device, 16, 2, 8, None)
    host_rows = torch.empty(2 * 8 * 128 + 2 * 2 * 2 * 128, dtype=torch.float16).pin_memory()
    host_out = torch.empty(2, 8, 128, dtype=torch.float16).pin_memory()

    def step():
        query, key, value = inputs()
        host_rows.copy_(torch.cat([query.flatten(), key.flatten(), value.flatten()]))
        torch.cuda.synchronize()
        stepped.decode_step_host(host_rows, host_out, 8)
        plain.append(key, value)
        want = plain.attend(query)
        assert rel_l2(host_out, want) <= 1e-3 and rel_l2(stepped.attend(query), want) <= 1e-3
        assert torch.equal(stepped.key, plain.key) and torch.equal(stepped.value, plain.value)

    step()
    for cache in (stepped, plain):
        cache.window = 8
    step()
    left, before = stepped.key, stepped.key.clone()
    for cache in (stepped, plain):
        cache.window = None
        cache.key, cache.value = cache.key.flip(0).contiguous(), cache.value.flip(0).contiguous()
    step()
    assert torch.equal(left, before)
    tables = [make_tables(gen, 2, 2, 16, 8, [0.2, 0.1]).to(device) for _ in range(2)]
    for cache in (stepped, plain):
        cache.key_tables, cache.value_tables = tables[0].clone(), tables[1].clone()
    step()


def test_a_result_may_be_the_next_steps_query(device):
    """Nothing runs between the steps: the second one's table preparation follows the first one's attention directly."""
    from tac_vq_kv_cache_b200.code_cache import VQCodeCache

    gen = torch.Generator().manual_seed(8615)
    tables = [make_tables(gen, 2, 2, 16, 8) for _ in range(2)]
    caches = [VQCodeCache(*tables, batch=2, max_tokens=4200, device=device) for _ in range(2)]
    prompt = [make_states(gen, (2, 2, 4096, 128)).to(device) for _ in range(2)]
    rows = [[make_states(gen, (2, 2, 1, 128)).to(device) for _ in range(2)] for _ in range(60)]
    first = (torch.randn(2, 8, 128, generator=gen) / 128**0.5).half().to(device)
    results = []
    for cache, alone in zip(caches, (False, True)):
        cache.append(*prompt)
        query, outs = first, [torch.empty_like(first) for _ in rows]
        for out, (key, value) in zip(outs, rows):
            torch.cuda.synchronize() if alone else None
            query = cache.decode_step(query, key, value, out=out)
        results.append(torch.stack(outs))
    assert torch.equal(*results)
