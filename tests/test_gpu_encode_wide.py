"""GPU parity of the tensor-core encode of 64- and 128-wide groups, plain and whitened.

Row counts around the tile of 128, one and two tiles a block, blocks that walk over several tiles with resident tables
(up to two stages) and with the ring (an odd and an even number of stages), small codebooks, ties, and rows that are near
several words at once.  Codes and rows are bit-exact with the C oracle.
"""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from tests.util import make_states, make_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "batch,heads,tokens,sub,groups,stages,words,dtype,whitened",
    [
        (1, 2, 257, 128, 1, 2, 256, torch.float16, False),
        (1, 2, 385, 128, 1, 1, 256, torch.float32, False),
        (2, 2, 191, 64, 2, 3, 100, torch.float16, False),
        (1, 40, 1025, 128, 1, 2, 256, torch.float16, False),   # 360 tiles: two a block, several trips, resident tables
        (1, 80, 641, 64, 2, 3, 256, torch.float16, False),     # the same through the ring of tables
        (3, 100, 299, 128, 1, 4, 33, torch.float32, False),
        (1, 2, 1, 128, 1, 16, 256, torch.float16, True),
        (1, 2, 129, 64, 2, 2, 77, torch.float16, True),
        (1, 90, 513, 128, 1, 3, 256, torch.float32, True),
    ],
)
def test_wide_encode_is_bit_exact(device, batch, heads, tokens, sub, groups, stages, words, dtype, whitened):
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(sub + tokens)
    tables = make_tables(gen, heads, stages, groups, sub, [0.1 * 0.9**s for s in range(stages)])[:, :, :, :words].contiguous()
    if words > 8:
        tables[:, :, :, 5] = tables[:, :, :, 3]  # a tie: the lower index wins
    states = make_states(gen, (batch, heads, tokens, sub * groups), dtype, 4)
    cache = torch.full((batch, heads, tokens + 3, stages, groups), 0xEE, dtype=torch.uint8, device=device)
    if whitened:
        w = torch.eye(sub).expand(heads, groups, sub, sub) + 0.3 * torch.randn(heads, groups, sub, sub, generator=gen) / sub**0.5
        want, want_recon = C.encode_whitened(states, tables, w)
        codes, recon = ops.encode(states.to(device), tables.to(device), codes=cache, t0=2, whitener=w.to(device))
    else:
        want, want_recon = C.encode(states, tables)
        codes, recon = ops.encode(states.to(device), tables.to(device), codes=cache, t0=2)
    assert torch.equal(codes[:, :, 2 : 2 + tokens].cpu(), want)
    assert torch.equal(recon.cpu(), want_recon)
    assert bool((codes[:, :, :2] == 0xEE).all()) and bool((codes[:, :, 2 + tokens :] == 0xEE).all())
    assert ops.encode_tensor_memory_timeouts(device) == 0


@pytest.mark.parametrize("sub,groups,heads,tokens", [(128, 1, 2, 1), (128, 1, 3, 127), (128, 1, 60, 645), (64, 2, 2, 129), (64, 2, 40, 647)])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_fp32_rows_at_any_alignment(device, sub, groups, heads, tokens, shift):
    """Rows that are fetched together, 16 bytes a lane, and rows that start elsewhere; heads and tokens exchanged, with a gap between rows."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(sub + tokens)
    tables = make_tables(gen, heads, 2, groups, sub, [0.1, 0.08])
    states = make_states(gen, (2, heads, tokens, sub * groups), torch.float32, 4)
    room = torch.full((2, tokens, heads, sub * groups + 8), float("nan"), device=device)
    x = room[..., shift : shift + sub * groups].transpose(1, 2)
    x.copy_(states)
    want, want_recon = C.encode(states, tables)
    codes, recon = ops.encode(x, tables.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)


@pytest.mark.parametrize("sub,groups", [(128, 1), (64, 2), (32, 4)])
@pytest.mark.parametrize("batch,tokens,words,shift,dtype", [(1, 1, 256, 0, torch.float16), (1, 129, 256, 1, torch.float32), (1, 601, 99, 0, torch.float32), (3, 333, 256, 0, torch.float16), (1, 1500, 256, 1, torch.float16), (1, 2049, 256, 0, torch.float16)])
def test_whitener_at_every_tile_height(device, sub, groups, batch, tokens, words, shift, dtype):
    """One bit of a transformed row or word shows in the codes: four to eight rows a thread, ragged tiles, rows of several batch entries."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(sub + tokens)
    heads = 20
    tables = make_tables(gen, heads, 1, groups, sub, [0.1])[:, :, :, :words].contiguous()
    states = make_states(gen, (batch, heads, tokens, sub * groups), dtype)
    w = torch.eye(sub).expand(heads, groups, sub, sub) + 0.3 * torch.randn(heads, groups, sub, sub, generator=gen) / sub**0.5
    x = torch.zeros(batch, tokens, heads, sub * groups + 8, dtype=dtype, device=device)[..., shift : shift + sub * groups].transpose(1, 2)
    x.copy_(states)
    want, want_recon = C.encode_whitened(states, tables, w)
    codes, recon = ops.encode(x, tables.to(device), whitener=w.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)


def test_rows_between_words_take_the_exact_chains(device):
    """Every row lies on a bisector of two words, or at a word that occurs three times: nothing but the exact order decides."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(3)
    tables = make_tables(gen, 2, 2, 1, 128, [0.1, 0.1])
    tables[:, :, :, 200] = tables[:, :, :, 100] = tables[:, :, :, 7]
    pick = torch.randint(0, 256, (2, 2, 260), generator=gen)
    rows = torch.stack([(tables[h, 0, 0][pick[h, 0]].float() + tables[h, 0, 0][pick[h, 1]].float()) / 2 for h in range(2)])
    rows[:, ::9] = tables[:, 0, 0, 7, None].float()
    states = rows[None]
    want, want_recon = C.encode(states, tables)
    codes, recon = ops.encode(states.to(device), tables.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)


@pytest.mark.parametrize("sub,groups,tokens,dtype,whitened", [(128, 1, 300, torch.float16, False), (64, 2, 129, torch.float32, False), (128, 1, 260, torch.float16, True), (128, 1, 9500, torch.float32, False)])
@pytest.mark.parametrize("alike", [(3, 70, 200), (5, 6, 200), (8, 9, 10), (3, 70, 140, 250)])
def test_rows_near_three_words(device, sub, groups, tokens, dtype, whitened, alike):
    """Words that differ by a few units of their last place: in three shares of the table, in two, in one (which tells of two), and four of them."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(tokens + len(alike))
    tables = make_tables(gen, 2, 2, groups, sub, [0.1, 0.1])
    for i, k in enumerate(alike):
        apart = (1e-4, 4e-4, 4e-5, 2e-4)[i] * torch.randn(2, groups, sub, generator=gen)
        tables[:, 0, :, k] = (tables[:, 0, :, alike[0]].float() + apart).half()
    states = 10.0 * tables[:, 0, :, alike[0]].float().reshape(1, 2, 1, groups * sub) + 0.5 * torch.randn(1, 2, tokens, groups * sub, generator=gen)
    states[:, :, ::3] = torch.randn(1, 2, (tokens + 2) // 3, groups * sub, generator=gen)
    states = states.to(dtype)
    if whitened:
        w = torch.eye(sub).expand(2, groups, sub, sub) + 0.05 * torch.randn(2, groups, sub, sub, generator=gen) / sub**0.5
        want, want_recon = C.encode_whitened(states, tables, w)
        codes, recon = ops.encode(states.to(device), tables.to(device), whitener=w.to(device))
    else:
        want, want_recon = C.encode(states, tables)
        codes, recon = ops.encode(states.to(device), tables.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)


@pytest.mark.parametrize("tokens", [1, 8, 9, 40, 41, 136, 137, 300])
def test_whitened_words_of_few_and_of_many_rows(device, tokens):
    """Chosen words are fetched row by row where at most eight of 32 neighbouring rows exist, by whole lines otherwise."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(tokens)
    tables = make_tables(gen, 3, 4, 1, 128, [0.1 * 0.9**s for s in range(4)])
    w = torch.eye(128).expand(3, 1, 128, 128) + 0.3 * torch.randn(3, 1, 128, 128, generator=gen) / 128**0.5
    for dtype in (torch.float16, torch.float32):
        states = torch.randn(1, 3, tokens, 128, generator=gen).to(dtype)
        want, want_recon = C.encode_whitened(states, tables, w)
        codes, recon = ops.encode(states.to(device), tables.to(device), whitener=w.to(device))
        assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)
