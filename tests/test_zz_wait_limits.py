"""Encode kernels whose waits run out: the slower routes give the same codes and rows, and the blocks concerned are counted.

Runs after the tests that expect the count to be 0.
"""

from __future__ import annotations

import pytest
import torch

from oracle import c_oracle as C
from tests.util import make_states, make_tables

pytestmark = pytest.mark.gpu


def _encode(device, states, tables, spins, norms=None, whitener=None):
    from tac_vq_kv_cache_b200 import _lib, ops

    b, h, t, dim = states.shape
    s, g, k, d = tables.shape[1:]
    x, tab = states.to(device), tables.to(device)
    codes = torch.full((b, h, t, s, g), 0xEE, dtype=torch.uint8, device=device)
    recon = torch.empty_like(x)
    w = None if whitener is None else whitener.to(device)
    search_tables, search_rows = torch.empty(tab.shape, device=device), torch.empty(x.shape, device=device)
    need = ops._whitened_filter_bytes(h, dim, g, s, k)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device=device)
    status = _lib.load().tacvq_encode_wait_limited(
        x.data_ptr(), ops._DTYPE_TAG[x.dtype], *x.stride()[:3], tab.data_ptr(), ops._ptr(norms), ops._ptr(w), search_tables.data_ptr(),
        search_rows.data_ptr(), scratch.data_ptr(), need, codes.data_ptr(), recon.data_ptr(), ops._DTYPE_TAG[x.dtype], b, h, t, dim, g, s, k,
        0, t, spins, ops._stream(x.device),
    )
    _lib.check("tacvq_encode_wait_limited", status)
    torch.cuda.synchronize()
    return codes.cpu(), recon.cpu()


@pytest.mark.parametrize("spins", [0, 1, 3, 1 << 17])
@pytest.mark.parametrize(
    "heads,tokens,sub,groups,stages,words,norms,whitened",
    [
        (2, 300, 128, 1, 2, 256, False, False),    # one tile a block, resident tables
        (2, 300, 128, 1, 5, 200, True, False),     # the ring
        (100, 300, 64, 2, 5, 256, False, False),   # two tiles a block, several trips, the ring
        (60, 300, 128, 1, 4, 256, True, False),
        (2, 200, 64, 2, 3, 100, False, True),
        (60, 300, 128, 1, 4, 256, False, True),
        (2, 3, 128, 1, 7, 256, False, False),      # few rows
        (2, 5, 32, 4, 2, 256, True, False),
        (4, 1700, 8, 16, 2, 256, False, False),    # narrow groups, many rows
        (4, 1700, 4, 32, 1, 100, True, False),
        (2, 33, 8, 16, 2, 256, False, True),       # ... and fp32 words, whole pairs a block
        (4, 1700, 8, 16, 3, 200, False, True),
        (3, 700, 4, 32, 1, 256, False, True),
    ],
)
def test_codes_do_not_depend_on_waits_that_run_out(device, heads, tokens, sub, groups, stages, words, norms, whitened, spins):
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(sub + tokens)
    tables = make_tables(gen, heads, stages, groups, sub, [0.3 * 0.8**s for s in range(stages)])[:, :, :, :words].contiguous()
    states = make_states(gen, (1, heads, tokens, sub * groups))
    w = torch.eye(sub).expand(heads, groups, sub, sub) + 0.3 * torch.randn(heads, groups, sub, sub, generator=gen) / sub**0.5 if whitened else None
    want, want_recon = C.encode_whitened(states, tables, w) if whitened else C.encode(states, tables)
    before = ops.encode_tensor_memory_timeouts(device)
    for _ in range(4 if 0 < spins < 1 << 17 else 1):  # which waits run out differs from launch to launch
        codes, recon = _encode(device, states, tables, spins, ops.table_sqnorm(tables.to(device)) if norms else None, w)
        assert torch.equal(codes, want) and torch.equal(recon, want_recon)
    after = ops.encode_tensor_memory_timeouts(device)
    assert after > before if spins == 0 else after >= before if spins < 1 << 17 else after == before


@pytest.mark.parametrize("whitened", [False, True])
def test_a_tile_of_rows_that_need_every_word_beside_ordinary_ones(device, whitened):
    """Two tiles a block through the ring of tables, one of them far slower: the quick one neither overtakes it nor gives up."""
    from tac_vq_kv_cache_b200 import ops

    gen = torch.Generator().manual_seed(11)
    heads, stages = 90, 4
    tables = make_tables(gen, heads, stages, 1, 128, [0.3 * 0.8**s for s in range(stages)])
    states = make_states(gen, (1, heads, 256, 128))
    states[:, :, :128] = (make_states(gen, (1, heads, 128, 128)).float() * 4000).half()  # |r|^2 above 1e9
    before = ops.encode_tensor_memory_timeouts(device)
    if whitened:
        w = torch.eye(128).expand(heads, 1, 128, 128) + 0.3 * torch.randn(heads, 1, 128, 128, generator=gen) / 128**0.5
        want, want_recon = C.encode_whitened(states, tables, w)
        codes, recon = ops.encode(states.to(device), tables.to(device), whitener=w.to(device))
    else:
        want, want_recon = C.encode(states, tables)
        codes, recon = ops.encode(states.to(device), tables.to(device))
    assert torch.equal(codes.cpu(), want) and torch.equal(recon.cpu(), want_recon)
    assert ops.encode_tensor_memory_timeouts(device) == before
