"""The launches that the profile summaries of single kernels are about, one after the other, on seeded inputs of 8 heads x 128."""

from __future__ import annotations

import sys

import torch

from tac_vq_kv_cache_b200 import ops
from tac_vq_kv_cache_b200.code_cache import VQCodeCache

HEADS, DIM, WORDS = 8, 128, 256


def tables(gen, stages, groups):
    return (torch.randn(HEADS, stages, groups, WORDS, DIM // groups, device="cuda", generator=gen) * 0.3).half()


def rows(gen, batch, tokens, dtype=torch.float16):
    return torch.randn(batch, HEADS, tokens, DIM, device="cuda", generator=gen).to(dtype)


def encodes(gen):
    ops.encode(rows(gen, 4, 8192), tables(gen, 2, 16))
    ops.encode(rows(gen, 4, 8192), tables(gen, 2, 1))
    ops.encode(rows(gen, 1, 2048), tables(gen, 16, 1))
    ops.encode(rows(gen, 1, 1), tables(gen, 16, 1))
    codes = torch.randint(0, 256, (2, HEADS, 32768, 2, 16), device="cuda", generator=gen, dtype=torch.uint8)
    ops.decode(codes, tables(gen, 2, 16))


def whitened(gen):
    """Wide whitening and search of a 16-stage ladder, narrow search of 32 groups of 4."""
    for stages, groups, tokens, dtype in ((16, 1, 2048, torch.float16), (1, 32, 3001, torch.float32)):
        width = DIM // groups
        matrix = torch.eye(width, device="cuda").expand(HEADS, groups, width, width)
        matrix = matrix + 0.3 * torch.randn(HEADS, groups, width, width, device="cuda", generator=gen) / width**0.5
        ops.encode(rows(gen, 1, tokens, dtype), tables(gen, stages, groups), whitener=matrix)


def steps(gen):
    """Decode steps: a rotary ladder of 16 stages and the rotary benchmark layout; attention over slots."""
    for stages, groups, batch, tokens, window, theta in ((16, 1, 1, 6144, 4096, 1e6), (2, 16, 8, 32768, None, 1e6), (1, 16, 8, 32768, None, None)):
        cache = VQCodeCache(tables(gen, stages, groups), tables(gen, stages, groups), batch=batch, max_tokens=tokens, window=window, device="cuda", rope_theta=theta)
        for side in (cache.key, cache.value):
            side.random_(0, 256, generator=gen)
        cache.length = tokens - 1
        query = (torch.randn(batch, 4 * HEADS, DIM, device="cuda", generator=gen) / DIM**0.5).half()
        cache.decode_step(query, rows(gen, batch, 1), rows(gen, batch, 1))


if __name__ == "__main__":
    generator = torch.Generator(device="cuda").manual_seed(1)
    for name in sys.argv[1:] or ("encodes", "whitened", "steps"):
        {"encodes": encodes, "whitened": whitened, "steps": steps}[name](generator)
        torch.cuda.synchronize()
