"""Which kernel the C ABI hands a call to, and what it makes of its status (CPU).

abi.cu is compiled by itself and linked with stand-ins for the kernels' launchers, which write down how they were called and
return what the test tells them to.
"""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "tac_vq_kv_cache_b200"

STAND_INS = r"""
#include <map>
#include <string>
#include "common.cuh"
#include "ladder_plan.cuh"
#include "narrow_plan.cuh"
namespace {
std::string calls;
std::map<std::string, int> told;  // status, or number of splits
int called(const char *name, long long a = -1, long long b = -1) {
    calls += std::string(name) + " " + std::to_string(a) + " " + std::to_string(b) + "\n";
    auto it = told.find(name);
    return it == told.end() ? 0 : it->second;
}
int splits_of(const char *name) { auto it = told.find(std::string(name) + ".splits"); return it == told.end() ? 3 : it->second; }
}
extern "C" __attribute__((visibility("default"))) const char *stand_in_calls() { return calls.c_str(); }
extern "C" __attribute__((visibility("default"))) void stand_in_reset() { calls.clear(); told.clear(); }
extern "C" __attribute__((visibility("default"))) void stand_in_tell(const char *name, int value) { told[name] = value; }
extern "C" __attribute__((visibility("default"))) int ladder_splits(int B, int Hq, int Hkv, int S, int64_t T_cap, int64_t visible) {
    return tacvq::ladder::plan(B, Hq, Hkv, S, T_cap, visible, 148, 15).splits;
}
extern "C" __attribute__((visibility("default"))) int narrow_pays(int64_t rows, int64_t pairs, int stages) { return tacvq::narrow::pays(rows, pairs, stages, 148); }
extern "C" __attribute__((visibility("default"))) void narrow_deal(int64_t tiles, int64_t pairs, int *out) {
    const tacvq::narrow::Deal dealt = tacvq::narrow::deal(tiles, pairs, 148);
    out[0] = dealt.blocks, out[1] = 1 << dealt.shift, out[2] = dealt.rounds, out[3] = dealt.visits;
}
namespace tacvq {
int encode_dispatch(const EncodeArgs &) { return called("encode"); }
int decode_dispatch(const uint8_t *, const __half *, void *, int, int, int, int, int, int, int, int, int, int64_t, int64_t, cudaStream_t) { return called("decode"); }
int codeword_grad_dispatch(const uint8_t *, const float *, float *, int, int, int, int, int, int, int, int, int64_t, int64_t, cudaStream_t) { return called("grad"); }
int table_sqnorm_dispatch(const __half *, float *, int64_t, int, cudaStream_t) { return called("sqnorm"); }
int tensor_memory_timeouts(unsigned int *) { return 0; }
int round_words_dispatch(const float *, __half *, float *, int64_t, int, cudaStream_t) { return called("round_words"); }
int whiten_dispatch(const void *, int, int64_t, int64_t, int64_t, const __half *, const float *, float *, float *, int, int, int, int, int, int, int, cudaStream_t) { return called("whiten"); }
int rope_table_dispatch(__half *, int64_t, int, double, int64_t, cudaStream_t) { return called("rope"); }
int decode_prologue_dispatch(const void *, const void *, int, int64_t, int64_t, int64_t, const __half *, const __half *, uint8_t *, uint8_t *, int32_t *,
                             int32_t *, int start, int end, int, int, int, int, int, int, int, int64_t, int64_t, cudaStream_t) { return called("prologue", start, end); }
int attn_generic_splits(int, int, int64_t, int) { return splits_of("generic"); }
int attn_generic_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const int32_t *, const int32_t *, float *, int,
                          int, int, int, int, int, int, int64_t, int, cudaStream_t) { return called("generic"); }
int attn_combine_dispatch(const float *, int n, __half *, float *, int64_t, int, cudaStream_t) { return called("combine", n); }
bool attn_slots_supported(int, int Hq, int Hkv, int D, int G, int S, int K) { return D == 128 && K == 256 && S * G <= 32 && Hq / Hkv <= 4; }
int attn_slots_splits(int, int, int, int, int, int64_t visible, int) { calls += "slots.plan " + std::to_string(visible) + "\n"; return splits_of("slots"); }
int attn_slots_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const int32_t *, const int32_t *, float *, __half *,
                        float *, int, int, int, int, int, int64_t, int splits, bool after, cudaStream_t) { return called("slots", splits, after); }
bool attn_gsrq_supported(int Hq, int Hkv, int D, int G, int S, int K) { return D == 128 && G == 16 && S == 2 && K == 256 && Hq == 4 * Hkv; }
size_t attn_gsrq_workspace_bytes(int, int, int, int, int) { return 0; }
int attn_gsrq_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const int32_t *, const int32_t *, void *, __half *,
                       float *, int, int, int, int64_t, int, cudaStream_t, const GsrqNewToken *) { return called("gsrq"); }
int attn_rotary_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const __half *, const int32_t *, const int32_t *,
                         float *, int, int, int, int, int, int, int, int64_t, int, cudaStream_t) { return called("rotary"); }
bool attn_rotary_staged_supported(int, int, int D, int G, int S, int) { return D == 128 && S <= 2 && D / G >= 4; }
int attn_rotary_staged_splits(int, int, int64_t, int) { return splits_of("staged"); }
int attn_rotary_staged_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const __half *, const int32_t *,
                                const int32_t *, float *, int, int, int, int, int, int64_t, int, cudaStream_t) { return called("staged"); }
bool attn_rotary_mma_supported(int, int, int D, int G, int S, int) { return D == 128 && G == 16 && S == 2; }
int attn_rotary_mma_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const __half *, const int32_t *, const int32_t *,
                             float *, int, int, int, int64_t, int64_t visible, int, bool, int *splits, cudaStream_t) { *splits = splits_of("mma"); return called("mma", visible); }
bool attn_rotary_ladder_supported(int, int, int D, int G, int S, int) { return D == 128 && G == 1 && S >= 4 && S <= 16; }
int attn_rotary_ladder_dispatch(const __half *, const uint8_t *, const uint8_t *, const __half *, const __half *, const __half *, const int32_t *, const int32_t *,
                                float *, int, int, int, int, int64_t, int64_t visible, int, const LadderStep &step, int *splits, cudaStream_t) {
    *splits = splits_of("ladder");
    return called("ladder", visible, step.fresh);
}
}
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    from tac_vq_kv_cache_b200 import _lib, build

    if not (shutil.which("nvcc") or Path("/usr/local/cuda/bin/nvcc").exists()):
        pytest.skip("no nvcc")
    folder = tmp_path_factory.mktemp("dispatch")
    (folder / "stand_ins.cu").write_text(STAND_INS)
    target = folder / "libdispatch.so"
    done = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", str(PACKAGE / "csrc" / "abi.cu"), str(folder / "stand_ins.cu"), "-o", str(target)],
                          capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    lib = ctypes.CDLL(str(target), mode=ctypes.RTLD_LOCAL)
    for name, (restype, argtypes) in _lib._SIGNATURES.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = restype, argtypes
    lib.stand_in_calls.restype = ctypes.c_char_p
    lib.stand_in_tell.argtypes = [ctypes.c_char_p, ctypes.c_int]
    return lib


def _calls(lib):
    return [line.split() for line in lib.stand_in_calls().decode().splitlines()]


def _attend(lib, groups, stages, *, rope, t_cap=1000, batch=1, hq=8, hkv=2):
    dim, at = 128, 1 << 20  # addresses that nobody follows
    need = lib.tacvq_attn_workspace_bytes(batch, hq, hkv, dim, groups, stages)
    tail = (at, need, at, 0, batch, hq, hkv, dim, groups, stages, 256, t_cap, 0)
    if rope:
        return lib.tacvq_attn_decode_rotary(at, at, at, at, at, at, 0, 0, *tail)
    return lib.tacvq_attn_decode(at, at, at, at, at, 0, 0, *tail)


@pytest.mark.parametrize("kernel,groups,stages", [("ladder", 1, 16), ("mma", 16, 2), ("staged", 16, 1)])
def test_a_rotary_launch_that_fails_is_the_calls_status(library, kernel, groups, stages):
    """No other kernel is tried after an error: it would hide it, or fail for it."""
    for splits in (0, 3):
        library.stand_in_reset()
        library.stand_in_tell(kernel.encode(), 98)
        library.stand_in_tell(f"{kernel}.splits".encode(), splits)
        status = _attend(library, groups, stages, rope=True)
        if kernel == "staged" and splits == 0:  # does not take such a size, and is not launched
            assert status == 0 and [c[0] for c in _calls(library)] == ["rotary", "combine"]
        else:
            assert status == 98 and [c[0] for c in _calls(library)] == [kernel]


@pytest.mark.parametrize("kernel,groups,stages", [("ladder", 1, 16), ("mma", 16, 2), ("staged", 16, 1)])
def test_a_rotary_kernel_that_steps_aside_leaves_the_call_to_the_general_one(library, kernel, groups, stages):
    library.stand_in_reset()
    library.stand_in_tell(f"{kernel}.splits".encode(), 0)
    assert _attend(library, groups, stages, rope=True) == 0
    assert [c[0] for c in _calls(library) if c[0] != kernel] == ["rotary", "combine"]


@pytest.mark.parametrize("groups,stages,rope", [(1, 2, False), (1, 16, False), (16, 1, False), (1, 16, True), (16, 2, True)])
def test_a_step_and_attention_after_it_divide_the_work_alike(library, groups, stages, rope):
    """Both are told what is visible: 300 of 5000 positions."""
    from tac_vq_kv_cache_b200 import _lib

    at, batch, hq, hkv, dim, t_cap, length, window = 1 << 20, 2, 8, 2, 128, 5000, 4000, 300
    need = library.tacvq_attn_workspace_bytes(batch, hq, hkv, dim, groups, stages)
    plan = _lib.STEP_PLAN.pack(at, at, at if rope else 0, at, at, at, at, at, need, window, t_cap, batch, hq, hkv, dim, groups, stages, 256)
    library.stand_in_reset()
    assert library.tacvq_decode_step_planned(plan, at, at, at, 0, 1, length, at, 0, 0) == 0
    step = [c[:2] for c in _calls(library) if c[0] != "prologue"]
    library.stand_in_reset()
    assert library.tacvq_attn_decode_within(at, at, at, at, at, at if rope else 0, at, at, at, need, at, 0, batch, hq, hkv, dim, groups, stages, 256,
                                            t_cap, window, 0) == 0
    assert [c[:2] for c in _calls(library)] == step
    assert step[0][1] == "300" and step[-1][0] == "combine"
    library.stand_in_reset()
    assert _attend(library, groups, stages, rope=rope, t_cap=t_cap) == 0  # nothing is known: the whole buffer
    assert _calls(library)[0][1] == "5000"


# us a decode step through attn_rotary_kernel / the ladder kernel: 8 KV heads; stages, rows, query heads per KV head, tokens
LADDER_TIMES = """
4 1 4 600 43.6 19.9; 4 1 1 600 33.6 19.3; 4 4 4 2000 54.7 78.7; 4 4 1 2000 42.9 78.8; 4 8 4 300 39.2 61.8; 4 2 4 8192 101.1 124.9; 4 16 1 300 34.1 100.9
4 1 2 2500 40.6 31.7; 4 1 4 2500 49.1 31.8; 4 16 4 1000 95.7 144.7; 8 1 4 600 63.5 27.3; 8 1 2 6000 70.2 54.5; 8 4 1 2000 64.4 86.7; 8 8 4 300 55.3 70.0
8 16 4 300 64.1 111.6; 8 2 4 1000 69.7 41.3; 8 16 2 1000 115.2 156.4; 12 1 1 600 67.7 36.3; 12 8 4 2000 180.8 150.6; 12 16 4 300 80.5 134.1
12 4 2 2000 89.9 102.2; 16 1 4 130 81.8 39.6; 16 1 4 6000 130.2 72.7; 16 16 4 300 100.9 144.1; 16 16 1 300 85.9 144.6; 16 8 4 2000 223.3 159.3
16 2 1 8192 185.8 157.9; 16 8 2 300 72.5 94.9; 16 16 4 1000 227.8 192.9
"""


def test_ladders_go_to_the_kernel_that_is_quicker_for_them(library):
    library.ladder_splits.argtypes = [ctypes.c_int] * 4 + [ctypes.c_int64] * 2
    for line in LADDER_TIMES.replace("\n", ";").split(";"):
        if line.strip():
            stages, rows, rep, tokens, general, ladder = map(float, line.split())
            taken = library.ladder_splits(int(rows), int(8 * rep), 8, int(stages), int(tokens), int(tokens)) > 0
            assert taken == (ladder < general), line
    assert library.ladder_splits(1, 8, 2, 16, 1 << 20, 300000) == 0  # more than 64 splits of 4096
    for visible in (1, 4096, 4097):
        splits = library.ladder_splits(1, 32, 8, 16, 262144, visible)
        assert splits >= 1 and -(-visible // splits) <= 4096


# us a call of fp16 rows with rows wanted, through the mma.sync / the tcgen05 kernel of 8- and 4-wide groups; groups, stages, heads, rows
NARROW_TIMES = """
16 1 1 1500 6.2 7.1; 16 1 1 2250 7.2 7.4; 16 1 4 520 7.0 7.8; 16 1 8 256 7.0 7.2; 16 1 8 300 10.0 7.9; 16 1 8 520 12.0 10.0; 16 1 32 128 11.8 16.6
32 1 2 520 7.3 7.4; 32 1 4 300 10.1 7.4; 32 1 16 130 16.4 16.8; 16 1 16 700 27.5 17.9; 16 2 1 1500 8.7 9.3; 16 2 1 2250 10.3 9.5; 16 2 2 700 8.7 9.2
16 2 4 520 10.1 10.2; 16 2 8 300 14.1 10.2; 16 2 8 1030 31.9 19.8; 16 2 32 90 17.6 23.0; 16 2 32 130 24.0 25.8; 16 3 4 450 13.2 11.5; 16 3 8 190 11.2 11.5
16 4 2 520 11.8 13.6; 16 4 4 300 13.9 13.6; 16 4 4 450 23.0 13.5; 16 4 16 128 22.6 20.3; 16 8 2 512 19.9 22.4; 16 8 4 300 36.4 22.0
"""


def test_narrow_groups_go_to_the_kernel_that_is_quicker_for_them(library):
    """Or is no more than an eighth behind it."""
    library.narrow_pays.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    for line in NARROW_TIMES.replace("\n", ";").split(";"):
        if line.strip():
            groups, stages, heads, rows, small, tiled = map(float, line.split())
            taken = library.narrow_pays(int(rows), int(groups * heads), int(stages))
            assert (tiled if taken else small) <= 1.125 * min(small, tiled), line


@pytest.mark.parametrize("pairs", [1, 3, 16, 17, 64, 100, 128, 256, 512, 777])
def test_narrow_tiles_are_dealt_out_once_each(library, pairs):
    """As the kernel walks its part: span by span, pair by pair.  No block has more rounds and tables than the plan counts with."""
    library.narrow_deal.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_void_p]
    plan = (ctypes.c_int * 4)()
    for tiles in (*range(1, 34), 47, 63, 94, 127, 128, 129, 140, 256, 260):
        library.narrow_deal(tiles, pairs, plan)
        blocks, last_unit, rounds, visits = plan
        assert 1 <= blocks <= 148 and last_unit in (1, 2, 4)
        for span in range(0, tiles, 128):
            wide = min(128, tiles - span)
            unit = 4 if wide == 128 else last_unit
            units = -(-wide // unit)
            seen = [0] * (pairs * wide)
            for block in range(blocks):
                at, end, own = pairs * units * block // blocks, pairs * units * (block + 1) // blocks, []
                while at < end:
                    pair, first = divmod(at, units)
                    mine = min(units - first, end - at)
                    begin, stop = first * unit, min(wide, (first + mine) * unit)
                    for tile in range(begin, stop):
                        seen[pair * wide + tile] += 1
                    own.append(stop - begin)
                    at += mine
                if wide < 128 or tiles == 128:
                    assert len(own) <= visits and sum(-(-n // 4) for n in own) <= rounds, (tiles, block)
            assert set(seen) == {1}, tiles
