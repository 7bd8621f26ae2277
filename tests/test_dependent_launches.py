"""Source check of the kernels that may start before the kernel in front of them has ended (CPU).

What such a kernel reads of its predecessor's results must not be declared or fetched as constant memory, or the compiler may move
the read above the wait.  When that happens depends on the compiler and on timing, so the declarations are what is checked.
"""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tac_vq_kv_cache_b200" / "csrc"

# kernel -> what the launch before it may have written
WRITTEN_BEFORE = {
    "attn_slots_kernel": {"kcodes", "vcodes", "seq_start", "seq_end"},
    "attn_rotary_mma_kernel": {"kcodes", "vcodes", "seq_start", "seq_end"},
    "attn_rotary_ladder_kernel": {"kcodes", "vcodes", "seq_start", "seq_end"},
    "attn_gsrq_scan_kernel": {"kcodes", "vcodes", "lut_g", "scale_g", "vperm_g", "seq_start", "seq_end"},
    "attn_combine_kernel": {"states"},
    "attn_gsrq_prepare_kernel": {"q", "ktab", "vtab"},
}


def _kernels():
    for source in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", source.read_text())
        for match in re.finditer(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\(([^)]*)\)\s*\{", text):
            depth, at = 1, match.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield match.group(1), match.group(2), text[match.end() : at], text


def test_every_kernel_that_waits_is_listed():
    waiting = {name for name, _, body, _ in _kernels() if "wait_for_previous_kernel()" in body}
    assert waiting == set(WRITTEN_BEFORE)


@pytest.mark.parametrize("name", sorted(WRITTEN_BEFORE))
def test_results_of_the_kernel_before_are_not_constant_memory(name):
    ((params, body, text),) = [found[1:] for found in _kernels() if found[0] == name]
    for param in params.split(","):
        word = re.findall(r"\w+", param)[-1]
        if word in WRITTEN_BEFORE[name]:
            assert "__restrict__" not in param, param.strip()
    aliases = WRITTEN_BEFORE[name] | {"kc", "vc", "kc_row", "vc_row", "k_row", "v_row_g", "kp", "sg", "src_codes", "own"}
    for load in re.findall(r"__ldg\(.*?\);|ldg_in_place\(.*?\);", body):
        assert not aliases & set(re.findall(r"\w+", load)), load
    stream = re.search(r"ldg_stream\(const void \*p\) \{(.*?)\n\}", text, re.S)
    assert stream is None or ".nc" not in stream.group(1)


def test_the_table_preparation_waits_before_it_reads_anything():
    """It follows whatever kernel computed the query and the rows, also one that lets it start before they are stored."""
    ((_, body, _),) = [found[1:] for found in _kernels() if found[0] == "attn_gsrq_prepare_kernel"]
    head = body[: body.index("wait_for_previous_kernel()")]
    assert not {"q", "ktab", "vtab", "fresh"} & set(re.findall(r"\w+", head))


def test_the_table_preparation_lets_the_scan_start_only_after_its_own_wait():
    """The scan reads what is older than the preparation (V words, ranges) before its own wait."""
    ((_, body, _),) = [found[1:] for found in _kernels() if found[0] == "attn_gsrq_prepare_kernel"]
    assert body.index("wait_for_previous_kernel()") < body.index("launch_dependents()")
    ((_, scan, _),) = [found[1:] for found in _kernels() if found[0] == "attn_gsrq_scan_kernel"]
    before = scan[scan.index("while (cursor < my_end)") : scan.index("wait_once();\n        uint4 k0")]
    assert not {"lut_g", "scale_g", "part", "marks", "out"} & set(re.findall(r"\w+", before))


def test_no_kernel_lets_the_next_one_start_before_its_own_wait():
    """The next kernel reads what is older than the one in front of it (tables, old codes, ranges) before it waits itself."""
    triggers = {name: body for name, _, body, _ in _kernels() if "launch_dependents()" in body or "start_after_previous_kernel()" in body}
    assert {"decode_prologue_kernel", "encode_few_wide_kernel", "attn_slots_kernel", "attn_combine_kernel"} <= set(triggers)
    for name, body in triggers.items():
        if "launch_dependents()" in body:
            assert body.index("wait_for_previous_kernel()") < body.index("launch_dependents()"), name


def test_the_rows_and_tables_of_a_step_are_not_constant_memory_to_its_first_kernel():
    """It may be scheduled while the launch that computes them runs."""
    found = {name: (params, body) for name, params, body, _ in _kernels()}
    params, body = found["decode_prologue_kernel"]
    assert body.split(";")[0].strip() == "start_after_previous_kernel()"
    for param in params.split(","):
        if re.findall(r"\w+", param)[-1] in {"k_rows", "v_rows", "ktab", "vtab"}:
            assert "__restrict__" not in param, param.strip()
    assert "__ldg" not in (CSRC / "encode_rows.cuh").read_text() and "__ldg" not in found["encode_few_wide_kernel"][1]
