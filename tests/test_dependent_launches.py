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
    "attn_gsrq_scan_kernel": {"kcodes", "vcodes", "lut_g", "scale_g", "seq_start", "seq_end"},
    "attn_combine_kernel": {"states"},
    "attn_gsrq_prepare_kernel": {"q", "ktab", "vtab", "fresh"},
    "decode_prologue_kernel": {"k_rows", "v_rows", "ktab", "vtab"},
    "encode_few_wide_kernel": {"first", "second"},
}
# device functions through which the first kernels of a step read rows and tables -> the parameters
READ_THROUGH = {"encode_row_unit": {"x", "tables", "sqnorm_in"}, "nearest_word_in_warp": {"words", "sqnorm_in"}}
WAITS = ("wait_for_previous_kernel()", "start_after_previous_kernel()")


def _kernels(head=r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?", sources="*.cu"):
    for source in sorted(CSRC.glob(sources)):
        text = re.sub(r"//[^\n]*", "", source.read_text())
        for match in re.finditer(head + r"(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
            depth, at = 1, match.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield match.group(1), match.group(2), text[match.end() : at], text


def test_every_kernel_that_waits_is_listed():
    waiting = {name for name, _, body, _ in _kernels() if any(wait in body for wait in WAITS)}
    assert waiting == set(WRITTEN_BEFORE)


@pytest.mark.parametrize("name", sorted(WRITTEN_BEFORE))
def test_results_of_the_kernel_before_are_not_constant_memory(name):
    ((params, body, text),) = [found[1:] for found in _kernels() if found[0] == name]
    declared = {re.findall(r"\w+", param)[-1]: param for param in params.split(",")}
    assert WRITTEN_BEFORE[name] <= set(declared)
    for word in WRITTEN_BEFORE[name]:
        assert "__restrict__" not in declared[word], declared[word].strip()
    aliases = WRITTEN_BEFORE[name] | {"kc", "vc", "kc_row", "vc_row", "k_row", "v_row_g", "kp", "sg", "src_codes", "own"}
    for load in re.findall(r"__ldg\(.*?\);|ldg_in_place\(.*?\);", body):
        assert not aliases & set(re.findall(r"\w+", load)), load
    stream = re.search(r"ldg_stream\(const void \*p\) \{(.*?)\n\}", text, re.S)
    assert stream is None or ".nc" not in stream.group(1)


@pytest.mark.parametrize("name", ["attn_gsrq_prepare_kernel", "decode_prologue_kernel", "encode_few_wide_kernel"])
def test_the_first_kernel_of_a_step_waits_before_it_reads_anything(name):
    """It follows whatever kernel computed the query and the rows, also one that lets it start before they are stored."""
    ((_, body, _),) = [found[1:] for found in _kernels() if found[0] == name]
    head = body[: min(body.index(wait) for wait in WAITS if wait in body)]
    # (the tables' address and a request that is only made later are formed before)
    head = re.sub(r"const FewSide side = is_second \? second : first;|const __half \*words = side\.tables \+ [^;]*;|auto request = .*?\};", "", head, flags=re.S)
    assert not (WRITTEN_BEFORE[name] | {"side", "words", "words0", "words1"}) & set(re.findall(r"\w+", head))
    assert "__ldg" not in body and ".nc" not in body and "__restrict__" not in body


def test_the_scan_reads_only_what_is_older_than_the_table_preparation_before_its_wait():
    """V words and ranges; the preparation lets it start only after its own wait."""
    ((_, scan, _),) = [found[1:] for found in _kernels() if found[0] == "attn_gsrq_scan_kernel"]
    (loop,) = re.findall(r"while \(cursor < my_end\)(.*?)wait_once\(\);", scan, re.S)
    assert not {"lut_g", "scale_g", "part", "marks", "out", "ldg_stream", "cp_async16"} & set(re.findall(r"\w+", loop))


def test_no_kernel_lets_the_next_one_start_before_its_own_wait():
    """The next kernel reads what is older than the one in front of it (tables, old codes, ranges) before it waits itself."""
    triggers = {name: body for name, _, body, _ in _kernels() if "launch_dependents()" in body or "start_after_previous_kernel()" in body}
    assert {"decode_prologue_kernel", "encode_few_wide_kernel", "attn_slots_kernel", "attn_combine_kernel", "attn_gsrq_prepare_kernel"} <= set(triggers)
    for name, body in triggers.items():
        if "launch_dependents()" in body:
            assert body.index("wait_for_previous_kernel()") < body.index("launch_dependents()"), name
    ((params, body, _),) = [found[1:] for found in _kernels(r"__device__ __forceinline__ void ", "common.cuh") if found[0] == "start_after_previous_kernel"]
    assert [line.strip() for line in body.strip("}").split(";") if line.strip()] == ["wait_for_previous_kernel()", "launch_dependents()"]


@pytest.mark.parametrize("name", sorted(READ_THROUGH))
def test_the_rows_and_tables_of_a_step_are_not_constant_memory_to_its_first_kernel(name):
    """It may be scheduled while the launch that computes them runs."""
    ((params, body, _),) = [found[1:] for found in _kernels(r"__device__ __forceinline__ \w+ ", "encode*.cu*") if found[0] == name]
    declared = {re.findall(r"\w+", param)[-1]: param for param in params.split(",")}
    assert READ_THROUGH[name] <= set(declared)
    for word in READ_THROUGH[name]:
        assert "__restrict__" not in declared[word], declared[word].strip()
    body = re.sub(r"if constexpr \(CONSTANT\)[^;]*;", "", body)
    assert "__ldg" not in body and ".nc" not in body
    ((_, prologue, _),) = [found[1:] for found in _kernels() if found[0] == "decode_prologue_kernel"]
    assert re.findall(r"encode_row_unit<[^>]*>", prologue) == ["encode_row_unit<DSUB, XT, false>"]
