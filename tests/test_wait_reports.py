"""Every bounded wait of the kernels leaves HQ_DEV_WAIT_TIMEOUT in the status word when it runs out: a wait that gives up in
silence hides a stall of many milliseconds behind a right result.  Read from the source: no such wait can be made to run out
on the GPU one by one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "engine_b200", "csrc")
WAIT = re.compile(r"\b(warp_wait|warp_drain|mbar_wait|mbar_wait_backoff|dq_wait_cluster)\s*\(")
DEFINITION = re.compile(r"__device__ __forceinline__ bool \w+\(")


def silent_waits(text):
    """Lines with a wait whose result is not followed by a report within the branch it opens."""
    lines = text.split("\n")
    inside, out = False, []                   # inside: the body of one of the wait functions themselves
    for i, line in enumerate(lines):
        if DEFINITION.search(line):
            inside = True
        if not inside and WAIT.search(line.split("//")[0]) and "report_status" not in " ".join(lines[i:i + 4]):
            out.append(i + 1)
        if line.startswith("}"):
            inside = False
    return out


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_a_wait_that_runs_out_is_reported(name):
    assert silent_waits(open(os.path.join(CSRC, name)).read()) == []


def test_a_silent_wait_is_found():
    assert silent_waits("  for (;;)\n    if (!warp_wait(&full[i], 0, spin)) break;\n  }\n  next();\n  done();\n") == [2]


@pytest.mark.parametrize("name", ["hq_dq_gemm.cuh", "hq_fp8_grouped.cu", "hq_mx_grouped.cu", "hq_mx_rows.cu"])
def test_copies_are_waited_for_by_the_warps_that_issue_them(name):
    # after a time-out nobody else waits for a stage any more: the rings box copies signal are drained before the CTA exits,
    # by warp_drain or by a loop over the last stages of the sequence
    text = open(os.path.join(CSRC, name)).read()
    rings = set(re.findall(r"warp_tma_[23]d\([^;]*&([\w.]+)\[", text, re.S))
    drained = set(re.findall(r"warp_drain\(([\w.]+),", text))
    for loop in re.findall(r"for \(int i = [^;]*(?:next|it) - pl\.n[rs]\)?;.*?warp_wait\(&([\w.]+)\[", text, re.S):
        drained.add(loop)
    assert rings and rings <= drained, (rings, drained)


def short_waits(text):
    """Waits by short polls in a file whose limit counts polls that are suspended for 20 us each: 64 times shorter than meant."""
    limits = [1 << int(n) for n in re.findall(r"constexpr uint32_t k\w*Spin\w* = 1u << (\d+);", text)]
    code = "\n".join(line.split("//")[0] for line in text.split("\n"))
    return re.findall(r"\bmbar_(?:try_)?wait\w*\s*\(", code) if limits and min(limits) < 1 << 22 else []


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "hq_common.cuh"))
def test_a_limit_of_long_polls_is_not_used_with_short_ones(name):
    assert short_waits(open(os.path.join(CSRC, name)).read()) == []


def test_a_short_wait_is_found():
    assert short_waits("constexpr uint32_t kSpin = 1u << 16;\n  if (!mbar_wait_backoff(&empty[s], 0, spin)) {\n") != []
    assert short_waits("constexpr uint32_t kSpin = 1u << 22;\n  if (!mbar_wait(&empty[s], 0, spin)) {\n") == []


def handed_on(text):
    """Places where a role hands its work on although a wait of its own ran out: (branches that go on without telling the storing
    warps, roles that wait by value and arrive all the same)."""
    code = "\n".join(line.split("//")[0] for line in text.split("\n"))
    branches = [b for b in re.findall(r"if \([^;{]*!warp_wait\([^{]*\{(.*?)\n\s*\}", code, re.S)
                if "spin = 1" in b and "late = 1u" not in b and "failed = true" not in b]
    roles = re.split(r"\n(?=[^\n]*={20,}|[^\n]*={17} )", text)
    by_value = [r[:60] for r in roles if "spin = warp_wait_uni(" in r
                and not re.search(r"warp_mark_late\(|warp_arrive_live\(|spin != 0u\) mbar_arrive\(", r)]
    return branches, by_value


@pytest.mark.parametrize("name", ["hq_gemv.cu", "hq_gemv_int8.cu", "hq_mx_rows.cu", "hq_mx_grouped.cu"])
def test_what_a_late_warp_hands_on_is_not_stored(name):
    text = open(os.path.join(CSRC, name)).read()
    assert handed_on(text) == ([], [])
    # the storing warps remember a wait that ran out: nothing is stored from there on
    assert "failed = true" in text and re.search(r"\n {6,}bool failed = false", text) is None


def test_a_missing_mark_is_found():
    role = "// ===================== consumers\n  spin = warp_wait_uni(b, 0, spin) ? spin : 0u;\n  warp_arrive(&full);\n"
    assert handed_on(role)[1] != []
    assert handed_on("  if (!warp_wait(&empty[s], 0, spin)) {\n    report_status(s, 1, 2);\n    spin = 1;\n  }\n")[0] != []
