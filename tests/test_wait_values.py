"""Waits that leave no branch behind (warp_wait_uni) return 1, or 0 when they ran out; a caller keeps that in `spin`, where 0
says that a wait ran out, and reports that behind its loop.  Read from the source, as the waits with a branch are."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "engine_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "hq_warp_issue.cuh"
               and "warp_wait_uni(" in open(os.path.join(CSRC, f)).read())


def faults(text):
    code = "\n".join(line.split("//")[0] for line in text.split("\n"))
    kept = len(re.findall(r"spin = warp_wait_uni\([^;]*, spin\) \? spin : 0u;", code))
    uses = code.count("warp_wait_uni(")
    # every role that waits so has a check of `spin` with a report behind it
    reports = len(re.findall(r"spin == 0u[^;]*\)[^;]*\{?[^;]*report_status", code, re.S))
    return uses - kept, reports


@pytest.mark.parametrize("name", FILES)
def test_the_value_is_kept_and_reported(name):
    lost, reports = faults(open(os.path.join(CSRC, name)).read())
    assert lost == 0 and reports >= 1


def test_a_lost_value_is_found():
    assert faults("  warp_wait_uni(a, ph, spin);\n") == (1, 0)
    assert len(FILES) >= 5
