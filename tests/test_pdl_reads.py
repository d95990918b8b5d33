"""Launches that start before they have waited for the kernel in front (kPdlNext) read the activations past L1 and the read-only
path.  Read from the source."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_run_of_projections_reads_its_activations_from_l2():
    with open(os.path.join(ROOT, "engine_b200", "csrc", "hq_gemv_int8.cu")) as f:
        text = f.read()
    body = re.search(r"void q8_x_prefetch\(.*?\n}\n", text, re.S).group(0)
    assert "q8_load_x(" in body and "__ldg" not in body
    assert "asm volatile(\"ld.relaxed.gpu.global" in re.search(r"uint4 q8_load_x\(.*?\n}\n", text, re.S).group(0)
