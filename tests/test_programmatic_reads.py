"""Kernels that start before the one they follow has ended must not read its results as read-only data: a
non-coherent load (__ldg, or one the compiler makes of a `const ... __restrict__` pointer) is for memory that does
not change while the kernel runs, and nothing orders it behind griddepcontrol.wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "black-hole_b200", "csrc")

# kernel: what the launch before it writes and this one reads
READS = [("bh_post.cu", "composite_kernel", ["hblur"]),
         ("bh_sg_chain.cu", "weight_grad_kernel", ["slices"]),
         ("bh_sg_chain.cu", "chain_kernel", ["params"]),
         ("bh_sg_train.cu", "pack_kernel", ["parts", "m", "v"])]


@pytest.mark.parametrize("name, kernel, written", READS)
def test_results_of_the_launch_before_are_read_coherently(name, kernel, written):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    at = re.search(r"\n%s\(" % kernel, text).start()
    body = text[at:text.index("\n}\n", at)]
    assert "griddepcontrol.wait" in body or "wait_for_previous()" in body
    head = body[:body.index("{")]
    for data in written:
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+%s\b" % data, head)
        assert not re.search(r"__ldg\(\s*(?:\w+\.)?%s\b" % data, body)
