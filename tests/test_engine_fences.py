"""Every wait of the tensor-core kernels that a tcgen05 access may follow is fenced: an mbarrier wait orders
tcgen05 loads, stores and MMAs of the waiting thread only through tcgen05.fence::after_thread_sync. The order is
not observable reliably on a device, so it is read from the sources: the one function of each role through which its
waits go issues the fence.
"""
import os
import re

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "hignn_b200", "csrc")


def body(text, start):
    """The brace-delimited block that opens after position `start`."""
    depth, first = 0, text.index("{", start)
    for q in range(first, len(text)):
        depth += {"{": 1, "}": -1}.get(text[q], 0)
        if depth == 0:
            return text[first:q + 1]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("source,role,wait", [
    ("tc_mlp.cuh", r"struct MmaWarp ", r"bool wait\("),
    ("tc_mlp.cuh", r"struct Epi ", r"bool wait\("),
    ("three_body.cu", r"struct MmaWarpTb ", r"bool wait\("),
    ("three_body.cu", r"struct Epi ", r"bool wait\("),
    ("student.cu", r"k_far_student_tc\(", r"auto await = "),
])
def test_waits_are_fenced(source, role, wait):
    with open(os.path.join(CSRC, source)) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    text = body(text, re.search(role, text).start())
    waits = body(text, re.search(wait, text).start())
    assert "fence_after()" in waits
    # and no wait of the role goes around it, but for the drain before the CTA's teardown, which fences itself
    rest = re.sub(r"(wait_bar\(&s\.drain[^;]*;|while \(!tc::mbar_try\(&S\.bar, phase & 1\) &&[^;{]*\{)", "",
                  text.replace(waits, ""))
    assert not re.search(r"\b(mbar_try|mbar_try_sleep|mbar_wait|warp_wait|wait_bar|warp_wait_bar)\(", rest)
