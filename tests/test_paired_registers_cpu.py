"""The paired-query kernels run one block of 8 or 12 warps per SM with nearly all
of the registers a thread can have; a spill is paid on every column step.  The
compiler's report of the build says whether one crept in."""
import os
import re

import pytest

REPORT = os.path.join(os.path.dirname(__file__), "..", "swhybrid_b200", "_build", "sw_qp.o.ptxas")


def test_no_paired_kernel_spills():
    if not os.path.exists(REPORT):
        pytest.skip("no compiler report (library not built in tree)")
    text = open(REPORT).read()
    names = re.findall(r"Compiling entry function '(\S*sw_qpbatch\S*)'", text)
    spills = re.findall(r"(\d+) bytes spill stores, (\d+) bytes spill loads", text)
    assert len(names) == len(spills) > 0
    assert [n for n, s in zip(names, spills) if s != ("0", "0")] == []
