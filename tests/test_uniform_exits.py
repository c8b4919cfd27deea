"""What a kernel does after a wait has run out, read from its source: no GPU run can
bring that about without a hang.

A CTA whose warps wait on different barriers gives up through a shared flag that any
of them may raise.  If the flag decides a branch of the whole CTA, a barrier has to stand
directly before it: otherwise a slow warp sees the flag that a fast one has raised in the
meantime, leaves, and the others stay at their next barrier for good.  Likewise TMEM loads
are warp instructions: the wait before them has to decide for the whole warp.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qlens_gb300", "csrc")
FILES = sorted(os.path.basename(f) for e in ("*.cu", "*.cuh") for f in glob.glob(os.path.join(CSRC, e)))
# a branch on the flag itself (a bounded wait's result is another matter: single lanes)
FLAG = re.compile(r"\bif \((?!.*mbar_wait)(?!.*lane == 0)(?!.*wg_any)[^;]*\babort(_flag)?\b[^;]*\)\s*(break|return|continue);")
# (surrogate.cu's loads follow the wait whatever it returns)
TMEM = ("ozaki.cuh", "chol128.cuh", "tc_syrk.cuh")


def _lines(name):
    out = []
    for line in open(os.path.join(CSRC, name)):
        line = re.sub(r"//.*", "", line).strip()
        if line:
            out.append(line)
    return out


@pytest.mark.parametrize("name", FILES)
def test_a_barrier_stands_before_every_branch_on_the_flag(name):
    lines = _lines(name)
    for k, line in enumerate(lines):
        if FLAG.search(line) and "honor_abort" not in line:
            assert "__syncthreads" in lines[k - 1], (name, lines[k - 1], line)


@pytest.mark.parametrize("name", TMEM)
def test_tmem_loads_follow_a_wait_of_the_whole_warp(name):
    last, seen = None, 0
    for line in _lines(name):
        for m in re.finditer(r"mbar_wait_bounded|mbar_wait_warp|__syncthreads_and|tmem_ld_\w+\(", line):
            w = m.group(0)
            if not w.startswith("tmem_ld_"):
                last = w
            elif "__device__" not in line:
                seen += 1
                assert last in ("mbar_wait_warp", "__syncthreads_and"), (name, line)
    assert seen
