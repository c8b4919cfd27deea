"""The list of buffers that one launch clears (ClearList) never writes past its end: one too
many is remembered, and the launch refuses the list.  Built for the host."""
import os
import shutil
import subprocess

import pytest

from qlens_gb300 import abi

CODE = r"""
#include "qlpix_internal.h"
#include <cstdio>
using namespace qlpix;
struct { ClearList l; unsigned guard[8]; } s;
int main()
{
    for (unsigned& g : s.guard) g = 0x5a5a5a5au;
    for (int i = 0; i < CLEAR_MAX; i++) s.l.add(&s, 9 + i, i);
    if (s.l.n != CLEAR_MAX || s.l.full || s.l.item[1].words != 3) return 1;
    s.l.add(&s, 4, 7);
    s.l.add(&s, 4, 7);
    if (s.l.n != CLEAR_MAX || !s.l.full) return 2;
    for (unsigned g : s.guard) if (g != 0x5a5a5a5au) return 3;
    return 0;
}
"""


def test_one_too_many_is_not_written(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not shutil.which("g++") or not os.path.isdir(os.path.join(cuda, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = str(tmp_path / "c.cpp"), str(tmp_path / "c")
    with open(src, "w") as f:
        f.write(CODE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(abi.package_dir(), "csrc"), "-I",
                           os.path.join(cuda, "include"), src, "-o", exe])
    assert subprocess.run([exe]).returncode == 0
