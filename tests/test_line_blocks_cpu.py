"""Block sizes of the register-line kernels: the kernels divide a block into
blockDim / th lines of th threads, so for every number of lines that a shape,
the autotuner or an environment variable can ask for, and for any mixture of
members that share a block, no thread may be left over."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastisostasy_gb300", "csrc")

PROGRAM = """
#include <cstdio>
#include "fi_shapes.h"
int main()
{
    for (int most = 512; most <= 1024; most *= 2)
        for (int lines = 1; lines <= 40; ++lines)
            for (int th = 1; th <= 512; th *= 2) std::printf("%d %d %d %d\\n", most, lines, th, fi::line_block(lines, th, most));
}
"""


def test_no_thread_without_a_line(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "blocks.cpp", tmp_path / "blocks"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([str(exe)], check=True, capture_output=True,
                                                               text=True).stdout.splitlines()]
    assert len(rows) == 2 * 40 * 10
    for most, lines, th, block in rows:
        assert 32 <= block <= most and block & (block - 1) == 0 and block % th == 0
        # as many lines as asked for, or as many as fit (a warp where they are less)
        assert block >= min(lines * th, most) or block * 2 > most
        assert block // 2 < max(lines * th, 32)
    # members that share a block: the largest one holds whole lines of every other
    for most in (512, 1024):
        sizes = [(th, block) for m, _, th, block in rows if m == most]
        for common in {b for _, b in sizes}:
            assert all(common % th == 0 for th, block in sizes if block <= common)
