"""The arrival count of the one-kernel solves across 2^32: no block may pass an exchange before every block has
arrived, and all may after, also where the count or the target has wrapped."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT
from test_sanitize_cpu import CSRC, _cuda_include

PROGRAM = r"""
#include <cstdio>
#include "hhp_internal.h"
int main() {
    for (unsigned blocks : {1u, 2u, 7u, 152u, 160u}) {
        // exchanges on either side of the count's wrap, and from a count that starts at any value
        for (unsigned start : {0u, 1u, 0xffffffffu, 0x80000000u}) {
            const unsigned wrap = (0u - start) / blocks;
            for (unsigned around : {1u, wrap > 5 ? wrap - 5 : 1u, 0x7fffffffu / blocks, 0x80000000u / blocks})
                for (unsigned e = around; e < around + 12; ++e) {
                    const unsigned before = start + (e - 1) * blocks, target = start + e * blocks;
                    for (unsigned arrived = 0; arrived <= blocks; ++arrived)
                        if (hhp::count_reached(before + arrived, target) != (arrived == blocks)) {
                            std::printf("%u blocks, start %u, exchange %u, %u arrived\n", blocks, start, e, arrived);
                            return 1;
                        }
                    // a block may already have arrived at the next exchange
                    if (!hhp::count_reached(target + blocks - 1, target)) return 2;
                }
        }
    }
    return 0;
}
"""


def test_count_across_the_wrap(tmp_path):
    gxx, inc = shutil.which("g++"), _cuda_include()
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are not available")
    src, exe = tmp_path / "count.cpp", tmp_path / "count"
    src.write_text(PROGRAM)
    cmd = [gxx, "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-I" + inc, str(src), "-o", str(exe)]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
