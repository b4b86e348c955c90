"""build_plan with another number of rows per lane for rows that need sorting: the plan of one call is, member by
member, the one that two calls would choose (the first kept unless it had to sort)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT
from test_sanitize_cpu import CSRC, _cuda_include

PROGRAM = r"""
#include <cstdarg>
#include <cstdio>
#include <random>
#include "hhp_internal.h"
namespace hhp {
void set_error(const char *, ...) {}
int env_int(const char *, int dflt) { return dflt; }
const Tuning &tuning() {
    static const Tuning t;
    return t;
}
}  // namespace hhp
using hhp::SellHost;
static bool same(const SellHost &a, const SellHost &b) {
    if (a.chunks.size() != b.chunks.size()) return false;
    for (size_t i = 0; i < a.chunks.size(); ++i)
        if (a.chunks[i].x != b.chunks[i].x || a.chunks[i].y != b.chunks[i].y || a.chunks[i].z != b.chunks[i].z ||
            a.chunks[i].w != b.chunks[i].w)
            return false;
    return a.rpl == b.rpl && a.H == b.H && a.n_slices == b.n_slices && a.sorted == b.sorted && a.has_perm == b.has_perm &&
           a.pos_row == b.pos_row && a.pos_len == b.pos_len && a.slice_ptr == b.slice_ptr && a.total == b.total &&
           a.short_nnz == b.short_nnz && a.padding == b.padding && a.long_rows == b.long_rows &&
           a.long_first == b.long_first && a.chunk_long == b.chunk_long;
}
int main() {
    std::mt19937 g(1);
    int kinds[3] = {0, 0, 0};  // natural order, sorted at the other rpl, natural there
    for (int it = 0; it < 400; ++it) {
        const int m = it < 20 ? it : 1 + static_cast<int>(g() % (it % 10 ? 3000 : 200000)), run = 1 << g() % 9;
        const unsigned spread = 1 + g() % 60, base = g() % 30, big = g() % 4;
        std::vector<int> rp(1, 0);
        int len = 0;
        for (int i = 0; i < m; ++i) {
            if (i % run == 0) len = static_cast<int>(base + g() % spread);
            rp.push_back(rp.back() + (big && g() % 997 == 0 ? 300 * static_cast<int>(big) : len));
        }
        for (int rpl : {4, 2}) {
            SellHost one, first, second;
            hhp::build_plan(m, rp.data(), rpl, 256, 2048, 8192, one, rpl / 2);
            hhp::build_plan(m, rp.data(), rpl, 256, 2048, 8192, first);
            hhp::build_plan(m, rp.data(), rpl / 2, 256, 2048, 8192, second);
            ++kinds[!first.sorted ? 0 : second.sorted ? 1 : 2];
            if (!same(one, first.sorted ? second : first)) {
                std::printf("m %d, rows per lane %d, case %d\n", m, rpl, it);
                return 1;
            }
        }
    }
    std::printf("%d %d %d\n", kinds[0], kinds[1], kinds[2]);
    return kinds[0] && kinds[1] && kinds[2] ? 0 : 2;
}
"""


def test_one_call_chooses_as_two_would(tmp_path):
    gxx, inc = shutil.which("g++"), _cuda_include()
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are not available")
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    cmd = [gxx, "-std=c++17", "-O2", "-pthread", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-I" + inc, str(src),
           os.path.join(CSRC, "hhp_plan.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
