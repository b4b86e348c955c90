"""The uniform-diagonal check against a plain restatement: random sets of diagonals around the limit of 16, rows
that miss some, empty rows, columns out of order, one diagonal found late, sizes over several host threads."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT
from test_plan_rows_cpu import PROGRAM as _PLAN
from test_sanitize_cpu import CSRC, _cuda_include

PROGRAM = _PLAN[:_PLAN.index("using hhp::SellHost;")].replace("#include <random>", "#include <map>\n#include <random>\n#include <set>") + r"""
static bool plain(int m, const std::vector<int> &rp, const std::vector<int> &col, int max_k, double pad,
                  std::vector<int> &off, std::vector<int> &mask) {
    std::set<int> d;
    if (rp[m] <= 0) return false;
    for (int i = 0; i < m; ++i)
        for (int p = rp[i]; p < rp[i + 1]; ++p) {
            if (p > rp[i] && col[p] <= col[p - 1]) return false;
            d.insert(col[p] - i);
        }
    if (static_cast<int>(d.size()) > max_k || static_cast<double>(d.size()) * m > (1.0 + pad) * rp[m]) return false;
    off.assign(d.begin(), d.end());
    std::map<int, int> at;
    for (size_t k = 0; k < off.size(); ++k) at[off[k]] = static_cast<int>(k);
    mask.assign(m, 0);
    for (int i = 0; i < m; ++i)
        for (int p = rp[i]; p < rp[i + 1]; ++p) mask[i] |= 1 << at[col[p] - i];
    return true;
}
int main() {
    std::mt19937 g(2);
    int yes = 0, no = 0;
    for (int it = 0; it < 600; ++it) {
        const int m = it % 40 == 0 ? 300000 : 1 + static_cast<int>(g() % 2000), n_off = 1 + static_cast<int>(g() % 18);
        std::set<int> off;
        while (static_cast<int>(off.size()) < n_off) off.insert(static_cast<int>(g() % 200) - 100);
        const unsigned miss = g() % 3 ? 50 : 4;
        std::vector<int> rp(1, 0), col;
        for (int i = 0; i < m; ++i) {
            for (int o : off)
                if (i + o >= 0 && i + o < m && g() % miss) col.push_back(i + o);
            if (g() % 100 == 0) col.resize(rp.back());
            rp.push_back(static_cast<int>(col.size()));
        }
        const int end = rp[m] - rp[m - 1];
        if (it % 7 == 0 && end > 1) std::swap(col[rp[m - 1]], col[rp[m - 1] + 1]);  // the last row out of order
        if (it % 11 == 0 && end > 0) col[rp[m] - 1] = m + 500;                      // a diagonal only there
        for (double pad : {0.1, 1e9})
            for (int max_k : {16, 5}) {
                int doff[hhp::kMaxDiag] = {}, K = 0;
                std::vector<int> mask, want_off, want_mask;
                const bool ok = hhp::uniform_diagonals(m, rp.data(), col.data(), max_k, pad, doff, K, mask);
                const bool want = plain(m, rp, col, max_k, pad, want_off, want_mask);
                ++(ok ? yes : no);
                if (ok != want) { std::printf("case %d: %d, not %d\n", it, ok, want); return 1; }
                if (ok && (std::vector<int>(doff, doff + K) != want_off || mask != want_mask)) { std::printf("case %d\n", it); return 2; }
            }
    }
    return yes > 100 && no > 100 ? 0 : 3;
}
"""


def test_against_a_plain_restatement(tmp_path):
    gxx, inc = shutil.which("g++"), _cuda_include()
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are not available")
    src, exe = tmp_path / "diag.cpp", tmp_path / "diag"
    src.write_text(PROGRAM)
    cmd = [gxx, "-std=c++17", "-O2", "-pthread", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-I" + inc, str(src),
           os.path.join(CSRC, "hhp_plan.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
