"""The kernels' index arithmetic at the top of the accepted range, on the host:
csrc/index_range.h compiled with overflow checks and driven as the kernels drive
it, at sizes that no test matrix could have."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WALK = r"""
#include <algorithm>
#include <climits>
#include <cstdio>
#include "index_range.h"
using namespace merbit;

// One warp over the last tile of a matrix: L merge items, `rows` of them row
// ends behind its nonzeros, in segments of `seg` items for `groups` groups (the
// segments past L are empty).
static int walk(int nrow, int nnz, int seg, int groups, int ch, int L) {
    const int x1 = nnz;
    for (int rows = 0; rows <= std::min(nrow, L); rows = rows ? rows * 2 : 1) {
        const int nz = L - rows, x0 = x1 - nz;
        auto at = [&](int g) { return x0 + std::min(std::min(g * seg, L), nz); };
        int steps = 0;
        for (int g = 0; g < groups; ++g)
            steps = std::max(steps, (at(g + 1) - at(g) + 2 * ch - 1) / (2 * ch));
        for (int g = 0; g < groups; ++g) {
            const int lx = at(g), end = at(g + 1);
            const int last = std::max(end - 1, x0);
            unsigned c = (unsigned)lx;
            int taken = 0;
            auto load = [&](unsigned from) {
                for (int t = 0; t < ch; ++t) {
                    const int e = walk_entry(from, t, last);
                    if (e < x0 || e >= std::max(x1, x0 + 1)) return false;
                }
                return true;
            };
            auto consume = [&](unsigned from) {
                if (walk_clear(end, from, ch)) {
                    taken += ch;
                } else {
                    for (int t = 0; t < ch; ++t) taken += walk_in(from, t, end);
                }
            };
            for (int i = 0; i < steps; ++i) {
                if (!load(c) || !load(c + ch) || !load(c + 2 * ch)) return 1;
                consume(c);
                consume(c + ch);
                c += 2 * ch;
            }
            if (taken != end - lx) return 2;
        }
    }
    return 0;
}

int main() {
    const int shapes[][3] = {{8, 32, 4}, {15, 32, 4}, {11, 32, 4}, {8, 32, 2}, {31, 16, 2}, {31, 16, 4},
                             {63, 8, 2}, {127, 4, 2}, {127, 4, 4}, {255, 2, 4}, {128, 2, 8}, {256, 1, 8}};
    for (int nrow : {1, 2, 7, 64, 300})
        for (int off : {64, 65, 80, 200, 600})
            for (auto& s : shapes) {
                const int nnz = INT_MAX - off - nrow;
                for (int L = 1; L <= s[0] * s[1]; L += L < 24 ? 1 : 37)
                    if (int r = walk(nrow, nnz, s[0], s[1], s[2], L)) {
                        std::printf("nrow %d nnz %d segment %d groups %d chunk %d items %d: %d\n", nrow, nnz,
                                    s[0], s[1], s[2], L, r);
                        return 1;
                    }
            }
    return 0;
}
"""

STRIDED = r"""
#include <climits>
#include <cstdio>
#include <initializer_list>
#include "index_range.h"
using namespace merbit;

int main() {
    const unsigned stride = 148u * 32u * 256u;  // the largest grid of the conversions
    for (unsigned n : {0u, 1u, stride, (unsigned)INT_MAX - stride, (unsigned)INT_MAX - 1u,
                       (unsigned)INT_MAX, (unsigned)INT_MAX + 1u})
        for (unsigned first : {0u, 1u, 255u, stride - 1u}) {
            unsigned long long calls = 0;
            bool ok = true;
            strided(first, stride, n, [&](int i) {
                ok = ok && i >= 0 && (unsigned)i < n && (unsigned)i == first + calls * stride;
                ++calls;
            });
            const unsigned long long want = n > first ? (n - first + (unsigned long long)stride - 1) / stride : 0;
            if (!ok || calls != want) {
                std::printf("n %u first %u: %llu calls, %llu expected\n", n, first, calls, want);
                return 1;
            }
        }
    return 0;
}
"""

ROWS = r"""
#include <climits>
#include <cstdio>
#include <initializer_list>
#include "index_range.h"
using namespace merbit;

// Every lane of a row group takes the row's entries once and none beyond it.
static bool row(int s, int e, int lpr, int unr) {
    long long taken = 0;
    for (int jl = 0; jl < lpr; ++jl)
        for (unsigned i = (unsigned)(s + jl); before_end(i, 0u, e); i += unr * lpr)
            for (int u = 0; u < unr; ++u)
                if (before_end(i, u * lpr, e)) {
                    const unsigned k = i + u * lpr;
                    if (k < (unsigned)s || k >= (unsigned)e) return false;
                    ++taken;
                }
    return taken == e - s;
}
// ... and a warp those of a staged run of at most 32 * unr.
static bool run(int bs, int be, int unr) {
    long long taken = 0;
    for (int lane = 0; lane < 32; ++lane)
        for (int u = 0; u < unr; ++u)
            if (before_end((unsigned)(bs + lane), 32u * u, be)) {
                const unsigned k = (unsigned)(bs + lane) + 32u * u;
                if (k < (unsigned)bs || k >= (unsigned)be) return false;
                ++taken;
            }
    return taken == be - bs;
}

int main() {
    for (int e : {INT_MAX - 65, INT_MAX - 66, INT_MAX - 300, 1000})
        for (int len : {0, 1, 31, 32, 33, 500, 512})
            for (int unr : {4, 8, 16}) {
                for (int lpr : {1, 2, 4, 8, 16, 32})
                    if (!row(e - len, e, lpr, unr)) return std::printf("row %d of %d, %d lanes\n", e, len, lpr), 1;
                if (len <= 32 * unr && !run(e - len, e, unr)) return std::printf("run %d of %d\n", e, len), 1;
            }
    return 0;
}
"""


def _run(tmp_path, source):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run([cxx, "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover=all", "-I", os.path.join(ROOT, "merbit_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_spmm_walk_at_the_largest_nonzero_count(tmp_path):
    _run(tmp_path, WALK)


def test_grid_stride_loops_at_the_largest_count(tmp_path):
    _run(tmp_path, STRIDED)


def test_row_groups_at_the_largest_nonzero_count(tmp_path):
    _run(tmp_path, ROWS)
