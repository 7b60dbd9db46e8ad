"""The size of a column grid (rs_pim.cu, grid_cells to grid_size, built here as they stand): scenes
of many small and of large boxes, long and flat ones, bounds and areas beyond a float's range,
up to 2^31 triangles.  No place of the boxes in the cells lists 2^32 entries, the number expected
stays within the budget, and ordinary scenes keep the size that grid_cells gives."""
import os
import re
import shutil
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rayspace3d_gb300", "csrc", "rs_pim.cu")

MAIN = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
SOURCE
static int bad = 0;
// n boxes of bw x bh (fractions of the bounds) in bounds of w x h
static void check(double n, double w, double h, double bw, double bh) {
    const double area1 = w * bw * h * bh;
    const double sum[3] = {n * w * bw, n * h * bh, area1 < 3.4e38 ? n * area1 : 0.0};
    const GridSize g = grid_size(n, w, h, sum);
    const double cu = g.gu * bw, cv = g.gv * bh;  // a box in cells
    const double expected = n * (cu + 1) * (cv + 1), most = n * std::min(cu + 2, (double)g.gu) * std::min(cv + 2, (double)g.gv);
    const double budget = std::max(kEntries * n, kFree);
    const bool one = g.gu == 1 && g.gv == 1;
    const bool safe = n >= 1073741824.0 ? n * (1 + cu) * (1 + cv) < 4294967296.0 || one : most < 4294967296.0;
    if (g.gu < 1 || g.gv < 1 || g.gu > 8192 || g.gv > 8192 || !(one || expected <= 2.01 * budget) || !safe) {
        std::printf("n %g bounds %g x %g boxes %g x %g: %d x %d, %g expected, %g at most\n", n, w, h, bw, bh, g.gu, g.gv, expected, most);
        ++bad;
    }
}
int main() {
    for (double n = 1; n < 2147483648.0; n *= 3.7)
        for (double aspect = 1e-7; aspect < 2e7; aspect *= 31)
            for (double size : {1.0, 1e-6, 1e6, 1e18, 1e30})
                for (double bw : {0.0, 1e-5, 1e-3, 0.03, 0.3, 1.0})
                    for (double bh : {0.0, 1e-5, 1e-3, 0.03, 0.3, 1.0}) check(n, size * aspect, size, bw, bh);
    for (double n : {1.0, 1e3, 1e6, 1e9})  // flat bounds
        for (double b : {0.0, 1e-4, 0.1, 1.0}) {
            check(n, 5.0, 0.0, b, 0.0);
            check(n, 0.0, 5.0, 0.0, b);
            check(n, 0.0, 0.0, 0.0, 0.0);
        }
    for (double n : {1e3, 1e6, 1e8, 9e8, 2e9}) {  // bounds without end
        const double sum[3] = {0.0, n * 1.0, 0.0};
        const GridSize g = grid_size(n, INFINITY, 4.0, sum), e = grid_size(n, INFINITY, INFINITY, sum);
        if (g.gu != 1 || g.gv < 1 || n * std::min(g.gv / 4.0 + 2, (double)g.gv) >= 4294967296.0 || e.gu * e.gv != 1)
            ++bad, std::printf("endless: %d x %d\n", g.gu, g.gv);
    }
    // Ordinary scenes: what the shape of grid_cells' own number is.
    for (double n : {320.0, 5120.0, 81920.0, 6.4e6})
        for (double b : {1e-4, 1e-3, 0.02}) {
            const double sum[3] = {n * b, n * b, n * b * b};
            const GridSize g = grid_size(n, 1.0, 1.0, sum), s = grid_shape(grid_cells(n, 1.0, 1.0, sum), 1.0, 1.0);
            if (g.gu != s.gu || g.gv != s.gv) ++bad, std::printf("ordinary: n %g box %g\n", n, b);
        }
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_grid_size(tmp_path):
    text = open(SRC).read()
    m = re.search(r"constexpr double kEntries = .*?(?=\ntemplate <int AXIS>\ncudaError_t build_grid)", text, re.S)
    (tmp_path / "main.cpp").write_text(MAIN.replace("SOURCE", m[0]))
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[:4000]
