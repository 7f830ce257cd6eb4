"""The geometry of the coverage count's tiles (csrc/cov_tiles_plan.h), compiled
here for the host with traps on undefined arithmetic: every cell that the
count accepts has one within the kernels' limits, and of the geometries with
at most a tile an SM, where a tile of fewer words is less to do for every SM
that works, only the one with the fewest words a tile is taken.  And the rule between
tiles and the transform for a recount takes the way that was measured
faster."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "cov_tiles_plan.h"
#define NEED(x) do { if (!(x)) { printf("q=%d n=%d R=%d M=%d nl=%d: %s\n", q, n, R, M, nl, #x); return 1; } } while (0)

static bool fits(int q, int n, int R, int l)
{
    const int nb = bt_block_digits(n);
    return l >= nb && n - l <= 8 && l - nb <= 8 && bt_ipow(q, l) <= (1 << 20) &&
           bt_smem_bytes(q, n, (uint32_t)bt_ipow(q, l)) <= BT_SMEM_MAX && bt_groups(q, l - nb, R) <= BT_ITEMS;
}

int main()
{
    int cells = 0;
    for (int q = 2; q <= 16; q++)
        for (int n = 1; n <= 16 && bt_ipow(q, n) < (1LL << 32) - 1; n++)
            for (int R = 0; R <= n; R++)
                for (int M : {0, 1, 50, 700, 5000, 20000, 65535, 1 << 20, 1 << 30})
                    for (int sms : {1, 16, 132, 152}) {
                        int nh = 0, nl = 0;
                        bt_geom(q, n, R, M, sms, &nh, &nl);
                        NEED(nl >= 1 && nh + nl == n && fits(q, n, R, nl));
                        if (M > 65535) continue;
                        cells++;
                        for (int l = 1; l < nl; l++)
                            NEED(!fits(q, n, R, l) || bt_ipow(q, n - l) > sms);
                    }
    printf("%d\n", cells);
    return 0;
}
"""


# Recounts of m random words timed both ways on 152 SMs, where one way took at
# least 1.3 times as long as the other: {q, n, R, m, by tiles}.
RECOUNTS = r"""
#include <cstdio>
#include "cov_tiles_plan.h"
static const int cases[][5] = {
    {2, 16, 2, 3000, 1}, {2, 16, 2, 30000, 0}, {3, 13, 2, 3000, 1}, {3, 13, 2, 30000, 0}, {4, 6, 1, 300, 1},
    {4, 11, 1, 10000, 1}, {4, 11, 1, 100000, 0}, {4, 11, 2, 10000, 1}, {4, 11, 2, 100000, 0}, {4, 11, 4, 300, 1},
    {4, 11, 4, 10000, 0}, {5, 9, 1, 3000, 1}, {5, 9, 1, 30000, 0}, {6, 6, 1, 3000, 1}, {6, 6, 1, 30000, 0},
    {6, 6, 3, 300, 1}, {6, 6, 3, 10000, 0}, {6, 9, 1, 10000, 1}, {6, 9, 1, 100000, 0}, {6, 9, 2, 10000, 1},
    {6, 9, 2, 30000, 0}, {6, 9, 4, 3000, 1}, {6, 9, 4, 10000, 0}, {7, 8, 1, 10000, 1}, {7, 8, 1, 100000, 0},
    {7, 8, 2, 10000, 1}, {7, 8, 2, 30000, 0}, {8, 7, 1, 3000, 1}, {8, 7, 1, 30000, 0}, {8, 7, 3, 3000, 1},
    {8, 7, 3, 10000, 0}, {8, 8, 1, 30000, 1}, {8, 8, 1, 100000, 0}, {9, 6, 1, 3000, 1}, {9, 6, 1, 30000, 0},
    {9, 6, 3, 300, 1}, {9, 6, 3, 10000, 0}, {10, 6, 2, 300, 1}, {10, 6, 2, 30000, 0}, {11, 6, 2, 3000, 1},
    {2, 16, 5, 300, 1}, {2, 16, 5, 3000, 0}, {4, 11, 6, 3000, 0}, {6, 9, 6, 3000, 0}, {7, 8, 6, 300, 1},
    {11, 6, 2, 30000, 0}, {13, 5, 2, 300, 1}, {13, 5, 2, 10000, 0}, {16, 5, 2, 300, 1}, {16, 5, 2, 10000, 0}};

int main()
{
    int wrong = 0;
    for (auto &c : cases) {
        const bool tiles = bt_tiles_pay(c[0], c[1], c[2], c[3], 152);
        if (tiles != (c[4] != 0)) { printf("q=%d n=%d R=%d m=%d\n", c[0], c[1], c[2], c[3]); wrong++; }
    }
    return wrong;
}
"""


def run_program(tmp_path, text):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(text)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(REPO, "coldcase_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout + p.stderr
    return p.stdout


def test_geometry_of_every_cell(tmp_path):
    assert int(run_program(tmp_path, PROGRAM)) > 5000


def test_recount_takes_the_faster_way(tmp_path):
    run_program(tmp_path, RECOUNTS)
