"""The geometry of the coverage count's tiles (csrc/cov_tiles_plan.h), compiled
here for the host with traps on undefined arithmetic: every cell that the
count accepts has one within the kernels' limits, and of the geometries with
at most a tile an SM, where a tile of fewer words is less to do for every SM
that works, only the one with the fewest words a tile is taken."""
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


def test_geometry_of_every_cell(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(REPO, "coldcase_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout + p.stderr
    assert int(p.stdout) > 5000
