"""The plan of the transform engine's map sweeps (csrc/cov_map_plan.h) for
every cell that the engine accepts, compiled here for the host with traps on
undefined arithmetic: a division by zero, an overflow or a plan outside the
kernels' limits fails.  Among the cells are those that one tile holds, which
have no strip sweep."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "cov_map_plan.h"
#define NEED(x) do { if (!(x)) { printf("q=%d n=%d R=%d: %s\n", q, n, R, #x); return 1; } } while (0)
int main()
{
    int cells = 0, single = 0;
    for (int q = 2; q <= 16; q++)
        for (int n = 1; n <= 16 && map_ipow(q, n) < (1LL << 31); n++)
            for (int R = 0; R <= (n < 8 ? n : 8); R++, cells++) {
                int nb = 0;
                uint32_t blk = 1;
                while (nb < n && (long long)blk * q <= 64) { nb++; blk *= (uint32_t)q; }
                const long long N = map_ipow(q, n);
                MapPlan p;
                map_plan(p, q, n, R, (uint32_t)N, nb, blk);
                NEED(p.kl >= nb && p.kl <= n && p.ng >= 0 && p.ng <= n - p.kl);
                int axes = p.kl;
                for (int i = 0; i < p.ng; i++) {
                    NEED(p.gs[i] >= 1 && p.slots[i] >= 3 && p.slots[i] <= 9);
                    NEED(map_hi(R, axes + p.gs[i]) - map_lo(n, R, axes) + 1 <= p.slots[i]);
                    NEED(map_ipow(q, p.gs[i]) * p.slots[i] * 4 * MAP_W_MIN <= MAP_SMEM_MAX);
                    axes += p.gs[i];
                }
                NEED(axes == n);
                NEED(map_hi(R, p.kl) + 1 <= p.low_slots(R));
                NEED(map_low_smem(q, p.low_slots(R), p.kl, nb, blk) <= MAP_SMEM_MAX);
                NEED(p.at_once >= 1 && p.at_once <= p.parts);
                if (p.ng == 0) {
                    single++;
                    NEED(p.parts == 1 && p.whole_ints == 0);
                } else {
                    const long long cols = N / p.parts / map_ipow(q, p.kl) * map_cols(q, p.kl);
                    NEED(p.parts == (p.ng >= 2 ? map_ipow(q, p.gs[p.ng - 1]) : 1));
                    for (int i = 0; i < std::max(1, p.ng - 1); i++)
                        NEED((long long)p.scratch_ints >= cols * p.at_once * p.slots[i]);
                    if (p.ng >= 2) NEED((long long)p.whole_ints >= cols * p.parts * p.slots[p.ng - 1]);
                }
            }
    printf("%d cells, %d of one tile\n", cells, single);
    return 0;
}
"""


# Where the word counts that a transform may start from lie: the sweeps of a
# part read its own, and nothing that a part leaves in the layers of the last
# sweep reaches the counts of a later one.
COUNTS = r"""
#include <cstdio>
#include "cov_map_plan.h"
#define NEED(x) do { if (!(x)) { printf("q=%d n=%d R=%d: %s\n", q, n, R, #x); return 1; } } while (0)
int main()
{
    int several = 0;
    for (int q = 2; q <= 16; q++)
        for (int n = 1; n <= 16 && map_ipow(q, n) < (1LL << 31); n++)
            for (int R = 0; R <= (n < 8 ? n : 8); R++) {
                int nb = 0;
                uint32_t blk = 1;
                while (nb < n && (long long)blk * q <= 64) { nb++; blk *= (uint32_t)q; }
                const long long N = map_ipow(q, n);
                MapPlan p;
                map_plan(p, q, n, R, (uint32_t)N, nb, blk);
                if (p.ng < 2) {
                    NEED((long long)p.counts_ints >= N);
                    continue;
                }
                NEED(p.counts_ints == 0 && p.counts_at + N <= p.whole_ints);
                const long long T = map_ipow(q, p.kl), Tp = map_cols(q, p.kl), part = N / p.parts / T;
                for (uint32_t k = 0; k < p.parts; k += p.at_once, several++) {
                    const long long t1 = std::min<long long>(k + p.at_once, p.parts) * part;
                    NEED(t1 * Tp * p.slots[p.ng - 1] <= (long long)p.counts_at + t1 * T);
                }
            }
    printf("%d\n", several);
    return several < 100;
}
"""


# A greedy launch in which every placement, and the refresh at the end, comes
# after as many steps of one count each as the kernel allows: it stays within
# the bound at which the kernel gives up, and a launch that went on would not.
STEPS = r"""
#include <cstdio>
#include "cov_map_plan.h"
int main()
{
    for (int room : {1, 2, 7, 1000, 40000})
        for (int eval_cap : {64, 76, 256, 1024}) {
            long long steps = 0;
            for (int placed = 0, since = 0;;) {
                if (placed >= room) break;
                steps++;
                if (since < eval_cap) { since++; continue; }
                placed++;
                since = 0;
            }
            steps += eval_cap + 1;
            if (steps > greedy_max_steps(room, eval_cap) || steps + eval_cap < greedy_max_steps(room, eval_cap)) {
                printf("room=%d eval_cap=%d: %lld steps\n", room, eval_cap, steps);
                return 1;
            }
        }
    return 0;
}
"""


def run_program(tmp_path, text):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(text)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error",
                    "-I", os.path.join(REPO, "coldcase_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout + p.stderr
    return p.stdout.split()


def test_plan_of_every_cell(tmp_path):
    words = run_program(tmp_path, PROGRAM)
    assert int(words[0]) > 300 and 50 < int(words[2]) < int(words[0])


def test_place_of_the_word_counts(tmp_path):
    run_program(tmp_path, COUNTS)


def test_bound_on_the_greedys_steps(tmp_path):
    run_program(tmp_path, STEPS)
