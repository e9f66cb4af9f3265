"""Launch plan of a batch (CPU): csrc/tube_plan.h, compiled with the host
compiler.  Whatever cluster sizes a device refuses, every problem is launched
exactly once, on a cluster that holds it or in the persistent kernel."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "tube_plan.h"
// sm_count, refused sizes as a bit mask (1, 2, 4, 8, 16), problem sizes, largest first
int main(int argc, char **argv) {
    const int sms = atoi(argv[1]), mask = atoi(argv[2]);
    std::vector<int> n;
    for (int i = 3; i < argc; ++i) n.push_back(atoi(argv[i]));
    std::vector<int> seen(n.size(), 0), size(n.size(), -1);
    bool fits = true, calls = true;
    int last = -1;
    const bool ok = cumc::run_plan(cumc::tube_plan(n, sms),
        [&](const cumc::TubeLaunch &l) {
            if (l.size & mask) return false;
            for (int p = l.first; p < l.first + l.count; ++p) {
                ++seen[p];
                size[p] = l.size;
                fits = fits && n[p] <= l.size * (l.wide ? 254 : 126);
            }
            return true;
        },
        [&](int first, int count) {
            calls = calls && first > last && count > 0;  // neighbours were joined
            last = first + count;
            for (int p = first; p < first + count; ++p) { ++seen[p]; size[p] = 0; }
            return true;
        });
    bool once = true;
    for (int s : seen) once = once && s == 1;
    printf("%d %d %d %d", ok, fits, calls, once);
    for (int s : size) printf(" %d", s);
    printf("\n");
}
"""

MIXED = [5000, 4065, 4064, 2033, 2032, 2017, 2016, 1017, 1016, 1009, 1008, 600, 508, 255, 254, 127, 126, 16, 3, 1]


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = str(d / "t.cpp"), str(d / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "cumc3d_b200", "csrc"), src, "-o", exe], check=True)

    def run(sms, mask, sizes):
        out = subprocess.run([exe, str(sms), str(mask)] + [str(n) for n in sizes], capture_output=True, text=True,
                             check=True).stdout.split()
        assert out[:4] == ["1", "1", "1", "1"], (sms, mask, out[:4])
        return [int(v) for v in out[4:]]
    return run


@pytest.mark.parametrize("mask", [0, 16, 8, 24, 4, 20, 1, 2, 31])
@pytest.mark.parametrize("sms", [148, 16, 1])
def test_every_problem_runs_once(plan, sms, mask):
    for sizes in (MIXED, sorted(MIXED * 12, reverse=True), [800], [2032, 1500], [4064], [1]):
        got = plan(sms, mask, sizes)
        assert not any(s and s & mask for s in got)
        assert all(s == 0 for n, s in zip(sizes, got) if n > 4064)


def test_refused_class_that_is_no_prefix(plan):
    """In a small batch 2017 to 2032 cells take 8 CTAs of 254 and come before
    1009 to 2016 on 16 of 126: a device without 16-CTA clusters still runs both."""
    assert plan(148, 0, [2032, 1500]) == [8, 16]
    assert plan(148, 16, [2032, 1500]) == [8, 0]
