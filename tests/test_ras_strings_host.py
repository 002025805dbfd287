"""The CI space's bit strings, from the library's own host source: every small space against a filter of
all strings, and spaces whose RAS limits are far wider than their electrons allow within a
memory limit of 512 MB (their subsets up to the limits alone would take gigabytes)."""
import math
import os
import resource
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dirac_caspt2_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "dcg_strings.h"
using namespace dcg;

static bool kept(uint64_t I, const RasSpace &r) {
    if (r.ras1) {
        const int n1 = __builtin_popcountll(I & ((1ull << r.ras1) - 1));
        if (!(r.ras1 - r.max_hole <= n1 && n1 <= r.ras1 - r.min_hole)) return false;
    }
    if (r.ras3) {
        const int n3 = __builtin_popcountll(I >> (r.ras1 + r.ras2));
        if (!(n3 <= r.max_elec && r.min_elec <= n3)) return false;
    }
    return true;
}

int main(int argc, char **argv) {
    if (argc > 1) {   // the number of strings of one space
        int v[9];
        for (int q = 0; q < 9; q++) v[q] = atoi(argv[q + 1]);
        printf("%zu\n", ras_strings(v[0], v[1], {v[2], v[3], v[4], v[5], v[6], v[7], v[8]}).size());
        return 0;
    }
    long cases = 0, strings = 0, bad = 0;
    for (int na = 0; na <= 9; na++)
        for (int ne = -1; ne <= na + 1; ne++)
            for (int r1 = 0; r1 <= na + 1; r1++)
                for (int r2 = 0; r1 + r2 <= na + 1; r2++)
                    for (int r3 = 0; r3 <= 2; r3++)
                        for (int mh = 0; mh <= 5; mh++)
                            for (int me = 0; me <= 5; me++)
                                for (int lh = -1; lh <= 2; lh++)
                                    for (int le = -1; le <= 2; le++) {
                                        const RasSpace r{r1, r2, r3, mh, lh, me, le};
                                        std::vector<uint64_t> want;
                                        for (uint64_t I : gosper_all(na, ne))
                                            if (kept(I, r)) want.push_back(I);
                                        bad += want != ras_strings(na, ne, r);
                                        cases++;
                                        strings += (long)want.size();
                                    }
    printf("%ld %ld %ld\n", cases, strings, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("ras")
    (d / "ras.cpp").write_text(DRIVER)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", CSRC, str(d / "ras.cpp"), "-o", str(d / "ras")], check=True)
    return str(d / "ras")


def test_small_spaces_against_a_filter(program):
    cases, strings, bad = map(int, subprocess.run([program], check=True, capture_output=True, text=True).stdout.split())
    assert cases > 100000 and strings > 100000
    assert bad == 0


# na, ne, ras1, ras2, ras3, most holes, least holes, most RAS3 electrons, least
WIDE = [((30, 2, 0, 2, 28, 0, 0, 14, 0), math.comb(30, 2)),       # more RAS3 electrons allowed than there are
        ((30, 28, 2, 0, 28, 2, 0, 28, 0), math.comb(30, 28)),     # nearly full: few RAS3 electrons cannot be
        ((30, 2, 28, 2, 0, 28, 0, 0, 0), math.comb(30, 2)),       # as many RAS1 holes as spinors
        ((32, 2, 28, 2, 2, 28, 0, 2, 0), math.comb(32, 2))]


@pytest.mark.parametrize("space,count", WIDE)
def test_wide_limits_cost_no_more_than_their_strings(program, space, count):
    out = subprocess.run([program, *map(str, space)], check=True, capture_output=True, text=True, timeout=60,
                         preexec_fn=lambda: resource.setrlimit(resource.RLIMIT_AS, (512 << 20, 512 << 20))).stdout
    assert int(out) == count
