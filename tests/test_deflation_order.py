"""The deflation scan of a divide-and-conquer merge gives the same bits in every order of its threads:
the scan's own source, compiled for the host, runs the maximal runs of close pairs first to
last, last to first and shuffled, and one thread over all pairs.  A run whose look-ahead saw a
neighbour already rotated would miss a conflict in one order and report it in the other."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dirac_caspt2_gb300", "csrc")

DRIVER = r"""
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
namespace dcg { inline double fast_rsqrt(double x) { return 1.0 / std::sqrt(x); } }
using std::fma; using std::fabs; using std::hypot;
#include "dcg_deflate.cuh"
using namespace dcg;

struct Out { std::vector<double> sd, sz, rC, rS; std::vector<int> fold, hm; int conflict; };

// runs in the given order (order < 0: one thread over all pairs)
static Out run(const std::vector<double> &d, const std::vector<double> &z, int n1, double tol, int order, unsigned seed) {
    const int k = (int)d.size();
    std::vector<int> K0(k), close(k, 0);
    for (int m = 0; m < k; m++) K0[m] = m;
    auto source = [&](int i, double &dv, double &zv) { dv = d[i]; zv = z[i]; };
    Out o{d, z, std::vector<double>(k, 0.0), std::vector<double>(k, 0.0), std::vector<int>(k, 0), std::vector<int>(k), 0};
    for (int m = 0; m < k; m++) o.hm[m] = m < n1 ? 1 : 2;
    for (int m = 1; m < k; m++) close[m] = dc_close(d[m] - d[m - 1], z[m - 1], z[m], tol);
    const DeflScan a{K0.data(), close.data(), o.fold.data(), o.hm.data(), o.sd.data(), o.sz.data(), o.rC.data(), o.rS.data(), k, n1, tol};
    auto serial = [&] {
        o.sd = d; o.sz = z;
        std::fill(o.fold.begin(), o.fold.end(), 0);
        for (int m = 0; m < k; m++) o.hm[m] = m < n1 ? 1 : 2;
        if (k > 1) dc_deflate_scan(a, 1, true, source);
    };
    if (order < 0) { serial(); return o; }
    std::vector<int> starts;
    for (int m = 1; m < k; m++) if (close[m] && !close[m - 1]) starts.push_back(m);
    if (order == 1) std::reverse(starts.begin(), starts.end());
    if (order == 2) { std::mt19937 g(seed); std::shuffle(starts.begin(), starts.end(), g); }
    for (int m : starts) if (dc_deflate_scan(a, m, false, source)) o.conflict = 1;
    if (o.conflict) serial();
    return o;
}

static bool same(const Out &x, const Out &y) {
    if (x.fold != y.fold || x.hm != y.hm || x.sd != y.sd || x.sz != y.sz) return false;
    for (size_t m = 0; m < x.fold.size(); m++)
        if (x.fold[m] && (x.rC[m] != y.rC[m] || x.rS[m] != y.rS[m])) return false;
    return true;
}

int main(int argc, char **argv) {
    FILE *f = fopen(argv[1], "rb");
    long cases = 0, conflicts = 0, folds = 0, bad = 0;
    int head[2];
    double tol;
    while (fread(head, sizeof(int), 2, f) == 2 && fread(&tol, sizeof tol, 1, f) == 1) {
        std::vector<double> d(head[0]), z(head[0]);
        if (fread(d.data(), 8, d.size(), f) != d.size() || fread(z.data(), 8, z.size(), f) != z.size()) return 2;
        const Out ref = run(d, z, head[1], tol, -1, 0);
        const Out up = run(d, z, head[1], tol, 0, 0);
        conflicts += up.conflict;
        for (int x : ref.fold) folds += x;
        for (int o = 0; o < 3; o++) {
            const Out v = run(d, z, head[1], tol, o, (unsigned)cases);
            if (!same(v, ref) || v.conflict != up.conflict) { bad++; break; }
        }
        cases++;
    }
    printf("%ld %ld %ld %ld\n", cases, conflicts, folds, bad);
    return 0;
}
"""


def _cases(rng):
    # two runs of which the first one's rotation reaches the second one's start
    yield np.array([0.0, 0.5, 3.5, 203.5]), np.array([100.0, 1.0, 1.0, 1e-3]), 2, 1.0
    for _ in range(4000):
        k = int(rng.integers(2, 40))
        # gaps and components over many magnitudes, so that runs end, touch and fold on
        d = np.cumsum(10.0 ** rng.uniform(-3, 2, size=k))
        z = 10.0 ** rng.uniform(-3, 2, size=k) * rng.choice([-1.0, 1.0], size=k)
        yield d, z, int(rng.integers(0, k + 1)), 10.0 ** rng.uniform(-2, 1)


def test_scan_is_independent_of_thread_order(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    src, exe, data = tmp_path / "scan.cpp", tmp_path / "scan", tmp_path / "cases.bin"
    src.write_text(DRIVER)
    subprocess.run([gxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    with open(data, "wb") as f:
        for d, z, n1, tol in _cases(np.random.default_rng(11)):
            f.write(np.array([len(d), n1], np.int32).tobytes() + np.float64(tol).tobytes() + d.tobytes() + z.tobytes())
    out = subprocess.run([str(exe), str(data)], check=True, capture_output=True, text=True).stdout
    cases, conflicts, folds, bad = map(int, out.split())
    assert cases == 4001 and conflicts > 100 and folds > 10000   # the cases do reach the paths in question
    assert bad == 0
