// Bit strings of the CI space on the host (bit t set: active spinor t occupied).
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace dcg {

// All strings of ne electrons in na spinors, ascending.
inline std::vector<uint64_t> gosper_all(int na, int ne) {
    std::vector<uint64_t> out;
    if (ne < 0 || ne > na || na > 64) return out;
    if (ne == 0) {
        out.push_back(0);
        return out;
    }
    uint64_t cur = (ne == 64) ? ~0ull : ((1ull << ne) - 1ull);
    const uint64_t lim = (na == 64) ? 0 : (1ull << na);
    while (true) {
        out.push_back(cur);
        uint64_t t = (cur | (cur - 1)) + 1;
        uint64_t nxt = t | ((((t & (~t + 1)) / (cur & (~cur + 1))) >> 1) - 1);
        if (nxt <= cur) break;
        if (na < 64 && nxt >= lim) break;
        cur = nxt;
    }
    return out;
}

// Subsets of w spinors with lo to hi electrons, ascending.
inline std::vector<uint64_t> subsets_between(int w, int lo, int hi) {
    std::vector<uint64_t> out;
    for (int n = std::max(lo, 0); n <= std::min(hi, w); n++) {
        const std::vector<uint64_t> g = gosper_all(w, n);
        out.insert(out.end(), g.begin(), g.end());
    }
    std::sort(out.begin(), out.end());
    return out;
}

struct RasSpace {
    int ras1, ras2, ras3;          // spinors of each part, RAS1 in the low bits
    int max_hole, min_hole;        // of RAS1
    int max_elec, min_elec;        // of RAS3
};

// search_cas_configuration.F90:91-110 + ras_det_check.F90:1-59: the bit strings of ne electrons
// with their RAS1 holes and RAS3 electrons in range, ascending, put together from the parts
// RAS3, RAS2 and RAS1 (high to low bits) instead of filtered out of all strings: 10 electrons in
// 8 + 10 + 8 spinors with two holes and two particles are 5.3 million strings, 30 ms on the
// host, of which 74,273 stay.  Each part's numbers of electrons are cut to those that the other
// two can complete to ne, so that every subset made is part of some result: the limits of the
// input may be far wider (28 RAS3 spinors with up to 14 electrons of 2 in all would be 154
// million subsets where a few hundred count).
inline std::vector<uint64_t> ras_strings(int na, int ne, const RasSpace &r) {
    if (ne < 0 || ne > na || na > 64) return {};
    if (!r.ras1 && !r.ras3) return gosper_all(na, ne);
    const int w1 = std::min(std::max(r.ras1, 0), na);              // RAS1: bits 0 .. w1 - 1
    const int sh = r.ras3 ? std::min(r.ras1 + r.ras2, na) : na;    // RAS3: bits sh .. na - 1
    const int w2 = sh - w1, w3 = na - sh;
    if (w2 < 0) return {};
    int lo1 = r.ras1 ? std::max(r.ras1 - r.max_hole, 0) : 0, hi1 = r.ras1 ? std::min(r.ras1 - r.min_hole, w1) : 0;
    int lo3 = r.ras3 ? std::max(r.min_elec, 0) : 0, hi3 = r.ras3 ? std::min(r.max_elec, w3) : 0;
    lo3 = std::max(lo3, ne - w2 - hi1), hi3 = std::min(hi3, ne - lo1);
    lo1 = std::max(lo1, ne - w2 - hi3), hi1 = std::min(hi1, ne - lo3);
    std::vector<uint64_t> out;
    if (lo1 > hi1 || lo3 > hi3) return out;
    std::vector<std::vector<uint64_t>> low(w1 + 1), mid(w3 + 1);
    for (int n = lo1; n <= hi1; n++) low[n] = gosper_all(w1, n);
    for (int n = lo3; n <= hi3; n++) mid[n] = subsets_between(w2, ne - n - hi1, ne - n - lo1);
    for (uint64_t h : subsets_between(w3, lo3, hi3)) {
        const int n3 = __builtin_popcountll(h);
        for (uint64_t m : mid[n3])
            for (uint64_t l : low[ne - n3 - __builtin_popcountll(m)])
                out.push_back((w3 > 0 ? h << sh : 0) | (w2 > 0 ? m << w1 : 0) | l);
    }
    return out;
}

}  // namespace dcg
