// The pair rotations of a divide-and-conquer merge's deflation (Dongarra & Sorensen, SIAM J. Sci.
// Stat. Comput. 8 (1987) s139): the criterion, one rotation, and the scan of a run of close
// poles.  Plain functions of their arguments, so that a host program can run the scan with its
// threads in any order.  fast_rsqrt comes from the including file.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define DCG_DEFL __device__ __forceinline__
#else
#define DCG_DEFL inline
#endif

namespace dcg {

// Whether the rank-one components zp, zn of neighbouring poles a distance t apart combine into
// one by a rotation (|t c s| <= tol for c = zn / |z|, s = zp / |z|), without a division.
DCG_DEFL bool dc_close(double t, double zp, double zn, double tol) {
    return fabs(t * zp * zn) <= tol * fma(zp, zp, zn * zn);
}

// One pair rotation of the deflation scan: component zp folds into zn.
DCG_DEFL void dc_rotate(double &dp, double zp, double &dn, double &zn, double &C, double &S) {
    const double t2 = fma(zn, zn, zp * zp), a = dp, c = dn;
    if (t2 > 1e-280) {
        const double ri = fast_rsqrt(t2);
        C = zn * ri;
        S = -zp * ri;
        zn = t2 * ri;
    } else {   // the squares are out of range
        const double tt = hypot(zn, zp);
        C = zn / tt;
        S = -zp / tt;
        zn = tt;
    }
    dp = a * C * C + c * S * S;
    dn = a * S * S + c * C * C;
}

// The kept entries of a node in merged order.  close, K0 and the unrotated values (`orig`) do not
// change while the runs are scanned; a scan writes the entries from its run's start up to the
// next run's start, and nobody else's.
struct DeflScan {
    const int *K0;      // node-local column of each entry
    const int *close;   // close[m]: the pair (m - 1, m) qualifies for a rotation on unrotated values
    int *fold;          // fold[m]: entry m was folded into m + 1 (zero before)
    int *hm;            // halves of the node each entry's column reaches (bit 0 first, bit 1 second)
    double *sd, *sz;    // poles and components by column, rotated in place
    double *rC, *rS;    // rotation of each folded entry
    int k0, n1;         // entries, columns of the first half
    double tol;
};

// Scan from the pair (m - 1, m).  One run (whole = false): from its start until a test past its end
// fails; true when a rotation would change the start of the next run, nothing of which has been
// written then.  An entry behind the run's end may be that start, which another thread rotates at
// the same time: it is read from its unrotated source, orig(column, pole, component), so the
// outcome does not depend on the order of the threads.  whole: all pairs, by one thread.
template <class Orig>
DCG_DEFL bool dc_deflate_scan(const DeflScan &a, int m, bool whole, const Orig &orig) {
    int pj = a.K0[m - 1], hp = a.hm[m - 1];
    double dp = a.sd[pj], zp = a.sz[pj];
    bool dirty = false;   // entry m - 1 carries rotated values
    for (; m < a.k0; m++) {
        const int nj = a.K0[m];
        const bool inrun = a.close[m] != 0;
        if (!whole && !inrun && !dirty) break;   // past the run's end
        double dn, zn, C, S;
        int hn;
        if (whole || inrun) {
            dn = a.sd[nj], zn = a.sz[nj], hn = a.hm[m];
        } else {
            orig(nj, dn, zn);
            hn = nj < a.n1 ? 1 : 2;
        }
        if (dc_close(dn - dp, zp, zn, a.tol)) {
            // folding into an entry whose own pair starts the next run
            if (!whole && !inrun && m + 1 < a.k0 && a.close[m + 1]) return true;
            dc_rotate(dp, zp, dn, zn, C, S);
            a.rC[m - 1] = C;
            a.rS[m - 1] = S;
            a.sd[pj] = dp;
            a.fold[m - 1] = 1;
            hn |= hp;
            a.hm[m - 1] = hn;   // a folded column mixes both as well
            dirty = true;
            a.sd[nj] = dn;
            a.sz[nj] = zn;
            a.hm[m] = hn;
        } else {
            dirty = false;
            if (!whole && !inrun) break;
        }
        pj = nj;
        dp = dn;
        zp = zn;
        hp = hn;
    }
    return false;
}

}  // namespace dcg
