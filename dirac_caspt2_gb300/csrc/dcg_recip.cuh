// Reciprocals and inverse square roots in few FP64 instructions.  A division or a root takes five to
// eight times as long on the FP64 pipe (368 and 615 clocks against 77 an instruction), which is
// what bounds the kernels that use these.
//
// fast_rcp and fast_rsqrt refine the hardware's approximation r (about 20 bits) by one step of the
// binomial series.  With e = 1 - x r, 1/x = r (1 - e)^-1 = r (1 + e + e^2 + ...); with
// e = 1 - x r^2, 1/sqrt(x) = r (1 - e)^(-1/2) = r (1 + e/2 + 3 e^2/8 + ...).  Cut after e^2 the
// rest is of the order of e^3, below 2^-56 of the result, so that rounding decides: within 1 unit
// in the last place for the reciprocal, 1.5 for the root.
#pragma once

namespace dcg {

// 1/x for 2^-959 <= |x| < 2^960 (x, r and the series' terms are normal numbers).  Zero gives NaN, not
// infinity: for callers whose argument cannot leave the range, or who test the result.
__device__ __forceinline__ double fast_rcp(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
// 1/x for any x: a division outside fast_rcp's range (zero, infinity and NaN as there).
__device__ __forceinline__ double safe_rcp(double x) {
    const int ex = (__double2hiint(x) >> 20) & 0x7FF;
    return ex < 64 || ex > 1982 ? 1.0 / x : fast_rcp(x);
}
// 1/sqrt(x) for normal x > 0 (callers guard the ends of the range).
__device__ __forceinline__ double fast_rsqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y, fma(0.375, e, 0.5) * e, y);
}

// 1/e within 2^-46: the FP32 reciprocal r0 of e rounded to FP32, widened and refined by one
// Newton-Raphson step r0 + r0 (1 - e r0), whose relative error is the square of r0's (2^-24 each
// from the two roundings).  A denominator whose FP32 forms would leave the normal numbers takes
// 1.0 / e.  The narrowing cuts the bits and the widening shifts them: as conversions both would
// run on the FP64 pipe.
__device__ __forceinline__ double h_recip(double e) {
    const int hi = __double2hiint(e);
    const int ex = ((hi >> 20) & 0x7FF) - 896;   // exponent field in FP32
    if (ex < 3 || ex > 250) return 1.0 / e;
    // e rounded to 23 fraction bits: half a unit of them added to the bits (a carry goes on into
    // the exponent)
    const uint32_t lo = (uint32_t)__double2loint(e), lo2 = lo + 0x10000000u;
    const uint32_t h2 = (uint32_t)hi + (lo2 < lo ? 1u : 0u);
    const uint32_t m = ((h2 & 0x7FFFFFFFu) - (896u << 20)) << 3 | lo2 >> 29;
    const uint32_t r = __float_as_uint(__frcp_rn(__uint_as_float((h2 & 0x80000000u) | m)));
    const double r0 = __hiloint2double((int)((r & 0x80000000u) | (((r & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(r << 29));
    return fma(r0, fma(-e, r0, 1.0), r0);
}

}  // namespace dcg
