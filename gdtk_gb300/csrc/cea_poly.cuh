// cea_poly.cuh -- compares of doubles on the integer pipe and the NASA-9 curves in polynomial form, for the kernels
// compiled at run time (chem_fast.cuh, chem_group.cuh) and the two-temperature kernels.  Needs fast_exp.h.
#pragma once

#define GDTK_TH_STRIDE 120
#define GDTK_TH_SEG0 24

namespace gdtk_fast {

using gdtk::gdtk_exp;
using gdtk::gdtk_div;
using gdtk::gdtk_rcp;
using gdtk::gdtk_log;

enum { ST_OK = 0, ST_H_MIN = 1, ST_MAX_ATTEMPTS = 2, ST_MAX_SUBCYCLES = 3, ST_NEWTON = 4, ST_BAD = 5, ST_FROZEN = 6,
       ST_CEA = 7 };

// ---------------------------------------------------------------- compares on the integer pipe
// An FP64 compare (DSETP) takes an FP64 issue slot, as costly as an FMA on this GPU, while the
// bit patterns of doubles can be compared on the integer pipe: for doubles of the same sign the
// patterns order like the values.  Each helper below gives exactly the IEEE result, NaN included,
// for the operands its comment allows; the kernel's hot loops compare through them.
constexpr long long ABS_BITS = 0x7fffffffffffffffLL;
constexpr long long INF_BITS = 0x7ff0000000000000LL;
__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }
// x < c, any x, c > 0 finite
__device__ __forceinline__ bool lt_pos(double x, double c) {
    const long long b = dbits(x);
    return b < dbits(c) && (b >= 0 || (b & ABS_BITS) <= INF_BITS);
}
// x > c, any x, c >= 0 finite
__device__ __forceinline__ bool gt_pos(double x, double c) {
    const long long b = dbits(x);
    return b > dbits(c) && b <= INF_BITS;
}
// x >= c, any x, c > 0 finite
__device__ __forceinline__ bool ge_pos(double x, double c) {
    const long long b = dbits(x);
    return b >= dbits(c) && b <= INF_BITS;
}
// fmin(x, c), any x, c > 0 finite
__device__ __forceinline__ double min_pos(double x, double c) { return lt_pos(x, c) ? x : c; }
// a > b for a, b >= +0 or NaN of either sign (not -0.0)
__device__ __forceinline__ bool gt_nn(double a, double b) {
    const unsigned long long ua = (unsigned long long)dbits(a), ub = (unsigned long long)dbits(b);
    return ua > ub && ua <= (unsigned long long)INF_BITS && ub <= (unsigned long long)INF_BITS;
}
// a >= b for a, b >= +0 or NaN of either sign (not -0.0)
__device__ __forceinline__ bool ge_nn(double a, double b) {
    const unsigned long long ua = (unsigned long long)dbits(a), ub = (unsigned long long)dbits(b);
    return ua >= ub && ua <= (unsigned long long)INF_BITS && ub <= (unsigned long long)INF_BITS;
}
// x != 0.0 (either sign of zero), any x
__device__ __forceinline__ bool nonzero(double x) { return (dbits(x) & ABS_BITS) != 0; }
// |x| as a double with the sign bit cleared (an integer operation)
__device__ __forceinline__ double abs_bits(double x) { return __longlong_as_double(dbits(x) & ABS_BITS); }
// fmax(|a|, |b|), any a, b
__device__ __forceinline__ double larger_abs(double a, double b) {
    const double x = abs_bits(a), y = abs_bits(b);
    return (dbits(y) > dbits(x) && dbits(y) <= INF_BITS) || dbits(x) > INF_BITS ? y : x;
}
// ---------------------------------------------------------------- species thermo
// Segment choice of cea_thermo_curves.d:150-182: coefficients sa blended towards sb by wb.
// th[10] holds the segment count as integer bits; th[10 + i] and th[13 + i] the blend window
// [break_i - blend_{i-1}/2, break_i + blend_{i-1}/2] around break i (i = 1..nseg-1, formed on the
// host with the reference's arithmetic), th[16 + i] 1 / blend_{i-1}.  The bounds are positive, so
// for any T but NaN (rejected first) the compares are exact on the bit patterns.
__device__ __forceinline__ bool seg_of(const double* th, double T, int& sa, int& sb, double& wb) {
    const int nseg = (int)dbits(th[10]);
    const long long t = dbits(T);
    wb = 0.0;
    if ((t & ABS_BITS) > INF_BITS) return false;   // NaN
    if (nseg == 1) { sa = sb = 0; return true; }
    if (t < dbits(th[11])) { sa = sb = 0; return true; }
    if (t > dbits(th[12 + nseg])) { sa = sb = nseg - 1; return true; }
    for (int i = 1; i < nseg; ++i) {
        const long long lo = dbits(th[10 + i]), hi = dbits(th[13 + i]);
        if (t >= lo && t <= hi) { wb = th[16 + i] * (T - th[10 + i]); sa = i - 1; sb = i; return true; }
        if (t > hi && i < nseg - 1 && t < dbits(th[11 + i])) { sa = sb = i; return true; }
    }
    sa = sb = 0;
    return false;
}

__device__ __forceinline__ double poly_H(const double* c, double T, double lnT, double rT) {   // H/R [K]
    return fma(T, fma(T, fma(T, fma(T, fma(T, c[6], c[5]), c[4]), c[3]), c[2]), fma(c[0], rT, fma(c[1], lnT, c[7])));
}
__device__ __forceinline__ double poly_Cp(const double* c, double T, double rT, double rT2) {   // Cp/R
    return fma(T, fma(T, fma(T, fma(T, c[6], c[5]), c[4]), c[3]), fma(c[0], rT2, fma(c[1], rT, c[2])));
}
__device__ __forceinline__ double poly_G(const double* c, double T, double rT, double rT2, double t1, double t2) {
    // G/RT = g0/T^2 + (g1 (ln T + 1) + g2)/T + g3 (1 - ln T) + g4 + T (g5 + T (g6 + T (g7 + T g8)))
    return fma(T, fma(T, fma(T, fma(T, c[8], c[7]), c[6]), c[5]),
               fma(fma(c[1], t1, c[2]), rT, fma(c[0], rT2, fma(c[3], t2, c[4]))));
}

// H/R and Cp/R of species i (extrapolated with constant Cp beyond the curve, as the reference).
__device__ __forceinline__ void sp_H_Cp(const double* TH, int i, double T, double lnT, double rT, double rT2, double& H,
                                        double& Cp, int& err) {
    const double* th = TH + i * GDTK_TH_STRIDE;
    if (lt_pos(T, th[0])) { H = th[2] - th[4] * (th[0] - T); Cp = th[4]; return; }
    if (gt_pos(T, th[1])) { H = th[3] + th[5] * (T - th[1]); Cp = th[5]; return; }
    int sa, sb;
    double wb;
    if (!seg_of(th, T, sa, sb, wb)) { err = ST_CEA; H = 0.0; Cp = 1.0; return; }
    const double* ca = th + GDTK_TH_SEG0 + 24 * sa;
    H = poly_H(ca, T, lnT, rT);
    Cp = poly_Cp(ca + 8, T, rT, rT2);
    if (nonzero(wb)) {
        const double* cb = th + GDTK_TH_SEG0 + 24 * sb;
        H = fma(wb, poly_H(cb, T, lnT, rT) - H, H);
        Cp = fma(wb, poly_Cp(cb + 8, T, rT, rT2) - Cp, Cp);
    }
}

__device__ __noinline__ double sp_G(const double* TH, int i, double T, double lnT, double rT, double rT2, double t1,
                                       double t2, int& err) {
    const double* th = TH + i * GDTK_TH_STRIDE;
    if (lt_pos(T, th[0])) {
        double H = th[2] - th[4] * (th[0] - T), S = th[6] - th[4] * (th[8] - lnT);
        return fma(H, rT, -S);
    }
    if (gt_pos(T, th[1])) {
        double H = th[3] + th[5] * (T - th[1]), S = th[7] + th[5] * (lnT - th[9]);
        return fma(H, rT, -S);
    }
    int sa, sb;
    double wb;
    if (!seg_of(th, T, sa, sb, wb)) { err = ST_CEA; return 0.0; }
    double g = poly_G(TH + i * GDTK_TH_STRIDE + GDTK_TH_SEG0 + 24 * sa + 15, T, rT, rT2, t1, t2);
    if (nonzero(wb)) g = fma(wb, poly_G(TH + i * GDTK_TH_STRIDE + GDTK_TH_SEG0 + 24 * sb + 15, T, rT, rT2, t1, t2) - g, g);
    return g;
}

// ln(T (1 + x)) from ln T: ln T + log1p(x) by its Taylor series to x^6 when |x| < 2^-10 (the
// truncation is below 2^-60 |x|), else a fresh log.  The kernel carries ln T with each cell this way,
// because a library log costs as much FP64 issue as about 36 FMAs.
// Below 2^-20, where every Newton iteration but the first lies, x^3 is enough (2^-62 |x|).
__device__ __forceinline__ double ln_step(double lnT, double x, double T) {
    if ((dbits(x) & ABS_BITS) < dbits(0x1p-20)) return fma(x, fma(x, fma(x, 1.0 / 3.0, -0.5), 1.0), lnT);
    if ((dbits(x) & ABS_BITS) < dbits(0x1p-10))
        return lnT + x * fma(x, fma(x, fma(x, fma(x, fma(x, -1.0 / 6.0, 0.2), -0.25), 1.0 / 3.0), -0.5), 1.0);
    return gdtk_log(T);
}

}  // namespace gdtk_fast
