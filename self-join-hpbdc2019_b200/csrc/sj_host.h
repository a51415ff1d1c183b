// Host-side rules of the engine that need no device.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

// Host threads that write the keys of a delivered batch of cnt pairs over n point
// ids: one per half a million ids and pairs.  With every core in the team a small
// batch waits for whichever core is busy with something else; but the loop passes
// over all n run offsets however few pairs the batch has, so those count too.
inline int sj_expand_team(uint64_t n, uint64_t cnt, int threads)
{
    return (int)std::min<uint64_t>((uint64_t)std::max(threads, 1), 1 + (n + cnt) / (1u << 19));
}

// FP32 filter bounds.  Queries are taken relative to their home cell's centre
// (indexed dims) or the data centre (others): |a| <= Ra; candidates lie in the
// home cell or a neighbour: |b| <= Rb.  The kernel evaluates in FP32
//     y = fl(|b|^2 - tLo) + sum_l fl(-2 a_l) b_l     (D+2 roundings),
// with tLo = RD(T - |a|^2 - M).  With u = 2^-24 and r = Ra + Rb:
//   * chain rounding <= (D+2) u (r^2 + T + M),
//   * rounding the local coordinates moves |b - a|^2 by <= 2 u r^2,
//   * the FP64 predicate's own rounding (d2 vs the exact |dx|^2) <= 2^-49 r^2,
// so M = 2 (D+4) u (r^2 + T) + 2^-39 (r^2 + T) exceeds their sum: y <= 0 proves
// d2 <= T.  y >= delta proves d2 > T when delta >= 2M + 2u (T + Ra^2 + M) (the
// second term covers rounding tLo down).  Pairs with 0 < y < delta are
// re-evaluated in FP64.
// pruneT: two boxes of local FP32 coordinates whose squared distance s, in FP32,
// exceeds T + 2M hold no pair that satisfies the predicate: rounding the
// coordinates and the sum moves it by less than (D+6) u r^2 < M, the predicate's
// own rounding by less than M.  Outside the range in which FP32 squares keep
// that accuracy nothing is ruled out.
struct sj_filter_bounds {
    double margin;
    float delta;
    float pruneT;
};

// D dimensions, the first k indexed; thresh: the largest T with sqrt(T) <= eps;
// lo, hi: the data's range per dimension.
inline sj_filter_bounds sj_filter_bounds_of(int D, int k, double eps, double thresh, const double *lo,
                                            const double *hi)
{
    double ra2 = 0, rb2 = 0;
    for (int j = 0; j < D; j++) {
        if (j < k) {
            ra2 += (0.5 * eps * 1.01) * (0.5 * eps * 1.01);
            rb2 += (1.5 * eps * 1.01) * (1.5 * eps * 1.01);
        } else {
            const double h = 0.5 * (hi[j] - lo[j]) * 1.01 + 1e-300;
            ra2 += h * h;
            rb2 += h * h;
        }
    }
    const double r = std::sqrt(ra2) + std::sqrt(rb2);
    const double u = std::ldexp(1.0, -24);
    const double T = thresh;
    sj_filter_bounds b;
    b.margin = 2.0 * (D + 4) * u * (r * r + T) + std::ldexp(r * r + T, -39);
    const double d = (2.0 * b.margin + 2.0 * u * (T + ra2 + b.margin)) * (1.0 + std::ldexp(1.0, -20));
    float df = (float)d;
    if ((double)df < d) df = std::nextafter(df, INFINITY);
    b.delta = df;
    b.pruneT = INFINITY;
    if (eps >= 1e-15 && eps <= 1e15) {
        const double pt = (T + 2.0 * b.margin) * (1.0 + std::ldexp(1.0, -20));
        if (pt < 3.0e38) b.pruneT = std::nextafter((float)pt, INFINITY);
    }
    return b;
}
