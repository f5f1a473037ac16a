// screen_rule.cuh -- how many pairs the tensor form's screen (scan_mma.cu) is expected to pass on,
// which decides whether a scan is screened (epi_scan on the host, epi_scan_block_noalloc on the
// device) and into how many lists or parts.
//
// For unassociated genotypes SSB and SSI are about sigma^2 times chi-squared with 8 and 4 degrees of
// freedom. A pair is passed on when its root is within R = E / sigma of the threshold's, or of the
// largest lower bound so far, itself R below the largest of all pairs' draws.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace epi {

// upper tail of the chi-squared distribution with 8 or 4 degrees of freedom
__host__ __device__ inline double chi_tail(double x, int df)
{
    const double h = 0.5 * x;
    return exp(-h) * (df == 4 ? 1.0 + h : 1.0 + h * (1.0 + h / 2.0 * (1.0 + h / 3.0)));
}

// root of the largest of `pairs` draws of it, about (bisection; the tail falls from 1)
inline double chi_top(double pairs, int df)
{
    const double p = pairs > 2.0 ? 1.0 / pairs : 0.5;
    double lo = 0.0, hi = 1500.0;
    for (int k = 0; k < 60; ++k) {
        const double mid = 0.5 * (lo + hi);
        (chi_tail(mid, df) > p ? lo : hi) = mid;
    }
    return sqrt(lo);
}

// The share of a trait's pairs that the test with df = 8 or 4 passes on: nv valid individuals, R = r, top
// from chi_top, thr the threshold of F where the trait's hits are reported.
__host__ __device__ inline double screen_share_of(double thr, bool report, int df, double top, double r, double nv)
{
    double root = top > r ? top - r : 0.0;
    if (report) {
        if (!(thr > 0.0)) return 1.0;
        const double d2 = nv > 10.0 ? nv - 9.0 : 1.0, x = sqrt(df * thr * nv / (d2 + df * thr));
        root = x < root ? x : root;
    }
    root = root > r ? root - r : 0.0;
    return chi_tail(root * root, df);
}

}  // namespace epi
