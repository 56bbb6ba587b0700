/* Test helper (compiled by tests/test_spline_edges.py): the integer kernel integral
 * with nodes up to and beyond the edge of the support (fix_spline_sum<true> of
 * fake_spectra_gb300/csrc/fsg_spline_fix.cuh) as the end pixels of an FP32 column
 * density call it.  Reads lines of "cubic h dr2 zrange zlow zhigh" and prints the
 * trapezoid sum of the normalised kernel. */
#include <cmath>
#include <cstdio>

#include "fsg_spline_fix.cuh"

int main()
{
    int cubic;
    double h, dr2, zr, za, zb;
    while (scanf("%d %la %la %la %la %la", &cubic, &h, &dr2, &zr, &za, &zb) == 6) {
        const double inv = 1.0 / h, inv_h = fsg::fix_spline_scale(inv, h, zr);
        const uint64_t B = (uint64_t)llrint(dr2 * inv * inv * 9223372036854775808.0) * 2;
        int e;
        const int64_t s = fsg::fix_spline_sum<true>(cubic != 0, llrint(za * inv_h),
                                                    llrint(zb * inv_h), B, e);
        printf("%a\n", ldexp((double)s, -59 - (cubic ? 3 : 5) * e));
    }
    return 0;
}
