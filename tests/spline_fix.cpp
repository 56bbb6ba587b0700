/* Test helper (compiled by tests/test_spline_fix.py): the integer kernel
 * integral of fake_spectra_gb300/csrc/fsg_spline_fix.cuh on the host.  Reads
 * lines of "cubic za zb B" (za, zb in units of h, B = dr2 / h^2) and prints the
 * trapezoid sum of the normalised kernel. */
#include <cmath>
#include <cstdio>

#include "fsg_spline_fix.cuh"

int main()
{
    int cubic;
    double za, zb, B;
    while (scanf("%d %la %la %la", &cubic, &za, &zb, &B) == 4) {
        int e;
        const int64_t s = fsg::fix_spline_sum(cubic != 0, (int64_t)ldexp(za, 62),
                                              (int64_t)ldexp(zb, 62), (uint64_t)ldexp(B, 64), e);
        printf("%a\n", ldexp((double)s, -59 - (cubic ? 3 : 5) * e));
    }
    return 0;
}
