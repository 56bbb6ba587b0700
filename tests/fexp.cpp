/* Test helper (compiled by tests/test_fexp.py): exp(s t) of
 * fake_spectra_gb300/csrc/fsg_fexp.cuh on the host, for arguments whose result is a
 * normal double.  Reads lines "s t" of hexadecimal doubles. */
#include <cmath>
#include <cstdio>

#include "fsg_fexp.cuh"

int main()
{
    using namespace fsg;
    static uint64_t tab[EXP_TABLE];
    for (int k = 0; k < EXP_TABLE; k++)
        tab[k] = (uint64_t)(std::exp2l(63.0L - (long double)k / EXP_TABLE) + 0.5L);
    double s, t;
    while (scanf("%la %la", &s, &t) == 2) {
        const ExpScale sc = exp_scale(s);
        const int64_t b = exp_bits(t);
        int n;
        const uint64_t f = exp_split(b, 62 + 1023 - ((int)(b >> 52) & 0x7FF) - sc.es, sc, n);
        const uint64_t v = exp2_neg_frac(f, tab);
        printf("%a\n", exp_double((int64_t)((v + 512) >> 10) + ((int64_t)(1021 - n) << 52)));
    }
    return 0;
}
