/* Test helper (compiled by tests/test_voigt_fix.py): the integer node sums of
 * fake_spectra_gb300/csrc/fsg_voigt_fix.cuh on the host.  Reads lines of
 * "a u1 V w0 .. w6" (hexadecimal doubles) and prints the weighted sum of the
 * Voigt profile over the nodes (i - 3) u1 at V. */
#include <cmath>
#include <cstdio>

#include "fsg_voigt_fix.cuh"

using namespace fsg;

static const FixRow g_rows[FSG_FIX_ROWS] = FSG_FIX_INIT;
static const Fix62 g_pow2[64] = FSG_FIX_POW2_INIT;
struct Rows {
    FixRow load(int r) const { return g_rows[r]; }
};

int main()
{
    double a, u1, V, w[7];
    while (scanf("%la %la %la %la %la %la %la %la %la %la", &a, &u1, &V, w, w + 1, w + 2, w + 3,
                 w + 4, w + 5, w + 6) == 10) {
        FixPair p;
        fix_pair_damping(a, p);
        p.u1 = (int64_t)ldexp(u1, FIXV_BITS);
        for (int i = 0; i < 7; i++)
            p.w[i] = fix62(w[i] >= 1.0 ? ~0ull : (uint64_t)ldexp(w[i], 64));
        int64_t sg, sk;
        int eg, ek;
        fix_node_sums(p, (int64_t)ldexp(V, FIXV_BITS), Rows(), g_pow2, sg, eg, sk, ek);
        printf("%a\n", ldexp((double)sg, -60 - eg) * exp(a * a) +
                           a * ldexp((double)sk, -60 - ek));
    }
    return 0;
}
