/* Test helper (compiled by tests/test_voigt_fix.py): the integer arithmetic of
 * fake_spectra_gb300/csrc/fsg_voigt_fix.cuh on the host.  Reads lines of
 * hexadecimal doubles; without an argument "a u1 V w0 .. w6", printing the
 * weighted sum of the Voigt profile over the nodes (i - 3) u1 at V; with the
 * argument "far" "b vmp scale v2 n r1 .. r15", printing the wing's value scale
 * (y + r1 y^2 + ..), n terms, y = (vmp b / (v2 / 2))^2, and |v2| / 2 b. */
#include <cmath>
#include <cstdio>
#include <cstring>

#include "fsg_voigt_fix.cuh"

using namespace fsg;

static const FixRow g_rows[FSG_FIX_ROWS] = FSG_FIX_INIT;
static const Fix62 g_pow2[64] = FSG_FIX_POW2_INIT;
struct Rows {
    FixRow load(int r) const { return g_rows[r]; }
};

static int far_wing()
{
    double b, vmp, scale, v2, n, r[15];
    while (scanf("%la %la %la %la %la", &b, &vmp, &scale, &v2, &n) == 5) {
        for (double &c : r)
            if (scanf("%la", &c) != 1)
                return 1;
        const FixNum ib = fix_num(1.0 / b), vs = fix_num(vmp * vmp), cA = fix_num(scale);
        FixFar f;
        f.vs = vs.m;
        f.ev = vs.e;
        f.cA = cA.m;
        f.eA = cA.e;
        for (int k = 0; k < 15; k++)
            f.A[k] = (int64_t)llrint(ldexp(r[k], 62 + k));
        const FixV v = fix_velocity(v2, ib.m, ib.e);
        int ye, e;
        const uint64_t ym = fix_far_y(f, v, ye);
        const uint64_t m = fix_far_sum(f, (int)n, ym, ye, e);
        printf("%a %a\n", fix_double(m, e, 0), ldexp((double)fix_v53(v), -FIXV_BITS));
    }
    return 0;
}

int main(int argc, char **argv)
{
    if (argc > 1 && !strcmp(argv[1], "far"))
        return far_wing();
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
        int e;
        const uint64_t m = fix_combine(sg, eg, fix_num(exp(a * a)), sk, ek, fix_num(a), e);
        printf("%a\n", fix_double(m, e, 0));
    }
    return 0;
}
