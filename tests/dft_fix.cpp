/* Test helper (compiled by tests/test_dft_fix.py): fixed-point transforms of
 * fake_spectra_gb300/csrc/fsg_dft_fix.cuh on the host.  Arguments: "dif" or "dit"
 * and the radices; input: the points as pairs of doubles, the table of
 * exp(-2 pi i k / n) as pairs.  Prints the transform (natural order) / n^(1/2)
 * rounded up to a power of two. */
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "fsg_dft_fix.cuh"

using namespace fsg;

template <int R>
static void pass(bool dif, FixC *x, const FixW *tw, unsigned n, unsigned m, int e)
{
    for (unsigned f = 0; f < n / R; f++)
        if (dif || m == 1)      // adjacent points: no twiddles either way
            dif_butterfly<R>(x, tw, f, m, e);
        else
            dit_butterfly<R>(x, tw, f, m, e);
}

int main(int argc, char **argv)
{
    const bool dif = !strcmp(argv[1], "dif");
    std::vector<int> radix;
    unsigned n = 1;
    for (int i = 2; i < argc; i++) {
        radix.push_back(atoi(argv[i]));
        n *= radix.back();
    }
    std::vector<double> in(2 * n), root(2 * n);
    for (double &v : in)
        if (scanf("%la", &v) != 1)
            return 1;
    for (double &v : root)
        if (scanf("%la", &v) != 1)
            return 1;
    std::vector<unsigned> m(radix.size()), freq(n);
    unsigned rest = n;
    for (size_t i = 0; i < radix.size(); i++)
        m[i] = rest /= radix[i];
    for (unsigned p = 0; p < n; p++) {
        unsigned r = p, k = 0, mul = 1;
        for (size_t i = 0; i < radix.size(); i++) {
            k += r / m[i] * mul;
            r %= m[i];
            mul *= radix[i];
        }
        freq[p] = k;
    }
    std::vector<FixC> x(n);
    for (unsigned p = 0; p < n; p++) {
        const unsigned q = dif ? p : freq[p];
        x[p] = {fix_from_double(in[2 * q], 60), fix_from_double(in[2 * q + 1], 60)};
    }
    double bits = 0;
    int done = 0;
    for (size_t s = 0; s < radix.size(); s++) {
        const size_t i = dif ? s : radix.size() - 1 - s;
        if (dif)
            bits += 0.5 * log2(radix[i]);
        std::vector<FixW> tw((radix[i] - 1) * m[i]);
        for (int q = 1; q < radix[i]; q++)
            for (unsigned j = 0; j < m[i]; j++) {
                const unsigned k = j * q * (n / (m[i] * radix[i]));
                tw[(q - 1) * m[i] + j] = {fix_v62(root[2 * k]), fix_v62(root[2 * k + 1])};
            }
        int e = (int)ceil(bits - 1e-9) - done;
        e = m[i] == 1 ? 0 : e < 1 ? 1 : e;
        done += e;
        switch (radix[i]) {
        case 2: pass<2>(dif, x.data(), tw.data(), n, m[i], e); break;
        case 3: pass<3>(dif, x.data(), tw.data(), n, m[i], e); break;
        case 4: pass<4>(dif, x.data(), tw.data(), n, m[i], e); break;
        case 5: pass<5>(dif, x.data(), tw.data(), n, m[i], e); break;
        case 7: pass<7>(dif, x.data(), tw.data(), n, m[i], e); break;
        case 8: pass<8>(dif, x.data(), tw.data(), n, m[i], e); break;
        default: pass<16>(dif, x.data(), tw.data(), n, m[i], e);
        }
        if (!dif)
            bits += 0.5 * log2(radix[i]);
    }
    std::vector<FixC> y(n);
    for (unsigned p = 0; p < n; p++)
        y[dif ? freq[p] : p] = x[p];
    for (unsigned k = 0; k < n; k++)
        printf("%a %a\n", fix_to_double(y[k].x, done - 60), fix_to_double(y[k].y, done - 60));
    return 0;
}
