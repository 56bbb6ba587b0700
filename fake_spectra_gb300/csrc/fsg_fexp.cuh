// exp(s t) for the flux-statistics passes, in 64-bit integer arithmetic.
//
// This GPU runs FP64 at 1/64 of the FP32 rate: a table-driven FP64 exponential
// took ten FP64 operations (the time of 160 others on the SM) and bound every
// flux pass.  Here |s t| log2(e) = n + f is one 64 x 64-bit product of the
// mantissas (the product with log2(e) is taken once, in ExpScale), and
//     2^-f = T[k] (1 - q(x)),  k = top 10 bits of f, x = the rest in [0, 1),
//     q = c1 x - c2 x^2 + c3 x^3 - c4 x^4,  c_m = (ln 2 / 1024)^m / m!
// (the next term is below 2^-59), with T[k] = 2^(-k/1024) to 63 bits.  f is
// held to 2^-54 or better, the value to 2^-55, and one rounding makes the
// double.  A positive argument uses 2^(n+f) = 2^-((-n-1) + (1-f)): the
// complement of both.  Within about one ulp of exp (tested against CUDA's exp
// and numpy's).  Flux PDF and power of 3600 x 6691 pixels at a fixed mean flux:
// 11.6 ms with the FP64 exponential, 8.3 ms so (with the same FP64 transforms).
//
// tab: T[k] in units of 2^-63, k < EXP_TABLE (exp_table_host computes it).
#pragma once

#include "fsg_voigt_fix.cuh"

namespace fsg {

constexpr int EXP_TABLE = 1024;
constexpr double EXP_LN2 = 0.693147180559945309417232121458;

// exp(s t) = 2^-(n + f): |s t| log2(e) = P 2^(et + es - 62), P the upper word of
// the product of t's mantissa (63 - 52 bits up) with m.
struct ExpScale {
    uint64_t m;       // mantissa of |s| log2(e), upper bit set
    int es;           // s log2(e) = m 2^(es - 63)
    int64_t neg;      // sign bit of s in bit 63
    bool finite;
};

FSG_HD int64_t exp_bits(double d)
{
#ifdef __CUDA_ARCH__
    return __double_as_longlong(d);
#else
    int64_t b;
    __builtin_memcpy(&b, &d, 8);
    return b;
#endif
}

FSG_HD double exp_double(int64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double d;
    __builtin_memcpy(&d, &b, 8);
    return d;
#endif
}

FSG_HD ExpScale exp_scale(double s)
{
    const int64_t b = exp_bits(s);
    uint64_t man = (uint64_t)b & 0xFFFFFFFFFFFFFull;
    int e = (int)((b >> 52) & 0x7FF);
    ExpScale r;
    r.finite = e != 0x7FF;
    r.neg = b;
    if (e)
        man |= 1ull << 52;
    else
        e = 1;
    if (man == 0) {                       // s = 0: far below every t
        r.m = 1ull << 63;
        r.es = -4000;
        return r;
    }
    while (!(man >> 52)) {
        man <<= 1;
        e--;
    }
    // log2(e) = FSG_FIX_LOG2E 2^-63 in [1, 2)
    const uint64_t p = fix_umulhi64(man << 11, FSG_FIX_LOG2E);   // 2^-62
    const uint64_t lo = (man << 11) * FSG_FIX_LOG2E;
    r.es = e - 1023 + (int)(p >> 63);
    r.m = p >> 63 ? p : (p << 1) | (lo >> 63);
    const uint64_t next = p >> 63 ? lo >> 63 : (lo >> 62) & 1;   // round to nearest
    if (next && ~r.m)
        r.m++;
    return r;
}

// 2^-f in units of 2^-63, f = frac 2^-64.
template <class Table>
FSG_HD uint64_t exp2_neg_frac(uint64_t frac, const Table *tab)
{
    constexpr double L = EXP_LN2 / 1024.0;
    // 1024 c1 in units of 2^-64, 1024 c2 of 2^-44 (rounded down, as the product
    // taken from it is), 1024 c3 and c4 of 2^-56
    constexpr uint64_t C1 = 12786308645202655660ull;
    constexpr uint32_t C2 = (uint32_t)(512.0 * L * L * 17592186044416.0);
    constexpr uint32_t C3 = (uint32_t)(1024.0 / 6.0 * L * L * L * 72057594037927936.0 + 0.5);
    constexpr uint32_t C4 = (uint32_t)(1024.0 / 24.0 * L * L * L * L * 72057594037927936.0 + 0.5);
    const uint64_t T = tab[frac >> 54];
    const uint64_t x = frac << 10;
    const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x;
    const uint32_t t = C3 - (uint32_t)(((uint64_t)C4 * xh) >> 32);
    const uint32_t u = C2 - (uint32_t)(((uint64_t)t * xh) >> 44);
    const uint64_t A = C1 - (((uint64_t)xh * u) >> 12);
    const uint32_t ah = (uint32_t)(A >> 32), al = (uint32_t)A;
    const uint64_t q = (uint64_t)ah * xh + (((uint64_t)ah * xl) >> 32) +
                       (((uint64_t)al * xh) >> 32);
    const uint32_t qh = (uint32_t)(q >> 32), ql = (uint32_t)q;
    const uint32_t th = (uint32_t)(T >> 32), tl = (uint32_t)T;
    const uint64_t tq = (uint64_t)th * qh + (((uint64_t)th * ql) >> 32) +
                        (((uint64_t)tl * qh) >> 32);
    return T - (tq >> 10);
}

// n and f of a finite t with 53 <= sh = 62 - et - es
FSG_HD uint64_t exp_split(int64_t tb, int sh, const ExpScale &s, int &n)
{
    const uint64_t man = (((uint64_t)tb & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 11;
    const uint64_t P = fix_umulhi64(man, s.m);
    uint64_t frac;
    int ni = 0;
    if (sh < 64) {
        // P is rounded down: half a unit makes it even
        const uint64_t one = 1ull << (64 - sh);
        ni = (int)(P >> sh);
        frac = P * one + (one >> 1);
    } else {
        frac = sh > 127 ? 0 : P >> (sh - 64);
    }
    const int64_t up = ~((tb ^ s.neg) >> 63);    // all ones for a positive argument
    n = ni ^ (int)up;
    return frac ^ (uint64_t)up;
}

#ifdef __CUDACC__

// Arguments outside the normal results' range, infinities, NaN.
template <class Table>
__device__ __noinline__ double fexp_wide(double t, double s, const Table *tab)
{
    const double y = s * t;
    if (!(fabs(y) < 800.0)) {
        if (y != y)
            return y + y;
        return y > 0.0 ? __longlong_as_double(0x7FF0000000000000ll) : 0.0;
    }
    const ExpScale one = exp_scale(1.0);
    const long long yb = __double_as_longlong(y);
    const int e = (int)((yb >> 52) & 0x7FF) - 1023;
    int n;
    const uint64_t v = exp2_neg_frac(exp_split(yb, 62 - e - one.es, one, n), tab);
    const double r = __longlong_as_double((1021ll << 52) + (long long)((v + 512) >> 10));
    // 2^-n as two exact powers of two, one rounding
    const int n1 = n / 2, n2 = n - n1;
    return r * __longlong_as_double((long long)(1023 - n1) << 52) *
           __longlong_as_double((long long)(1023 - n2) << 52);
}

// exp(s t); sc = exp_scale(s)
template <class Table>
__device__ __forceinline__ double fexp(double t, double s, const ExpScale &sc, const Table *tab)
{
    const long long tb = __double_as_longlong(t);
    const int eb = (int)(tb >> 52) & 0x7FF;
    const int sh = 62 + 1023 - eb - sc.es;
    if (sh < 53 || eb == 0x7FF || !sc.finite) {
        // at least 2^10 log2 units: underflows when finite and negative past 2^11
        if (sh < 52 && eb != 0x7FF && sc.finite && (tb ^ sc.neg) < 0)
            return 0.0;
        return fexp_wide(t, s, tab);
    }
    int n;
    const uint64_t frac = exp_split(tb, sh, sc, n);
    if (n > 1020 || n < -1020)
        return fexp_wide(t, s, tab);
    const uint64_t v = exp2_neg_frac(frac, tab);
    return __longlong_as_double((long long)((v + 512) >> 10) + ((long long)(1021 - n) << 52));
}

#endif

}  // namespace fsg
