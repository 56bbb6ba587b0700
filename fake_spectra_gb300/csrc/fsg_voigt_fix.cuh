// Sum of Voigt profiles over the 7 line-of-sight nodes of a pair in 64-bit
// integer arithmetic (FP64 form of the optical depth).
//
// GB300 issues an FP64 instruction at 1/64 of the FP32 rate: one costs a warp
// scheduler the time of 16 others on its SM.  A profile value takes about 120
// FP64 operations (voigt_taylor_f64), or about 170 integer ones here, and the
// integer form is the more exact: the node distance x = |U_i - V| is held to
// 2^-53 absolute and every value below to 2^-55 or better relative, against
// 2^-53 relative for x and about 3e-15 for the value in FP64.
//
// For 1e-8 <= a <= 2^-8 (Ly-a above 40 K, CIV above 500 K) the profile splits
// exactly into H = G + a K',
//   G  = exp(a^2 - x^2) cos(2 a x)
//      = exp(a^2) 2^-(k1 x^2 + k2 x^4 + k3 x^6),   from log cos t =
//        -t^2/2 - t^4/12 - t^6/45 - ... (t = 2 a x; the next term is below
//        1e-15 where G is not negligible against a K'),
//   K' = K - a^2 K''/6 + a^4 K''''/120 - ...,  K = -(2/sqrt(pi)) F'(x),
//        F Dawson's integral (the Taylor series of w in Im z: A&S 7.1.20).
// 2^-y comes from a table of 2^(-k/64) and a degree-6 polynomial; K from one
// polynomial of degree 8 per interval of 1/32 below x = 8 and of 1/32 octave
// above (voigt_table.h, values from x = 2 on scaled by the octave's 4^e), and K'',
// K'''' from the same coefficients.  The node sums of G and K' are kept apart,
// each as a 64-bit integer with a binary exponent taken from the nearest node,
// so small values keep their relative precision.
#pragma once

#include <math.h>
#include <stdint.h>

#include "voigt_table.h"

#ifdef __CUDACC__
#define FSG_HD __host__ __device__ __forceinline__
#else
#define FSG_HD inline
#endif

namespace fsg {

constexpr int FIXV_BITS = 53;              // V and U are integers in units of 2^-53
constexpr double FIXV_MAX = 1000.0;        // |V| + |U| must stay below (10 integer bits)
constexpr double FIXV_A_MIN = 1e-8, FIXV_A_MAX = 0.00390625;
constexpr uint32_t FIXV_NEAR = 8u << 21;   // x < 8: fine rows; G is dropped beyond (1.6e-28)

// A row of the K table: C0..C5 in units of 2^-61 and C6..C8 in units of 2^-52
// of K(x) 4^e = sum_n C_n t^n, t = (x - row start) / (2 row width).
struct FixRow {
    int64_t c[6];
    int32_t s[3];
    int32_t pad;
};

// A number in [0, 1) as two 31-bit halves: v / 2 = hi 2^-32 + lo 2^-63.
struct Fix62 {
    int32_t hi, lo;
};

FSG_HD Fix62 fix62(uint64_t q64)           // v = q64 2^-64
{
    Fix62 f;
    f.hi = (int32_t)(uint32_t)(q64 >> 33);
    f.lo = (int32_t)((uint32_t)(q64 >> 2) & 0x7FFFFFFFu);
    return f;
}

// Per-pair constants.
struct FixPair {
    int64_t u1;          // node spacing, units of 2^-53
    uint64_t k1;         // log2(e) (1 + 2 a^2), units of 2^-63
    int32_t k2, k3;      // log2(e) (4/3) a^4 and (64/45) a^6, units of 2^-57 and 2^-67
    int32_t al, be;      // a^2 and a^4 factors of K'' and K'''' (30-bit mantissas) ...
    int32_t sal, sbe;    // ... and their right shifts in rows below x = 8
    Fix62 w[7];          // node weights / largest weight
};

FSG_HD int fix_mulhi32(int32_t a, int32_t b)
{
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return (int32_t)(((int64_t)a * b) >> 32);
#endif
}

FSG_HD uint64_t fix_umulhi64(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

FSG_HD int fix_clz32(uint32_t v)           // v != 0
{
#ifdef __CUDA_ARCH__
    return __clz((int)v);
#else
    return __builtin_clz(v);
#endif
}

// c + a v / 2 (a signed, rounded down within two units)
FSG_HD int64_t fix_fma(int64_t a, Fix62 v, int64_t c)
{
    const int32_t ah = (int32_t)(a >> 32);
    const uint32_t al = (uint32_t)a;
    const uint64_t cross = (uint64_t)al * (uint32_t)v.hi;
    const int64_t low = (int64_t)ah * v.lo;
    return (int64_t)ah * v.hi + (c + (int64_t)(cross >> 32) + (low >> 31));
}

// the same with the upper half of v only
FSG_HD int64_t fix_fma_hi(int64_t a, int32_t vhi, int64_t c)
{
    const int32_t ah = (int32_t)(a >> 32);
    const uint32_t al = (uint32_t)a;
    return (int64_t)ah * vhi + (c + (int64_t)(((uint64_t)al * (uint32_t)vhi) >> 32));
}

// 2^(-k/64), k = 0 .. 63, as halves of a number in (1/2, 1]: hi 2^-31 + lo 2^-62
// of 2^(-k/64), i.e. fix62 of it (1 itself is stored one unit below).
// 2^-(rho/64) = sum_m P_m (rho/2)^m, P_m = (-ln2/32)^m / m! in units of 2^-62.
constexpr double FIX_LN2_32 = 0.693147180559945309417232121458 / 32.0;

// Node sums at V (units of 2^-53): sum_i w_i G_i = sg 2^(-60 - eg) exp(a^2),
// sum_i w_i K'_i = sk 2^(-60 - ek).  Rows: load(r) gives row r of the K table;
// pow2: the 2^(-k/64) table.
template <class Rows>
FSG_HD void fix_node_sums(const FixPair &p, int64_t V, const Rows &rows, const Fix62 *pow2,
                          int64_t &sg, int &eg, int64_t &sk, int &ek)
{
    // nearest node: the common exponents
    uint32_t xmin = 0xFFFFFFFFu;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < 7; i++) {
        const int64_t d = (int64_t)(i - 3) * p.u1 - V;
        const uint32_t xh = (uint32_t)((uint64_t)(d < 0 ? -d : d) >> 32);
        xmin = xh < xmin ? xh : xmin;
    }
    // x^2 log2(e) of the nearest node, rounded down (x < 8: xmin < 2^24)
    eg = xmin < FIXV_NEAR
             ? (int)(((((uint64_t)xmin * xmin) >> 32) * 1477u) >> 20) : 0;
    ek = xmin < (1u << 22) ? 0 : 2 * (10 - fix_clz32(xmin));
    sg = 0;
    sk = 0;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int i = 0; i < 7; i++) {
        const int64_t d = (int64_t)(i - 3) * p.u1 - V;
        const uint64_t x = (uint64_t)(d < 0 ? -d : d);
        const uint32_t xh = (uint32_t)(x >> 32);
        const Fix62 w = p.w[i];
        if (xh < FIXV_NEAR) {
            const uint64_t x2 = fix_umulhi64(x << 8, x << 8);      // 2^-58
            const uint32_t x2h = (uint32_t)(x2 >> 32);             // 2^-26
            const uint32_t x4 = (uint32_t)(((uint64_t)x2h * x2h) >> 32);   // 2^-20
            uint64_t y = fix_umulhi64(x2, p.k1);                   // 2^-57
            y += ((uint64_t)x4 * (uint32_t)p.k2) >> 20;
            if (p.k3)
                y += ((uint64_t)(uint32_t)(((uint64_t)x4 * x2h) >> 32) * (uint32_t)p.k3) >> 24;
            const int n = (int)(y >> 57);
            const int k = (int)(y >> 51) & 63;
            const Fix62 r = fix62(y << 13);
            constexpr double U = 4611686018427387904.0;            // 2^62
            constexpr double L = FIX_LN2_32;
            constexpr int32_t P6 = (int32_t)(U * L * L * L * L * L * L / 720.0 + 0.5);
            constexpr int32_t P5 = -(int32_t)(U * L * L * L * L * L / 120.0 + 0.5);
            constexpr int64_t P4 = (int64_t)(U * L * L * L * L / 24.0 + 0.5);
            constexpr int64_t P3 = -(int64_t)(U * L * L * L / 6.0 + 0.5);
            constexpr int64_t P2 = FSG_FIX_P2, P1 = FSG_FIX_P1;    // voigt_table.h
            constexpr int64_t P0 = (int64_t)1 << 62;
            const int32_t s5 = P5 + fix_mulhi32(P6, r.hi);
            const int64_t a4 = P4 + fix_mulhi32(s5, r.hi);
            const int64_t a3 = fix_fma_hi(a4, r.hi, P3);
            const int64_t a2 = fix_fma(a3, r, P2);
            const int64_t a1 = fix_fma(a2, r, P1);
            const int64_t a0 = fix_fma(a1, r, P0);
            const int64_t g = fix_fma(fix_fma(a0, pow2[k], 0), w, 0);   // 2^-60
            const int sh = n - eg;
            sg += g >> (sh < 63 ? sh : 63);
        }
        // K'
        const bool near = xh < FIXV_NEAR;
        const int e = 31 - fix_clz32(xh | 1u);
        const int s = near ? 16 : e - 5;
        const int ri = (int)(xh >> s) + (near ? 0 : 32 * e - 544);
        const FixRow row = rows.load(ri < FSG_FIX_ROWS ? ri : FSG_FIX_ROWS - 1);
        const Fix62 t = fix62(x << (32 - s));
        const int64_t c5 = row.c[5], c4 = row.c[4], c3 = row.c[3], c2 = row.c[2];
        const int32_t s6 =
            row.s[0] + fix_mulhi32(row.s[1] + fix_mulhi32(row.s[2], t.hi), t.hi);
        const int64_t a5 = c5 + (((int64_t)s6 * t.hi) >> 23);
        const int64_t a4 = fix_fma_hi(a5, t.hi, c4);
        const int64_t a3 = fix_fma(a4, t, c3);
        const int64_t a2 = fix_fma(a3, t, c2);
        const int64_t a1 = fix_fma(a2, t, row.c[1]);
        int64_t a0 = fix_fma(a1, t, row.c[0]);
        // K''/2 in row units (2h)^2; K''''/24 in row units (2h)^4, >> 24
        const int32_t h4 = (int32_t)(c4 >> 19), h5 = (int32_t)(c5 >> 19);
        const int32_t h6 = row.s[0] >> 10, h7 = row.s[1] >> 10;
        int32_t d2 = 15 * h6 + fix_mulhi32(21 * h7, t.hi);
        d2 = 10 * h5 + fix_mulhi32(d2, t.hi);
        d2 = 6 * h4 + fix_mulhi32(d2, t.hi);
        const int64_t D2 = fix_fma_hi(3 * c3 + (((int64_t)d2 * t.hi) >> 13), t.hi, c2);
        int32_t d4 = 15 * h6 + fix_mulhi32(35 * h7, t.hi);
        d4 = 5 * h5 + fix_mulhi32(d4, t.hi);
        d4 = (h4 + fix_mulhi32(d4, t.hi)) >> 5;
        // K is scaled by 2^o; (2h)^2 is 2^-8 below x = 8 and grows by 2^g above
        const int o = xh < (1u << 22) ? 0 : 2 * e - 42, g = near ? 0 : o;
        const int sa = p.sal + g, sb = p.sbe + 2 * g;
        a0 -= fix_fma_hi(D2, p.al, 0) >> (sa < 63 ? sa : 63);
        a0 += ((int64_t)d4 * p.be) >> (sb < 63 ? sb : 63);
        const int64_t kw = fix_fma(a0, w, 0);     // 2^-60
        const int sh = o - ek;
        sk += kw >> (sh < 63 ? sh : 63);
    }
}

// a^2 and a^4 factors: v = m 2^-shift with m of 30 bits.
inline
#ifdef __CUDACC__
    __host__ __device__
#endif
    void fix_mantissa(double v, int32_t &m, int32_t &shift)
{
    int e;
    const double f = frexp(v, &e);          // v = f 2^e, f in [1/2, 1)
    m = (int32_t)(f * 1073741824.0 + 0.5);  // 2^30
    shift = 30 - e;
    if (!(v > 0.0)) {
        m = 0;
        shift = 0;
    }
}

// Pair constants from the damping a (FIXV_A_MIN <= a <= FIXV_A_MAX).
inline
#ifdef __CUDACC__
    __host__ __device__
#endif
    void fix_pair_damping(double a, FixPair &p)
{
    const double a2 = a * a;
    // log2(e) 2^63 and its product with 2 a^2
    p.k1 = FSG_FIX_LOG2E + (uint64_t)(a2 * 2.0 * 13306513097844322492.0);
    p.k2 = (int32_t)(1.4426950408889634 * (4.0 / 3.0) * a2 * a2 * 144115188075855872.0 + 0.5);
    p.k3 = (int32_t)(1.4426950408889634 * (64.0 / 45.0) * a2 * a2 * a2 *
                     147573952589676412928.0 + 0.5);
    // -a^2 K''/6: K''/2 = D2 / (2h)^2, (2h)^-2 = 256 below x = 8
    fix_mantissa(a2 / 3.0 * 256.0, p.al, p.sal);
    p.sal -= 32;         // the product drops its low 32 bits first
    // a^4 K''''/120: K''''/24 = d4 2^24 / (2h)^4
    fix_mantissa(a2 * a2 / 5.0 * 65536.0 * 16777216.0, p.be, p.sbe);
}

// ------------------------------------------------------------- numbers m 2^e
FSG_HD int fix_clz64(uint64_t v)   // v != 0
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}

FSG_HD uint64_t fix_bits(double d)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t u;
    __builtin_memcpy(&u, &d, 8);
    return u;
#endif
}

FSG_HD double fix_from_bits(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    __builtin_memcpy(&d, &u, 8);
    return d;
#endif
}

// A positive normal double as m 2^e, m in [2^63, 2^64).
struct FixNum {
    uint64_t m;
    int e;
};
FSG_HD FixNum fix_num(double d)
{
    const uint64_t u = fix_bits(d);
    FixNum r;
    r.m = (u << 11) | (1ull << 63);
    r.e = (int)((u >> 52) & 0x7FF) - 1086;
    return r;
}

// m 2^e as a double (the result must be normal; m = 0 gives 0), sign bit `neg`.
FSG_HD double fix_double(uint64_t m, int e, uint64_t neg)
{
    if (m == 0)
        return 0.0;
    const int lz = fix_clz64(m);
    const uint64_t n = m << lz;
    const uint64_t r = (n >> 11) + ((n >> 10) & 1ull);   // 53 bits, bit 52 set (or a carry)
    return fix_from_bits((neg << 63) | ((((uint64_t)(e + 1085 - lz)) << 52) + r));
}

// A velocity in units of b from twice its value: |V| = p 2^(-53 - s), p in
// [2^62, 2^64); ib, eb: 1/b = ib 2^eb.
struct FixV {
    uint64_t p;
    int s;
};
FSG_HD FixV fix_velocity(double v2, uint64_t ib, int eb)
{
    const uint64_t u = fix_bits(v2);
    const int E = (int)((u >> 52) & 0x7FF);
    FixV r;
    r.p = fix_umulhi64((u << 11) | (1ull << 63), ib);
    r.s = 970 - E - eb;       // v2 = 0: E = 0, a shift beyond the word
    return r;
}
// |V| in units of 2^-53 (saturating)
FSG_HD uint64_t fix_v53(FixV v)
{
    return v.s < 0 ? 0x7FFFFFFFFFFFFFFFull : (v.s > 63 ? 0ull : v.p >> v.s);
}

// 1 / (p 2^-64) for p in [2^63, 2^64), units of 2^-63 (error below 2^-61): the
// float reciprocal and one third-order Newton step.
FSG_HD uint64_t fix_recip(uint64_t p)
{
    const float pf = (float)(uint32_t)(p >> 32);
#ifdef __CUDA_ARCH__
    const uint32_t r0 = __float2uint_rz(fminf(9223372036854775808.0f * __frcp_rn(pf),
                                              4294967040.0f));
#else
    const float rf = 9223372036854775808.0f / pf;
    const uint32_t r0 = (uint32_t)(rf < 4294967040.0f ? rf : 4294967040.0f);
#endif
    // e = 1 - r0 p, units of 2^-63
    const uint64_t t = (p >> 32) * r0 + (((p & 0xFFFFFFFFull) * r0) >> 32);
    const int64_t e1 = (int64_t)((1ull << 63) - t);
    const int64_t e12 = e1 >> 12;
    const int64_t d = e1 + ((e12 * e12) >> 39);
    const int64_t dh = d >> 32;
    const uint64_t dl = (uint64_t)d & 0xFFFFFFFFull;
    return ((uint64_t)r0 << 32) + (uint64_t)(dh * (int64_t)r0 * 2) + ((dl * r0) >> 31);
}

// Far wing: A_1 y + A_2 y^2 + ..., y = (vmp / V)^2 < 1, as cA y times the sum of
// (A_r / A_1) y^(r-1).
constexpr int FIX_FAR_R = 16;
struct FixFar {
    uint64_t vs, cA;         // vmp^2 = vs 2^ev; scale A_1 = cA 2^eA
    int32_t ev, eA;
    int64_t A[FIX_FAR_R - 1];   // A_(r+1) / A_1 2^r, units of 2^-61
};

// y = ym 2^ye of a velocity beyond vmp, ym in [2^63, 2^64)
FSG_HD uint64_t fix_far_y(const FixFar &f, FixV v, int &ye)
{
    const int lz = (int)(~v.p >> 63);
    const uint64_t r = fix_recip(v.p << lz);
    const uint64_t m = fix_umulhi64(fix_umulhi64(r, r), f.vs);
    const int lm = fix_clz64(m);
    ye = f.ev - 20 + 2 * (v.s + lz) - lm;    // -126 - 2 q + ev, q = -53 - s - lz
    return m << lm;
}

// The wing's value m 2^e from n >= 2 terms (from the eighth on the upper half of y
// is enough).
FSG_HD uint64_t fix_far_sum(const FixFar &f, int n, uint64_t ym, int ye, int &e)
{
    const int sh = -64 - ye;                 // y 2^64 = ym >> sh
    const Fix62 y = fix62(sh > 63 ? 0ull : ym >> sh);
    int64_t acc = f.A[n - 2];
    int r = n - 3;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (; r >= 6; r--)
        acc = fix_fma_hi(acc, y.hi, f.A[r]);
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (; r >= -1; r--)
        acc = fix_fma(acc, y, r >= 0 ? f.A[r] : (int64_t)1 << 61);
    const uint64_t m1 = fix_umulhi64((uint64_t)acc << 2, ym);
    e = 65 + f.eA + ye;
    return fix_umulhi64(m1, f.cA);
}

// sg 2^(-60 - eg) cg + sk 2^(-60 - ek) ck as m 2^e (a positive sum).
FSG_HD uint64_t fix_combine(int64_t sg, int eg, FixNum cg, int64_t sk, int ek, FixNum ck, int &e)
{
    uint64_t gm = 0, km = 0;
    int xg = -100000, xk = -100000;
    if (sg > 0) {
        const int lz = fix_clz64((uint64_t)sg);
        gm = fix_umulhi64((uint64_t)sg << lz, cg.m) >> 2;   // room for the sum
        xg = 6 - lz + cg.e - eg;
    }
    if (sk != 0) {
        const uint64_t a = (uint64_t)(sk < 0 ? -sk : sk);
        const int lz = fix_clz64(a);
        km = fix_umulhi64(a << lz, ck.m) >> 2;
        xk = 6 - lz + ck.e - ek;
    }
    e = xg > xk ? xg : xk;
    const int dg = e - xg, dk = e - xk;
    gm = dg > 63 ? 0ull : gm >> dg;
    km = dk > 63 ? 0ull : km >> dk;
    const int64_t t = (int64_t)gm + (sk < 0 ? -(int64_t)km : (int64_t)km);
    return t > 0 ? (uint64_t)t : 0ull;
}

}  // namespace fsg
