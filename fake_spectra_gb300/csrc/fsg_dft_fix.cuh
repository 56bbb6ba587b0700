// Discrete Fourier transforms in 64-bit fixed point for the 1-D flux power.
//
// GB300 issues an FP64 instruction at 1/64 of the FP32 rate: an FP64 addition
// takes the time of 64 integer instructions on its SM, a 64-bit integer addition
// that of two, a product of a 64-bit number and a table value that of about 15.
// The transforms here hold each component as an integer in units of a power of
// two fixed per row and pass; additions are exact and each product is rounded
// once.
//
// Scaling.  By Cauchy's inequality no value of a partial transform that combines
// m inputs exceeds sqrt(m) |z|_2.  The input is scaled so that |z|_2 <= 2^60.8 and
// each pass divides by a power of two so that what m inputs have been combined
// into is divided by sqrt(m) at least: every stored modulus stays below 2^60.8 and,
// inside a pass of radix R <= 16, below sqrt(R) 2^60.8 <= 2^62.8.  A typical value is
// 2^60 / sqrt(m), so for transforms of 1e4 points values keep 53 bits and the
// rounding of all passes together stays below that of FP64 arithmetic.
//
// In place and without reordering: decimation in frequency takes natural order
// to digit-reversed order (dif_pass: butterfly, then twiddles), decimation in
// time back (dit_pass: twiddles, then butterfly).
#pragma once

#include "fsg_voigt_fix.cuh"

namespace fsg {

struct FixC {
    int64_t x, y;
};

// A number in [-1, 1] in units of 2^-62, as the words of a 64-bit integer with the
// lower word signed: v = hi 2^-30 + lo 2^-62.
struct FixV62 {
    int32_t hi, lo;
};
struct FixW {
    FixV62 c, s;      // a complex factor, modulus 1 at most
};

// |v| <= 1
FSG_HD FixV62 fix_v62(double v)
{
    const int64_t u = (int64_t)(v * 4611686018427387904.0);
    const int32_t lo = (int32_t)(uint32_t)u;
    // both words can be negated
    return {(int32_t)((u - lo) >> 32), lo == INT32_MIN ? -INT32_MAX : lo};
}

// a as ah 2^32 + al, both signed
struct FixSplit {
    int32_t hi, lo;
};
FSG_HD FixSplit fix_split(int64_t a)
{
    const int32_t lo = (int32_t)(uint32_t)a;
    return {(int32_t)((a - lo) >> 32), lo};
}

// a w / 2^e, e = 1 or 2, rounded, ties up or (odd = 1) down: a factor of 1 meets
// ties, and values of one column rounded the same way would add up.  A modulus of a
// up to 2^62.8 keeps the sums below 2^63: the products of a's low words (at most 2^31
// each) with w's high words (modulus 2^30) are below 2^61.5 together, those of a's high
// words (modulus 2^30.8) with w's low words below 2^62.3, those of the high words
// below 2^60.8 (2^61.8 shifted).
FSG_HD FixC fixc_mul(FixC a, FixW w, int e, int odd)
{
    const FixSplit x = fix_split(a.x), y = fix_split(a.y);
    const int32_t nh = -w.s.hi, nl = -w.s.lo;
    const int64_t half = (int64_t)((uint32_t)1 << (29 + e)) - odd;
    int64_t r = (int64_t)x.lo * w.c.hi + half;
    r += (int64_t)y.lo * nh;
    r += (int64_t)x.hi * w.c.lo;
    r += (int64_t)y.hi * nl;
    int64_t i = (int64_t)x.lo * w.s.hi + half;
    i += (int64_t)y.lo * w.c.hi;
    i += (int64_t)x.hi * w.s.lo;
    i += (int64_t)y.hi * w.c.lo;
    const int64_t p = (int64_t)x.hi * w.c.hi + (int64_t)y.hi * nh;
    const int64_t q = (int64_t)x.hi * w.s.hi + (int64_t)y.hi * w.c.hi;
    return {(int64_t)((uint64_t)p << (2 - e)) + (r >> (30 + e)),
            (int64_t)((uint64_t)q << (2 - e)) + (i >> (30 + e))};
}

// v / 2^e, rounded, ties up or down (e >= 1)
FSG_HD int64_t fix_shift(int64_t v, int e, int odd)
{
    return (v + (((int64_t)1 << (e - 1)) - odd)) >> e;
}

FSG_HD FixC operator+(FixC a, FixC b) { return {a.x + b.x, a.y + b.y}; }
FSG_HD FixC operator-(FixC a, FixC b) { return {a.x - b.x, a.y - b.y}; }
// -i a
FSG_HD FixC fixc_mi(FixC a) { return {a.y, -a.x}; }

// a V / 2^63, V a constant
template <int64_t V>
FSG_HD int64_t fix_const_mul(int64_t a)
{
    constexpr int32_t lo = (int32_t)(uint32_t)V;
    constexpr int32_t hi = (int32_t)((V - lo) >> 32);
    // twice the half product, the bit below kept: mid is taken one bit lower
    const FixSplit s = fix_split(a);
    int64_t mid = (int64_t)s.lo * hi + 1073741824ll;
    mid += (int64_t)s.hi * lo;
    return (((int64_t)s.hi * hi) << 1) + (mid >> 31);
}

namespace dftc {
constexpr int64_t H = 6521908912666391106ll;      // cos(pi/4) 2^63
constexpr int64_t C1 = 8521284645587064995ll;     // cos(pi/8)
constexpr int64_t S1 = 3529631669043774883ll;     // sin(pi/8)
constexpr int64_t S3 = 7987674492471257551ll;     // sin(2 pi/3)
constexpr int64_t C51 = 2850178704830799621ll;    // cos(2 pi/5)
constexpr int64_t C52 = -7461864723258187525ll;   // cos(4 pi/5)
constexpr int64_t S51 = 8771948077865237882ll;    // sin(2 pi/5)
constexpr int64_t S52 = 5421362059670026167ll;    // sin(4 pi/5)
constexpr int64_t C71 = 5750678403727967667ll;    // cos(2 pi/7)
constexpr int64_t C72 = -2052393359867478633ll;   // cos(4 pi/7)
constexpr int64_t C73 = -8309971062287876938ll;   // cos(6 pi/7)
constexpr int64_t S71 = 7211122632928341039ll;    // sin(2 pi/7)
constexpr int64_t S72 = 8992122843167040398ll;    // sin(4 pi/7)
constexpr int64_t S73 = 4001871146622878209ll;    // sin(6 pi/7)
}  // namespace dftc

FSG_HD void fixc_dft4(FixC &x0, FixC &x1, FixC &x2, FixC &x3)
{
    const FixC t0 = x0 + x2, t1 = x0 - x2, t2 = x1 + x3, t3 = fixc_mi(x1 - x3);
    x0 = t0 + t2;
    x2 = t0 - t2;
    x1 = t1 + t3;
    x3 = t1 - t3;
}

// exp(-i pi E / 8) a
template <int E>
FSG_HD FixC fixc_rot16(FixC a)
{
    using namespace dftc;
    if constexpr (E == 2)
        return {fix_const_mul<H>(a.x + a.y), fix_const_mul<H>(a.y - a.x)};
    else if constexpr (E == 4)
        return fixc_mi(a);
    else if constexpr (E == 6)
        return {fix_const_mul<H>(a.y - a.x), fix_const_mul<-H>(a.x + a.y)};
    else if constexpr (E == 1)
        return {fix_const_mul<C1>(a.x) + fix_const_mul<S1>(a.y),
                fix_const_mul<C1>(a.y) - fix_const_mul<S1>(a.x)};
    else if constexpr (E == 3)
        return {fix_const_mul<S1>(a.x) + fix_const_mul<C1>(a.y),
                fix_const_mul<S1>(a.y) - fix_const_mul<C1>(a.x)};
    else {
        static_assert(E == 9, "rotation not used by the 8- and 16-point transforms");
        return {fix_const_mul<-C1>(a.x) - fix_const_mul<S1>(a.y),
                fix_const_mul<S1>(a.x) - fix_const_mul<C1>(a.y)};
    }
}

// Forward transform of R points in registers, natural order.
template <int R>
FSG_HD void fixc_dft(FixC (&v)[R])
{
    using namespace dftc;
    if constexpr (R == 2) {
        const FixC t = v[0];
        v[0] = t + v[1];
        v[1] = t - v[1];
    } else if constexpr (R == 4) {
        fixc_dft4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        // n = 2 n1 + n2, k = k1 + 4 k2
        fixc_dft4(v[0], v[2], v[4], v[6]);
        fixc_dft4(v[1], v[3], v[5], v[7]);
        const FixC a0 = v[0], a1 = v[2], a2 = v[4], a3 = v[6];
        const FixC b0 = v[1], b1 = fixc_rot16<2>(v[3]), b2 = fixc_rot16<4>(v[5]),
                   b3 = fixc_rot16<6>(v[7]);
        v[0] = a0 + b0;
        v[4] = a0 - b0;
        v[1] = a1 + b1;
        v[5] = a1 - b1;
        v[2] = a2 + b2;
        v[6] = a2 - b2;
        v[3] = a3 + b3;
        v[7] = a3 - b3;
    } else if constexpr (R == 16) {
        // n = 4 n1 + n2, k = k1 + 4 k2: after the first transforms index (n2, k1)
        // is at v[4 k1 + n2]
        fixc_dft4(v[0], v[4], v[8], v[12]);
        fixc_dft4(v[1], v[5], v[9], v[13]);
        fixc_dft4(v[2], v[6], v[10], v[14]);
        fixc_dft4(v[3], v[7], v[11], v[15]);
        v[5] = fixc_rot16<1>(v[5]);
        v[9] = fixc_rot16<2>(v[9]);
        v[13] = fixc_rot16<3>(v[13]);
        v[6] = fixc_rot16<2>(v[6]);
        v[10] = fixc_rot16<4>(v[10]);
        v[14] = fixc_rot16<6>(v[14]);
        v[7] = fixc_rot16<3>(v[7]);
        v[11] = fixc_rot16<6>(v[11]);
        v[15] = fixc_rot16<9>(v[15]);
        fixc_dft4(v[0], v[1], v[2], v[3]);
        fixc_dft4(v[4], v[5], v[6], v[7]);
        fixc_dft4(v[8], v[9], v[10], v[11]);
        fixc_dft4(v[12], v[13], v[14], v[15]);
        // X[k1 + 4 k2] is at v[4 k1 + k2]: transpose
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int k1 = 0; k1 < 4; k1++)
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int k2 = k1 + 1; k2 < 4; k2++) {
                const FixC t = v[4 * k1 + k2];
                v[4 * k1 + k2] = v[k1 + 4 * k2];
                v[k1 + 4 * k2] = t;
            }
    } else if constexpr (R == 3) {
        const FixC a = v[1] + v[2], b = v[1] - v[2];
        const FixC re = {v[0].x - fix_shift(a.x, 1, 0), v[0].y - fix_shift(a.y, 1, 1)};
        const FixC im = {fix_const_mul<S3>(b.y), fix_const_mul<-S3>(b.x)};   // -i sin b
        v[0] = v[0] + a;
        v[1] = re + im;
        v[2] = re - im;
    } else if constexpr (R == 5) {
        const FixC a1 = v[1] + v[4], a2 = v[2] + v[3], b1 = v[1] - v[4], b2 = v[2] - v[3];
        const FixC r1 = {v[0].x + fix_const_mul<C51>(a1.x) + fix_const_mul<C52>(a2.x),
                         v[0].y + fix_const_mul<C51>(a1.y) + fix_const_mul<C52>(a2.y)};
        const FixC r2 = {v[0].x + fix_const_mul<C52>(a1.x) + fix_const_mul<C51>(a2.x),
                         v[0].y + fix_const_mul<C52>(a1.y) + fix_const_mul<C51>(a2.y)};
        const FixC s1 = {fix_const_mul<S51>(b1.y) + fix_const_mul<S52>(b2.y),
                         fix_const_mul<-S51>(b1.x) - fix_const_mul<S52>(b2.x)};
        const FixC s2 = {fix_const_mul<S52>(b1.y) - fix_const_mul<S51>(b2.y),
                         fix_const_mul<-S52>(b1.x) + fix_const_mul<S51>(b2.x)};
        v[0] = v[0] + a1 + a2;
        v[1] = r1 + s1;
        v[4] = r1 - s1;
        v[2] = r2 + s2;
        v[3] = r2 - s2;
    } else {
        static_assert(R == 7, "radix");
        const FixC a1 = v[1] + v[6], a2 = v[2] + v[5], a3 = v[3] + v[4];
        const FixC b1 = v[1] - v[6], b2 = v[2] - v[5], b3 = v[3] - v[4];
        const FixC z = v[0];
        v[0] = z + a1 + a2 + a3;
        const FixC r1 = {z.x + fix_const_mul<C71>(a1.x) + fix_const_mul<C72>(a2.x) +
                             fix_const_mul<C73>(a3.x),
                         z.y + fix_const_mul<C71>(a1.y) + fix_const_mul<C72>(a2.y) +
                             fix_const_mul<C73>(a3.y)};
        const FixC s1 = {fix_const_mul<S71>(b1.y) + fix_const_mul<S72>(b2.y) +
                             fix_const_mul<S73>(b3.y),
                         fix_const_mul<-S71>(b1.x) - fix_const_mul<S72>(b2.x) -
                             fix_const_mul<S73>(b3.x)};
        v[1] = r1 + s1;
        v[6] = r1 - s1;
        const FixC r2 = {z.x + fix_const_mul<C72>(a1.x) + fix_const_mul<C73>(a2.x) +
                             fix_const_mul<C71>(a3.x),
                         z.y + fix_const_mul<C72>(a1.y) + fix_const_mul<C73>(a2.y) +
                             fix_const_mul<C71>(a3.y)};
        const FixC s2 = {fix_const_mul<S72>(b1.y) - fix_const_mul<S73>(b2.y) -
                             fix_const_mul<S71>(b3.y),
                         fix_const_mul<-S72>(b1.x) + fix_const_mul<S73>(b2.x) +
                             fix_const_mul<S71>(b3.x)};
        v[2] = r2 + s2;
        v[5] = r2 - s2;
        const FixC r3 = {z.x + fix_const_mul<C73>(a1.x) + fix_const_mul<C71>(a2.x) +
                             fix_const_mul<C72>(a3.x),
                         z.y + fix_const_mul<C73>(a1.y) + fix_const_mul<C71>(a2.y) +
                             fix_const_mul<C72>(a3.y)};
        const FixC s3 = {fix_const_mul<S73>(b1.y) - fix_const_mul<S71>(b2.y) +
                             fix_const_mul<S72>(b3.y),
                         fix_const_mul<-S73>(b1.x) + fix_const_mul<S71>(b2.x) -
                             fix_const_mul<S72>(b3.x)};
        v[3] = r3 + s3;
        v[4] = r3 - s3;
    }
}

// Butterfly f of a decimation-in-frequency pass over blocks of m R points: the
// transform of the points m apart, then element q times exp(-2 pi i j q / (m R))
// (tw[(q - 1) m + j]) / 2^e.  m = 1: no twiddles, no division.
template <int R>
FSG_HD void dif_butterfly(FixC *x, const FixW *tw, unsigned f, unsigned m, int e)
{
    const unsigned b = f / m, j = f - b * m;
    FixC *p = x + (size_t)b * m * R + j;
    FixC v[R];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int r = 0; r < R; r++)
        v[r] = p[r * m];
    fixc_dft<R>(v);
    if (m > 1) {
        p[0] = {fix_shift(v[0].x, e, b & 1), fix_shift(v[0].y, e, b & 1)};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int q = 1; q < R; q++)
            p[q * m] = fixc_mul(v[q], tw[(q - 1) * m + j], e, b & 1);
    } else {
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
        for (int q = 0; q < R; q++)
            p[q] = v[q];
    }
}

// Butterfly f of a decimation-in-time pass (m > 1): the twiddles and divisions, then
// the transform.
template <int R>
FSG_HD void dit_butterfly(FixC *x, const FixW *tw, unsigned f, unsigned m, int e)
{
    const unsigned b = f / m, j = f - b * m;
    FixC *p = x + (size_t)b * m * R + j;
    FixC v[R];
    v[0] = {fix_shift(p[0].x, e, b & 1), fix_shift(p[0].y, e, b & 1)};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int r = 1; r < R; r++)
        v[r] = fixc_mul(p[r * m], tw[(r - 1) * m + j], e, b & 1);
    fixc_dft<R>(v);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int q = 0; q < R; q++)
        p[q * m] = v[q];
}

// The last pass of a transform to digit-reversed order, the product with the
// filter w / 2^e (the result conjugated) and the first pass back, on the R adjacent
// points of butterfly f.
template <int R>
FSG_HD void filter_butterfly(FixC *x, const FixW *w, unsigned f, unsigned L, int e)
{
    FixC *p = x + (size_t)f * R;
    w += f * R % L;          // rows one after another
    FixC v[R];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int r = 0; r < R; r++)
        v[r] = p[r];
    fixc_dft<R>(v);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int r = 0; r < R; r++) {
        v[r] = fixc_mul(v[r], w[r], e, f & 1);
        v[r].y = -v[r].y;
    }
    fixc_dft<R>(v);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int r = 0; r < R; r++)
        p[r] = v[r];
}

// d in units of 2^-sh, rounded (|d| < 2^(63 - sh); d = 0 below 2^-1022)
FSG_HD int64_t fix_from_double(double d, int sh)
{
#ifdef __CUDA_ARCH__
    const int64_t b = __double_as_longlong(d);
#else
    int64_t b;
    __builtin_memcpy(&b, &d, 8);
#endif
    const int e = (int)(b >> 52) & 0x7FF;
    const int64_t man = (b & 0xFFFFFFFFFFFFFll) | (1ll << 52);
    const int s = e - 1075 + sh;
    int64_t v = s >= 0 ? man << (s & 63) : s < -62 ? 0 : (man + (1ll << (-s - 1))) >> -s;
    v = e ? v : 0;
    return b < 0 ? -v : v;
}

// v 2^e as a double, rounded (2^-1022 <= |v 2^e| < 2^1024 or v = 0)
FSG_HD double fix_to_double(int64_t v, int e)
{
    const uint64_t a = (uint64_t)(v < 0 ? -v : v);
    if (a == 0)
        return 0.0;
#ifdef __CUDA_ARCH__
    const int z = __clzll((long long)a);
#else
    const int z = __builtin_clzll(a);
#endif
    // upper bit at 62, rounded at bit 10
    const uint64_t m = (a << z) >> 1;
    const int64_t b = (int64_t)((m + 512) >> 10) + ((int64_t)(1022 + 63 - z + e) << 52) +
                      (int64_t)((uint64_t)v & (1ull << 63));
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double d;
    __builtin_memcpy(&d, &b, 8);
    return d;
#endif
}

}  // namespace fsg
