// Line-of-sight kernel integral of one pixel in 64-bit integer arithmetic
// (FP64 form of the column density).
//
// The reference's rule is a trapezoid over 9 nodes of the SPH kernel at
// q = sqrt(dr2 + z^2) / h (absorption.cpp:53-97): a square root, a division and
// a polynomial per node, about 37 FP64 operations on hardware that issues one
// FP64 instruction in the time of 64 others.  Here z / h is an integer in units
// of 2^-62 and q, s = q^2 and t = 1 - q are integers in units of 2^-64; the
// square root starts from the float reciprocal root and takes two Newton steps
// (error below 2^-62), about 80 integer operations a node.  t is shifted up by
// the pixel's common exponent before its powers are taken, so kernel tails
// keep their relative precision (about 2^-53).  For pixels with
// 1 - s >= 2^-8 at both ends; there the double arithmetic of the reference is
// itself good to about 2^-53 / (1 - q), 3e-13 at worst, and the values agree
// to that.
#pragma once

#include "fsg_voigt_fix.cuh"

namespace fsg {

// q = sqrt(s), units of 2^-64, s >= 2^-16: error below 2^-61.
FSG_HD uint64_t fix_sqrt64_upper(uint64_t s)
{
    const float sf = (float)((uint32_t)(s >> 32) | 1u);
#ifdef __CUDA_ARCH__
    const float rs = rsqrtf(sf);
    const uint32_t q0 = __float2uint_rz(fminf(sf * rs * 65536.0f, 4294967040.0f));
#else
    const float rs = 1.0f / sqrtf(sf);
    const float qf = sf * rs * 65536.0f;
    const uint32_t q0 = (uint32_t)(qf < 4294967040.0f ? qf : 4294967040.0f);
#endif
    const int64_t e1 = (int64_t)(s - (uint64_t)q0 * q0);
    const int32_t d1 = (int32_t)((float)(int32_t)(e1 >> 16) * (rs * 524288.0f));
    const uint64_t q1 = ((uint64_t)q0 << 32) + (uint64_t)((int64_t)d1 << 12);
    const int32_t e2 = (int32_t)(s - fix_umulhi64(q1, q1));
    return q1 + (uint64_t)(int64_t)(int32_t)((float)e2 * (rs * 32768.0f));
}

// q = sqrt(s): small s (nodes near the particle) is shifted into the range
// above, where the float root has enough bits to start from.
FSG_HD uint64_t fix_sqrt64(uint64_t s)
{
    if (s >= (1ull << 48))
        return fix_sqrt64_upper(s);
    if (s == 0)
        return 0;
    const int sh = fix_clz64(s) & ~1;
    return fix_sqrt64_upper(s << sh) >> (sh / 2);
}

// 2^62 / h from inv = 1 / h, a few units lower where the half-chord zrange is h to the
// last bits (the particle on its sightline): |z| <= zrange then stays below 2^62 in
// units of h / 2^62, and the squares of 4 |z| in fix_spline_sum within 64 bits.
FSG_HD double fix_spline_scale(double inv, double h, double zrange)
{
    const uint64_t s = fix_bits(4611686018427387904.0 * inv);
    return fix_from_bits(fix_bits(zrange) + 4 >= fix_bits(h) ? s - 8 : s);
}

// Trapezoid sum over the 9 nodes from z = za to zb (units of 2^-62 of h) of the
// cubic (W / (8/pi)) or quintic (W / (9/(40 pi)) / 243) kernel, B = dr2 / h^2 in
// units of 2^-64.  The sum is (return value) 2^(-59 - 3e) or 2^(-59 - 5e).  EDGE:
// nodes may reach q >= 1, where the kernel is zero (|z| < 2^62 units, see
// fix_spline_scale): s wraps past 1, and from 1 - s = 2^-32 on, where the rounding
// of the float root could take q past 1, the kernel (below 2^-98) is taken as zero.
// (On the upper word, the cheapest of four forms: column densities of 5 channels
// 25.60 ms; a 64-bit comparison 25.80, without the second test 25.64.)
template <bool EDGE = false>
FSG_HD int64_t fix_spline_sum(bool cubic, int64_t za, int64_t zb, uint64_t B, int &e)
{
    const uint64_t ua = (uint64_t)(za < 0 ? -za : za), ub = (uint64_t)(zb < 0 ? -zb : zb);
    const uint64_t um = (za ^ zb) < 0 ? 0ull : (ua < ub ? ua : ub) << 2;
    // t <= 1 - s: shifted by e it stays below 1
    e = fix_clz64(~(B + fix_umulhi64(um, um)) | 1ull);
    const int64_t dz = (zb - za) >> 3;          // rounded down by less than 2^-62
    int64_t sum = 0;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int j = 0; j <= 8; j++) {
        const int64_t z = j == 8 ? zb : za + dz * j;
        const uint64_t u = (uint64_t)(z < 0 ? -z : z) << 2;
        const uint64_t s = B + fix_umulhi64(u, u);
        const uint64_t q = fix_sqrt64(s);
        const uint64_t t = ~q;                  // 1 - q, one unit low (q = 0: no wrap)
        const uint64_t T = t << e;
        int64_t w;
        if (cubic) {
            // q < 1/2: 1 - 6 s (1 - q); else 2 (1 - q)^3
            const bool in = (int64_t)q >= 0;
            const uint64_t m = fix_umulhi64(T, in ? s : T);
            w = in ? ((int64_t)1 << 59) - 6 * (int64_t)(m >> 5)
                   : (int64_t)(fix_umulhi64(m, T) >> 4);
        } else {
            // t^5 - 6 (t - 1/3)^5 + 15 (t - 2/3)^5, positive parts
            const uint64_t third = 6148914691236517205ull;
            const auto pow5 = [](uint64_t x) {
                const uint64_t x2 = fix_umulhi64(x, x);
                return (int64_t)(fix_umulhi64(fix_umulhi64(x2, x2), x) >> 5);
            };
            w = pow5(T);
            if (t > third)
                w -= 6 * pow5((t - third) << e);
            if (t > 2 * third)
                w += 15 * pow5((t - 2 * third) << e);
        }
        if (EDGE && (s < B || (uint32_t)(s >> 32) == 0xFFFFFFFFu))
            w = 0;
        sum += (j == 0 || j == 8) ? w >> 1 : w;
    }
    return sum;
}

}  // namespace fsg
