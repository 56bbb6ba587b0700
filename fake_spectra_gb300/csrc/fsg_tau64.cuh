// Optical-depth deposit, FP64 form (included by fsg_deposit.cu inside its
// anonymous namespace).
//
// Same sum as walk_tau<0>: per (particle, sightline) pair the 7-node kernel
// sum of Voigt profiles at every pixel of its window (singleabs.h:104-167,
// absorption.cpp:239-278), added exactly in 128-bit fixed point.  What differs
// is how the values are formed.  GB300 runs FP64 at 1/64 of the FP32 rate, so
// the evaluation of 7 profiles per pixel (about 850 FP64 operations) bounds
// the direct walk; most of those pixels lie far out in the damping wing.
//
//  * Pair constants are set up a chunk of pairs at a time, a few lanes per pair,
//    and staged in shared memory; the direct walk repeats them in all 32 lanes.
//  * Beyond vmp = max(4.5 Umax, Umax + 12) (Umax = max |U_i|, in units of b)
//    the node sum is one polynomial in (vmp/V)^2: the asymptotic series of H
//    in 1/u summed over the symmetric nodes, 16 terms, truncation below 2e-16
//    of the sum (mpmath, all weight on the outer nodes); 11 terms from 2 vmp
//    and 7 from 4 vmp are as exact.
//  * Farther out the pair adds its value at T64_M Chebyshev nodes of a tile of
//    pixels instead of at each pixel.  Tiles come in three widths (w0, 4 w0,
//    16 w0); a tile is used once its near edge is T64_DIST widths from the
//    line centre, where 16 nodes interpolate 1/V^2 to 2e-17 and 1/V^4 (a few
//    percent of the value) to 1.2e-15.  A pixel finally adds the interpolants
//    of the tiles that hold it.
//  * The window ends after the first pixel below tautail.  The far wing falls
//    monotonically (non-negative coefficients, checked), so tiles inside
//    0.999 of the radius where it equals tautail hold no such pixel; the pixel
//    that ends the window is found by the pixel walk.
//  * All of it after the velocity is integer arithmetic (fsg_voigt_fix.cuh), whose
//    instructions issue 16 to 64 times as fast as FP64 ones: the 7 profiles
//    inside vmp, the wing's polynomial, the value itself.
//
// Measured (GB300, whole call): 72 sightlines x 6691 pixels of a 256^3 snapshot
// 1766 to 2092 ms with the direct walk, 255 ms with FP64 profiles inside vmp,
// 20.5 ms with integer profiles, 10.5 ms with all of the above and sightlines
// shared between blocks (fsg_fast64.cuh); 400 sightlines x 1115 pixels of 128^3,
// CIV (little wing) 1030, 588, 26.8 and 16.4 ms.  Bound by the integer pipes and
// the latency of their chains (2.35 instructions per cycle, FP64 pipe 37% busy).
//
// Pairs outside the series' conditions (a <= 0 or a > 0.1, non-finite
// constants, a pixel width within 1e-9 of a sub-sampling boundary) take the
// direct walk.

constexpr int T64_R = 16;
constexpr int T64_M = 16;
constexpr int T64_LEVELS = 3;
constexpr int T64_DIST = 3;
constexpr int T64_RUNS = 2 * T64_LEVELS - 1;
constexpr int T64_THREADS = 768;
constexpr int T64_CHUNK = 8;

constexpr int S64_SKIP = 1 << 30, S64_CAREFUL = 1 << 29, S64_TILES = 1 << 28;
constexpr int S64_FIX = 1 << 27;         // node sums in integers (fsg_voigt_fix.cuh)
constexpr int S64_NP = (1 << 27) - 1;

struct __align__(16) Stage64 {
    double vel, zoff;        // particle velocity; its pixel zmax less I2D_BIAS
    double base2;            // twice the velocity of pixel zmax's low edge - vel
    uint64_t ib;             // 1/b = ib 2^eb
    uint64_t vmp53;          // vmp, units of 2^-53
    FixFar far;
    FixNum cg, ck;           // S64_FIX: factors of the two integer sums
    union {
        struct {             // the node sum in FP64
            double w[NODES]; // kernel weights
            double u1;       // node spacing / b: node i at (i - 3) u1
            double aa, half_inv_b, scale;
        } dbl;
        FixPair fix;
    };
    int eb;
    int neg;                 // the pair's amplitude is negative
    float vk, vmp;           // pixel width / b; vmp
    float vsure;             // tiles out to this |V| hold no pixel below tautail
    int j0, flags, pad;
};
static_assert(sizeof(Stage64) % 16 == 0, "Stage64 rows stay aligned");

// (double)i for a 32-bit i without the conversion unit: the bits of 2^52 + 2^31 + i
// less that constant (one FP64 add, which a following add can absorb).
constexpr double I2D_BIAS = 4503601774854144.0;
__device__ __forceinline__ double i2d_biased(int i)
{
    return __hiloint2double(0x43300000, i ^ (int)0x80000000);
}

__host__ __device__ constexpr double binom_d(int n, int k)
{
    double r = 1.0;
    for (int i = 1; i <= k; i++)
        r = r * (double)(n - k + i) / (double)i;
    return r;
}

// (2k-1)!! / 2^k
__host__ __device__ constexpr double asym_c(int k)
{
    double r = 1.0;
    for (int i = 1; i <= k; i++)
        r *= (2.0 * i - 1.0) * 0.5;
    return r;
}

// C(2r-1, 2r-2j) of the far-wing coefficients, row r - 1, column j - 1 (r >= j), and
// asym_c(j-1-m) C(2j-1, 2m+1), row j - 1, column m.
struct FarTables {
    double binom[T64_R][T64_R];
    double gam[T64_R][4];
};
constexpr FarTables far_tables()
{
    FarTables t{};
    for (int r = 1; r <= T64_R; r++)
        for (int j = 1; j <= r; j++)
            t.binom[r - 1][j - 1] = binom_d(2 * r - 1, 2 * r - 2 * j);
    for (int j = 1; j <= T64_R; j++)
        for (int m = 0; m < 4 && m <= j - 1; m++)
            t.gam[j - 1][m] = asym_c(j - 1 - m) * binom_d(2 * j - 1, 2 * m + 1);
    return t;
}
__device__ const FarTables d_far = far_tables();

// x^n, n >= 0
__device__ __forceinline__ double pow_n(double x, int n)
{
    double r = 1.0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        if (n & (1 << b))
            r *= x;
        x *= x;
    }
    return r;
}

// Sets up the pairs [cb, cb + n) of a chunk, whole warp, 32 / chunk lanes per
// pair: the lanes of a pair form its geometry together (the same instructions)
// and share the node weights and the far-wing coefficients.  (One lane per pair
// takes 1200 FP64 instructions per chunk, 19 thousand cycles of the SM's FP64
// pipe; a third of the kernel on short windows.)
//
// Far-wing coefficients of the node sum: H(u, a) ~ sum_j gamma_j u^(-2j),
//   gamma_j = 1/sqrt(pi) sum_m (-1)^m a^(2m+1) c_(j-1-m) C(2j-1, 2m+1)
// (A&S 7.1.23 expanded in a/u; m <= 3 is exact to 1e-17 for a <= 0.1 beyond
// u = 12), and summed over symmetric nodes A_r = sum_j gamma_j C(2r-1, 2r-2j)
// M_(r-j), M the even moments.  V and U are in units of vmp, so that no power
// overflows.
__device__ __forceinline__ void stage64_chunk(const DepositArgs &a, int axis, long long cb, int n,
                                              Stage64 *stage, double bintov, int lane)
{
    const LineParams &lp = a.lp;
    const int L = 32 / a.chunk;              // lanes per pair: 4, 8 or 16 (chunk 8, 4, 2)
    const int sub = lane & (L - 1), pair = lane / L;
    const unsigned group = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane & ~(L - 1));
    Stage64 &st = stage[pair];
    // scratch within the row until its fields are written: gamma and M (bytes 0 to
    // 255), the weights (from byte 256)
    double *scratch = reinterpret_cast<double *>(&st);
    static_assert(sizeof(Stage64) >= 39 * sizeof(double), "scratch fits the row");
    int flags = S64_SKIP;
    double vel = 0, inv_b = 1, aa = 0, u1 = 0, vmp = 1, sc = 0, zd = 0, vk = 0, iv2 = 0;
    double btherm = 1, vdr2 = 0, vsmooth = 1, vhigh = 0, deltav = 0, umax = 0;
    int np = 1, j0 = 0;
    if (pair < n) {
        // SingleAbsorber (singleabs.h:81-90) and add_tau_particle's constants, as Tau64
        const PairInput in = load_pair(a.p, a.pl, cb + pair, axis, true, a.dev_err);
        const bool vor = lp.kernel == VORONOI;
        double pos1 = (double)in.ppos;
        bool miss;
        if (vor) {
            const double lim = 2 * lp.vbox / lp.velfac;
            miss = in.dr2 > lim || (double)in.smooth > lim;
            pos1 = (in.dr2 + (double)in.smooth) / 2.;
        } else {
            miss = (double)__fmul_rn(in.smooth, in.smooth) - in.dr2 <= 0;
        }
        if (!miss) {
            btherm = lp.bfac * sqrt((double)in.temp);
            inv_b = 1.0 / btherm;
            vel = __dadd_rn(__dmul_rn(lp.velfac, pos1), (double)in.pvel);
            vdr2 = vor ? lp.velfac * in.dr2 : (lp.velfac * in.dr2) * lp.velfac;
            vsmooth = lp.velfac * (double)in.smooth;
            aa = lp.voigt_fac / btherm;
            const double vs2 = __dmul_rn(vsmooth, vsmooth);
            vhigh = vs2 > vdr2 ? __dsqrt_rn(__dsub_rn(vs2, vdr2)) : 0;
            if (vor)
                vhigh = (vdr2 > 0 && vsmooth > 0) ? (vsmooth - vdr2) / 2. : 0.;
            deltav = 2. * vhigh / NGRID;
            const double amp = lp.sigma_a / sqrt(PI_D) * (LIGHT_KMS / btherm);
            sc = amp * (double)in.dens * deltav / lp.velfac;
            zd = floor(vel / bintov);
            u1 = deltav * inv_b;
            vk = bintov * inv_b;
            umax = 3.0 * fabs(u1);
            vmp = fmax(4.5 * umax, umax + 12.0);
            // tau_kern_outer sub-samples (singleabs.h:104-126): uniform over the
            // pair unless the pixel width, which the reference rounds per pixel,
            // is at a boundary
            const double ratio = bintov / (btherm / 2.), half_ratio = 0.5 * ratio;
            const double npd = ratio < 1.0 ? 1.0 : 2.0 * ceil(half_ratio) + 1.0;
            const bool careful =
                !(aa > 0.0 && aa <= 0.1) || !(fabs(ratio - 1.0) > 1e-9) ||
                (ratio >= 1.0 && !(fabs(half_ratio - rint(half_ratio)) > 1e-9 * half_ratio)) ||
                !(npd <= MAX_SUBSAMPLES) || !(fabs(sc) < 1e200) || !(vmp < 900.0) ||
                !(fabs(vel) < 1e12) || !(fabs(zd) < 1e15) || !(fabs(sc) > 1e-200 || sc == 0.0);
            np = careful ? 1 : (int)npd;
            if (np > 1)
                sc /= (double)(np - 1);
            flags = careful ? S64_CAREFUL : 0;
            if (!careful && sc == 0.0)
                flags = S64_SKIP;            // adds nothing at any pixel
        }
    }
    // node weights, unfused and in the reference's order (singleabs.h:150-156)
    if (flags == 0) {
        j0 = wrap_bin((long long)zd, lp.nbins);
        for (int i = sub; i < NODES; i += L) {
            const double v = __dsub_rn(__dmul_rn((double)(i + 1), deltav), vhigh);
            scratch[2 * T64_R + i] = node_weight<double>(
                lp.kernel, __ddiv_rn(__dsqrt_rn(__dadd_rn(vdr2, __dmul_rn(v, v))), vsmooth));
        }
    }
    __syncwarp();
    double w[NODES], wsum = 0.0, wmax = 0.0;
#pragma unroll
    for (int i = 0; i < NODES; i++)
        w[i] = 0.0;
    if (flags == 0) {
#pragma unroll
        for (int i = 0; i < NODES; i++) {
            w[i] = scratch[2 * T64_R + i];
            wsum += w[i];
            wmax = fmax(wmax, w[i]);
        }
        if (wsum == 0.0)
            flags = S64_SKIP;
        else if (!(wsum > 1e-100))
            flags = S64_CAREFUL;
    }
    if (flags == 0) {
        const double iv = 1.0 / vmp;
        iv2 = iv * iv;
        const double q1 = (u1 * iv) * (u1 * iv);
        const double f0 = aa * FSG_INV_SQRT_PI, ma2 = -aa * aa;
        for (int k = sub; k < T64_R; k += L) {
            // M_k and gamma_(k+1), V and U in units of vmp
            const double p = pow_n(q1, k);
            const double p4 = pow_n(4.0, k), p9 = pow_n(9.0, k);
            scratch[T64_R + k] =
                p * (fma(w[1] + w[5], p4, fma(w[0] + w[6], p9, w[2] + w[4]))) + (k ? 0.0 : w[3]);
            const double *g = d_far.gam[k];
            scratch[k] = f0 * pow_n(iv2, k) * iv2 *
                         fma(ma2, fma(ma2, fma(ma2, __ldg(g + 3), __ldg(g + 2)), __ldg(g + 1)),
                             __ldg(g));
        }
    }
    __syncwarp();
    double A[T64_R / 4];                     // this lane's A_r, r = 1 + sub + L i
    bool mono = true;
#pragma unroll
    for (int i = 0; i < T64_R / 4; i++) {
        const int r = sub + L * i;           // r - 1
        A[i] = 0.0;
        if (flags == 0 && r < T64_R) {
            double acc = 0.0;
            for (int j = 0; j <= r; j++)
                acc = fma(scratch[j] * __ldg(&d_far.binom[r][j]), scratch[T64_R + r - j], acc);
            A[i] = acc;
            mono = mono && acc >= 0.0;
        }
    }
    const double A0 = __shfl_sync(0xffffffffu, A[0], lane & ~(L - 1));
    mono = (__ballot_sync(0xffffffffu, mono) & group) == group;
    if (flags == 0 && !(A0 > 0.0))
        flags = S64_CAREFUL;
    __syncwarp();                            // the scratch is free again
    if (pair >= n)
        return;
    if (flags != 0) {
        if (sub == 0)
            st.flags = flags;
        return;
    }
    const bool tiles = sc > 0.0 && mono;
    // the coefficients in units of A_1, and as floats (in the row's union) for the
    // stop radius
    const double inv0 = 1.0 / A0;
    float *cf = reinterpret_cast<float *>(&st.dbl);
    static_assert(sizeof(st.dbl) >= T64_R * sizeof(float), "float coefficients fit");
#pragma unroll
    for (int i = 0; i < T64_R / 4; i++) {
        const int r = sub + L * i;
        if (r < T64_R) {
            const double c = A[i] * inv0;
            cf[r] = (float)c;
            if (r > 0)
                st.far.A[r - 1] = __double2ll_rn(scalbn(c, 61 + r));
        }
    }
    __syncwarp(group);
    float vsure = 0.f;
    if (!(lp.tautail > 0.0)) {
        vsure = __int_as_float(0x7f800000);
    } else if (tiles) {
        // y = (vmp/V)^2 where the wing equals tautail, by Newton's method from
        // above (the polynomial is increasing and convex)
        const double yt = lp.tautail / (sc * A0 * (np > 1 ? (double)(np - 1) : 1.0));
        if (yt < 1.0 && yt > 1e-30) {
            const float t = (float)yt;
            float y = t;
#pragma unroll 1
            for (int it = 0; it < 4; it++) {
                float h = cf[T64_R - 1], d = (float)T64_R * h;
#pragma unroll
                for (int r = T64_R - 2; r >= 0; r--) {
                    const float c = cf[r];
                    h = fmaf(h, y, c);
                    d = fmaf(d, y, (float)(r + 1) * c);
                }
                y -= (h * y - t) / d;
            }
            vsure = y > 0.f ? 0.999f * (float)vmp * rsqrtf(y) : 0.f;
        } else if (yt <= 1e-30) {
            vsure = 1e14f;
        }
    }
    __syncwarp(group);
    // the integer node sums: V within their range for every pixel step that
    // reaches inside vmp (one step of 32 pixels and its outer edge beyond it)
    const bool fix = aa >= FIXV_A_MIN && aa <= FIXV_A_MAX && vmp + umax + 34.0 * vk < FIXV_MAX;
    const double asc = fabs(sc);
    if (fix) {
        const double inv_w = 4611686018427387904.0 / wmax;   // 2^62
#pragma unroll
        for (int i = 0; i < NODES; i++)
            if (sub == (i & (L - 1)))
                st.fix.w[i] = fix62(min(__double2ull_rn(w[i] * inv_w), (1ull << 62) - 1ull) << 2);
    } else if (sub == 0) {
#pragma unroll
        for (int i = 0; i < NODES; i++)
            st.dbl.w[i] = w[i];
        st.dbl.u1 = u1;
        st.dbl.aa = aa;
        st.dbl.half_inv_b = 0.5 * inv_b;
        st.dbl.scale = sc;
    }
    if (sub == 1) {
        if (fix) {
            fix_pair_damping(aa, st.fix);
            st.fix.u1 = __double2ll_rn(u1 * 9007199254740992.0);
            // exp(a^2), a <= 2^-8
            const double a2 = aa * aa;
            st.cg = fix_num(asc * wmax * fma(a2, fma(a2, fma(a2, 1. / 6, 0.5), 1.0), 1.0));
            st.ck = fix_num(asc * wmax * aa);
        }
        const FixNum v2 = fix_num(vmp * vmp), cA = fix_num(asc * A0);
        st.far.vs = v2.m;
        st.far.ev = v2.e;
        st.far.cA = cA.m;
        st.far.eA = cA.e;
    }
    if (sub == 0) {
        st.vel = vel;
        st.zoff = zd - I2D_BIAS;
        st.base2 = 2.0 * fma(zd, bintov, -vel);
        // 1/b to 64 bits
        const FixNum nb = fix_num(inv_b);
        const double lo = fma(-inv_b, btherm, 1.0) * inv_b;
        st.ib = nb.m + (uint64_t)__double2ll_rn(scalbn(lo, -nb.e));
        st.eb = nb.e;
        // beyond this V every node is in its asymptotic range; a little above vmp,
        // so that (vmp / V)^2 stays below 1 after rounding
        st.vmp53 = (uint64_t)__double2ll_rn(vmp * 1.000001 * 9007199254740992.0);
        st.neg = sc < 0.0;
        st.vk = (float)vk;
        st.vmp = (float)vmp;
        st.vsure = vsure;
        st.j0 = j0;
        st.pad = 0;
        st.flags = np | (tiles ? S64_TILES : 0) | (fix ? S64_FIX : 0);
    }
}

// Tile layout of a launch: w0 (64, 128 or 256; a power of two) and the first
// node of each level.  Level l has nbins / (w0 4^l) tiles.
struct Tiles64 {
    int w0, first[T64_LEVELS], nodes;
};

__host__ __device__ inline Tiles64 tiles64_layout(int w0, int nbins)
{
    Tiles64 t;
    t.w0 = w0;
    int n = 0;
    for (int l = 0; l < T64_LEVELS; l++) {
        t.first[l] = n;
        n += w0 > 0 ? T64_M * (nbins / (w0 << (2 * l))) : 0;
    }
    t.nodes = n;
    return t;
}

// cos(pi j / 32), j = 0 .. 63 (Chebyshev nodes and their transform), and the
// nodes' places in a tile, (1 + cos(pi (2m + 1) / 32)) / 2 of its width
__shared__ double s_cos64[64];
__shared__ double s_node64[T64_M];

// K table rows: in shared memory the 16-byte words of row r are exchanged by
// the bits of r / 2, so that 8 lanes reading the same word of different rows
// spread over all banks.
struct Rows64 {
    const FixRow *rows;
    int mask;                // 3 in shared memory, 0 in global memory
    __device__ __forceinline__ FixRow load(int r) const
    {
        const char *p = reinterpret_cast<const char *>(rows + r);
        const int sw = ((r >> 1) & mask) << 4;
        union {
            int4 q[4];
            FixRow row;
        } u;
#pragma unroll
        for (int i = 0; i < 4; i++)
            u.q[i] = *reinterpret_cast<const int4 *>(p + ((i << 4) ^ sw));
        return u.row;
    }
};

__device__ const FixRow d_fix_rows[FSG_FIX_ROWS] = FSG_FIX_INIT;
__device__ const Fix62 d_fix_pow2[64] = FSG_FIX_POW2_INIT;
__shared__ Fix62 s_pow2[64];

// d 2^-e (e >= 0) of a normal d that stays normal
__device__ __forceinline__ double exp_down(double d, int e)
{
    return __hiloint2double(__double2hiint(d) - (e << 20), __double2loint(d));
}

// The node sum in FP64, for dampings outside the integer form's range.
__device__ __noinline__ double nodes64(const Stage64 &st, double v2)
{
    const double V = v2 * st.dbl.half_inv_b, aa = st.dbl.aa, u1 = st.dbl.u1;
    double total = 0.0;
#pragma unroll 1
    for (int i = 0; i < NODES; i++)
        total = fma(voigt_f64(fma((double)(i - 3), u1, -V), aa), st.dbl.w[i], total);
    return st.dbl.scale * total;
}

// A pair's node sum times scale at the velocity v2 / 2 from the line centre (all
// lanes call it).  Everything after the velocity is integer arithmetic; the
// number of wing terms follows the largest y = (vmp / V)^2 of the warp: 16 terms
// leave 2e-16 of the sum at y = 1, and 11, 7, 6 and 4 no more than that below y
// = 2^-2, 2^-4, 2^-6 and 2^-10 (term r + 1 is at most (2r + 1) (y / 20)^r).
__device__ __forceinline__ double inner64(const Stage64 &st, const Rows64 &rows, double v2)
{
    const FixV v = fix_velocity(v2, st.ib, st.eb);
    const uint64_t v53 = fix_v53(v);
    uint64_t m;
    int e;
    if (__all_sync(0xffffffffu, v53 >= st.vmp53)) {
        int ye;
        const uint64_t ym = fix_far_y(st.far, v, ye);
        const int top = __reduce_max_sync(0xffffffffu, ye + 64);   // y < 2^top
        const int n = top > -2 ? 16 : (top > -4 ? 11 : (top > -6 ? 7 : (top > -10 ? 6 : 4)));
        m = fix_far_sum(st.far, n, ym, ye, e);
    } else {
        if (!(st.flags & S64_FIX))
            return nodes64(st, v2);
        int64_t sg, sk;
        int eg, ek;
        fix_node_sums(st.fix, v2 < 0.0 ? -(int64_t)v53 : (int64_t)v53, rows, s_pow2, sg, eg, sk,
                      ek);
        m = fix_combine(sg, eg, st.cg, sk, ek, st.ck, e);
    }
    return fix_double(m, e, (uint64_t)st.neg);
}

// Adds a finite value to a 128-bit accumulator.
__device__ __forceinline__ void add64(unsigned *dev_err, double v, int j, int S,
                                      unsigned long long *lo, unsigned long long *hi)
{
    unsigned long long l, h;
    if (to_fixed(v, S, l, h))
        fixed_add(lo, hi, j, l, h);
    else
        atomicOr(dev_err, (unsigned)DEVERR_FIXED_OVERFLOW);
}

__device__ __noinline__ void walk64_careful(const DepositArgs &a, const PairInput &in, int S,
                                            unsigned long long *lo, unsigned long long *hi,
                                            int *bad, int lane)
{
    Tau64 s;
    if (!s.setup(a.lp, in))
        return;
    Counters ct{};
    walk_tau<0, false, 0>(a, s, S, lo, hi, bad, lane, nullptr, ct);
}

// One staged pair, whole warp.  The walk runs in the coordinate c = bin
// (forward) or c = -(bin + 1) (backward), increasing in both directions;
// k = c - c0 counts pixels from the line centre, and c0 drops by nbins where
// the window wraps.  Tiles start where c is a multiple of their width.
__device__ __forceinline__ void walk_tau64(const DepositArgs &a, const Tiles64 &tl,
                                           const Rows64 &rows, const Stage64 &st, int S,
                                           unsigned long long *lo,
                                           unsigned long long *hi, unsigned long long *tlo,
                                           unsigned long long *thi, int *bad, int lane,
                                           double bintov)
{
    const int nbins = a.lp.nbins, half = nbins / 2;
    const double tautail = a.lp.tautail;
    // v < tautail on the bits: exact for tautail >= 0, whatever the sign of v
    const bool tail_bits = tautail >= 0.0;
    const int w0 = tl.w0;
    const bool tiles = w0 > 0 && (st.flags & S64_TILES);
    int kmp = 0, ksure = 0;
    if (tiles) {
        // one pixel for the centre's place in its own, up to half a pixel for the first
        // sample of the pixel about the first node: every sample of every node is
        // beyond vmp, so tiles never take the node sums, whose range ends a step of 32
        // pixels beyond it
        kmp = (int)fminf(st.vmp / st.vk * 1.00001f + 3.f, 1e9f);
        ksure = (int)fminf(st.vsure / st.vk - 2.f, 1e9f);
    }
    const int np = st.flags & S64_NP;
    for (int dir = 0; dir < 2; dir++) {
        int c0 = dir == 0 ? st.j0 : -st.j0;
        if (dir == 1 && st.j0 == 0)
            c0 = -nbins;
        const int limit = dir == 0 ? nbins : 0;
        int k = 0;
        // runs of tiles being deposited: counts, first places, the items (tile,
        // node) done and in all, the place behind them
        int rn[T64_RUNS] = {}, rc[T64_RUNS] = {}, base = 0, items = 0, cend = 0;
        while (k < half) {
            int c = c0 + k;
            if (c >= limit) {   // the window wraps to the other end of the row
                c0 -= nbins;
                c -= nbins;
            }
            int len = 32;
            if (items == 0 && tiles) {
                // first place a tile of the smallest width may start
                const int ts = (max(c, c0 + max(kmp, T64_DIST * w0)) + w0 - 1) & -w0;
                const int e = min(limit, c0 + min(half, ksure));
                if (ts == c && c + w0 <= e) {
                    // widths going up with the distance, then down towards e
                    int top = 0, cur = c;
                    bool up = true;
#pragma unroll
                    for (int l = 0; l < T64_LEVELS - 1; l++) {
                        const int wn = w0 << (2 * (l + 1));
                        const int t = (max(cur, c0 + max(kmp, T64_DIST * wn)) + wn - 1) & -wn;
                        rc[l] = cur;
                        rn[l] = 0;
                        if (up && t + wn <= e) {
                            rn[l] = (t - cur) / (w0 << (2 * l));
                            cur = t;
                            top = l + 1;
                        } else {
                            up = false;
                        }
                    }
#pragma unroll
                    for (int r = T64_LEVELS - 1; r < T64_RUNS; r++) {
                        const int l = T64_RUNS - 1 - r;
                        rc[r] = cur;
                        rn[r] = 0;
                        if (l <= top) {
                            rn[r] = (e - cur) / (w0 << (2 * l));
                            cur += rn[r] * (w0 << (2 * l));
                        }
                    }
#pragma unroll
                    for (int r = 0; r < T64_RUNS; r++)
                        items += T64_M * rn[r];
                    base = 0;
                    cend = cur;
                } else if (ts > c) {
                    len = min(len, ts - c);
                }
            }
            // one evaluation per lane (a single call site keeps the code within the
            // instruction cache: four copies of it cost a third more time): a tile
            // node or a pixel, as twice the velocity of its first and last sample
            double vfirst, vlast, width2;
            int idx = 0;
            bool on;
            if (items > 0) {
                on = base + lane < items;
                const int it = min(base + lane, items - 1);
                int t = it / T64_M;
                const int m = it % T64_M;
                int l = 0, ct = rc[0];
                bool found = false;
#pragma unroll
                for (int r = 0; r < T64_RUNS; r++) {
                    const int lr = r < T64_LEVELS ? r : T64_RUNS - 1 - r;
                    if (!found) {
                        if (t < rn[r]) {
                            found = true;
                            l = lr;
                            ct = rc[r] + t * (w0 << (2 * lr));
                        } else {
                            t -= rn[r];
                        }
                    }
                }
                const int w = w0 << (2 * l), kt = ct - c0;
                const int tile = dir == 0 ? ct / w : -(ct / w) - 1;
                idx = (l == 0 ? tl.first[0] : (l == 1 ? tl.first[1] : tl.first[2])) +
                      tile * T64_M + m;
                // node m lies s_node64[m] of the tile's width from its low edge, in the
                // middle of the pixel evaluated for it
                const int koff = dir == 0 ? kt : -kt - w;
                const double off2 = fma(i2d_biased(2 * w) - I2D_BIAS, s_node64[m],
                                        i2d_biased(2 * koff - 1) - I2D_BIAS);
                vfirst = fma(off2, bintov, st.base2);
                width2 = 2.0 * bintov;
                vlast = np == 1 ? vfirst + bintov : vfirst + width2;
            } else {
                // the pixel's edges rounded as the reference rounds them
                len = min(len, limit - c);
                on = lane < len && k + lane < half;
                idx = dir == 0 ? c + lane : -(c + lane) - 1;
                const double z = i2d_biased(dir == 0 ? k + lane : -1 - k - lane) + st.zoff;
                const double vlow = __dsub_rn(__dmul_rn(z, bintov), st.vel);
                const double vhigh = __dadd_rn(vlow, bintov);
                vfirst = vlow + vlow;
                width2 = 2.0 * (vhigh - vlow);
                vlast = np == 1 ? __dadd_rn(vhigh, vlow) : vhigh + vhigh;
            }
            // tau_kern_outer (singleabs.h:104-126): the pixel centre, or a trapezoid
            double v = 0.0, dv = 0.0;
            if (np > 1)
                dv = width2 / (np - 1);
#pragma unroll 1
            for (int i = 0; i < np; i++) {
                double at = vlast;
                if (i < np - 1)
                    at = fma(i2d_biased(i) - I2D_BIAS, dv, vfirst);
                const double f = inner64(st, rows, at);
                if (np == 1)
                    v = f;
                else
                    v = i == 0 || i == np - 1 ? fma(0.5, f, v) : v + f;
            }
            if (items > 0) {
                if (on)
                    add64(a.dev_err, v, idx, S, tlo, thi);
                base += 32;
                if (base >= items) {
                    k = cend - c0;
                    items = 0;
                }
                continue;
            }
            const bool below = tail_bits ? __double_as_longlong(v) < __double_as_longlong(tautail)
                                         : v < tautail;
            const unsigned m = __ballot_sync(0xffffffffu, on && below);
            const int last = m ? (__ffs(m) - 1) : 31;
            if (on && lane <= last)
                add64(a.dev_err, v, idx, S, lo, hi);
            if (m)
                break;
            k += len;
        }
    }
}

// One chunk of pairs [cb, cb + n) of a sightline, whole warp.
__device__ __forceinline__ void deposit_tau64(const DepositArgs &a, const Tiles64 &tl,
                                              const Rows64 &rows, int axis, long long cb, int n,
                                              int S, unsigned long long *lo,
                                              unsigned long long *hi, unsigned long long *tlo,
                                              unsigned long long *thi, int *bad, Stage64 *stage,
                                              double bintov, int lane)
{
    stage64_chunk(a, axis, cb, n, stage, bintov, lane);
    __syncwarp();
    for (int q = 0; q < n; q++) {
        const Stage64 &st = stage[q];
        if (st.flags & S64_SKIP)
            continue;
        if (st.flags & S64_CAREFUL) {
            const PairInput in = load_pair(a.p, a.pl, cb + q, axis, true, a.dev_err);
            walk64_careful(a, in, S, lo, hi, bad, lane);
            continue;
        }
        walk_tau64(a, tl, rows, st, S, lo, hi, tlo, thi, bad, lane, bintov);
    }
    __syncwarp();
}
