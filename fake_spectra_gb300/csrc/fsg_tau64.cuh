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
//  * Pair constants are set up by one lane per pair (chunks of T64_CHUNK pairs
//    per warp) and staged in shared memory; the direct walk repeats them in
//    all 32 lanes.
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
//  * Sightlines are few in many FP64 calls (fewer than the SMs), so a
//    thread-block cluster can share one: its blocks take chunks of pairs from
//    one counter, add into their own accumulators and sum them through
//    distributed shared memory at the end (integer sums: the same bits for
//    every cluster size).
//
//  * Inside vmp the 7 profiles are summed in 64-bit integers
//    (fsg_voigt_fix.cuh), whose instructions issue 16 to 64 times as fast as
//    FP64 ones.
//
// Measured (GB300, whole call): 72 sightlines x 6691 pixels of a 256^3
// snapshot 1766 ms with the direct walk, 255 ms with FP64 profiles inside vmp,
// 20.5 ms so; 400 sightlines x 1115 pixels of 128^3, CIV (little wing) 1028,
// 588 and 26.8 ms.
//
// Pairs outside the series' conditions (a <= 0 or a > 0.1, non-finite
// constants, a pixel width within 1e-9 of a sub-sampling boundary) take the
// direct walk.

constexpr int T64_R = 16;
constexpr int T64_M = 16;
constexpr int T64_LEVELS = 3;
constexpr int T64_DIST = 3;
constexpr int T64_RUNS = 2 * T64_LEVELS - 1;
constexpr int T64_THREADS = 512;
constexpr int T64_CHUNK = 8;

constexpr int S64_SKIP = 1 << 30, S64_CAREFUL = 1 << 29, S64_TILES = 1 << 28;
constexpr int S64_FIX = 1 << 27;         // node sums in integers (fsg_voigt_fix.cuh)
constexpr int S64_NP = (1 << 27) - 1;

struct __align__(16) Stage64 {
    double vel, zd;          // particle velocity; its pixel zmax as a double
    double inv_b, inv_lo;    // 1/b as a sum of two doubles
    double aa, vmp;
    double scale;            // amp dens / velfac x node spacing / (npoints - 1)
    double u1;               // node spacing / b: node i at (i - 3) u1
    double cg, ck;           // S64_FIX: factors of the two integer sums
    union {
        double w[NODES];     // kernel weights
        FixPair fix;
    };
    double A[T64_R];         // far-wing coefficients times vmp^(-2r)
    float vsure;             // tiles out to this |V| hold no pixel below tautail
    int j0, flags, pad;
};
static_assert(sizeof(Stage64) % 16 == 0, "Stage64 rows stay aligned");

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

// Far-wing coefficients of the node sum.  H(u, a) ~ sum_j gamma_j u^(-2j),
//   gamma_j = 1/sqrt(pi) sum_m (-1)^m a^(2m+1) c_(j-1-m) C(2j-1, 2m+1)
// (A&S 7.1.23 expanded in a/u; m <= 3 is exact to 1e-17 for a <= 0.1 beyond
// u = 12), and summed over symmetric nodes A_r = sum_j gamma_j C(2r-1, 2r-2j)
// M_(r-j), M the even moments.  Here V and U are in units of vmp, so that no
// power overflows.
__device__ __forceinline__ void far_coefficients64(const double *w, double u1, double a,
                                                   double vmp, double *A)
{
    const double iv = 1.0 / vmp, iv2 = iv * iv, a2 = a * a;
    const double q1 = (u1 * iv) * (u1 * iv), q2 = 4.0 * q1, q3 = 9.0 * q1;
    double p1 = w[2] + w[4], p2 = w[1] + w[5], p3 = w[0] + w[6];
    double M[T64_R];
    M[0] = p1 + p2 + p3 + w[3];
#pragma unroll
    for (int m = 1; m < T64_R; m++) {
        p1 *= q1;
        p2 *= q2;
        p3 *= q3;
        M[m] = p1 + p2 + p3;
    }
    double gam[T64_R + 1];
    double f = a * FSG_INV_SQRT_PI * iv2;
#pragma unroll
    for (int j = 1; j <= T64_R; j++) {
        double s = 0.0;
#pragma unroll
        for (int m = 3; m >= 0; m--)
            if (m <= j - 1)
                s = fma(s, -a2, asym_c(j - 1 - m) * binom_d(2 * j - 1, 2 * m + 1));
        gam[j] = f * s;
        f *= iv2;
    }
#pragma unroll
    for (int r = 1; r <= T64_R; r++) {
        double acc = 0.0;
#pragma unroll
        for (int j = 1; j <= r; j++)
            acc = fma(gam[j] * binom_d(2 * r - 1, 2 * r - 2 * j), M[r - j], acc);
        A[r - 1] = acc;
    }
}

// Fills a pair's stage; false for a pair that misses the sightline.
__device__ __forceinline__ bool stage64_setup(const LineParams &lp, const PairInput &in,
                                              Stage64 &st)
{
    Tau64 s;
    if (!s.setup(lp, in))
        return false;
    const double u1 = s.deltav * s.inv_b, vk = s.bintov * s.inv_b;
    const double umax = 3.0 * fabs(u1);
    const double vmp = fmax(4.5 * umax, umax + 12.0);
    // tau_kern_outer sub-samples (singleabs.h:104-126): uniform over the pair
    // unless the pixel width, which the reference rounds per pixel, is at a
    // boundary
    const double ratio = s.bintov / s.half_b;
    const double half_ratio = 0.5 * ratio;
    const double near = rint(half_ratio);
    bool careful = !(s.aa > 0.0 && s.aa <= 0.1) || !(fabs(ratio - 1.0) > 1e-9) ||
                   (ratio >= 1.0 && !(fabs(half_ratio - near) > 1e-9 * half_ratio));
    const double npd = ratio < 1.0 ? 1.0 : 2.0 * ceil(half_ratio) + 1.0;
    careful = careful || !(npd <= MAX_SUBSAMPLES);
    const int np = careful ? 1 : (int)npd;
    double sc = s.ampd * s.deltav / s.velfac;
    if (np > 1)
        sc /= (double)(np - 1);
    careful = careful || !(fabs(sc) < 1e300) || !(umax < 1e6) || !(fabs(s.vel) < 1e12);
    st.vel = s.vel;
    st.zd = (double)s.zmax;
    st.inv_b = s.inv_b;
    st.aa = s.aa;
    st.scale = sc;
    st.u1 = u1;
    st.vmp = vmp;
    st.inv_lo = fma(-s.inv_b, s.btherm, 1.0) * s.inv_b;
    st.j0 = s.bin0(lp.nbins);
    bool tiles = false;
    float vsure = 0.f;
    // the integer node sums: V within their range for every pixel step that
    // reaches inside vmp (one step of 32 pixels and its outer edge beyond it)
    double wmax = 0.0;
#pragma unroll
    for (int i = 0; i < NODES; i++)
        wmax = fmax(wmax, s.w[i]);
    const bool fix = !careful && s.aa >= FIXV_A_MIN && s.aa <= FIXV_A_MAX && wmax > 0.0 &&
                     fabs(sc) * wmax > 1e-200 && vmp + umax + 34.0 * vk < FIXV_MAX;
    if (fix) {
        const double inv_w = 1.0 / wmax;
        fix_pair_damping(s.aa, st.fix);
        st.fix.u1 = __double2ll_rn(u1 * 9007199254740992.0);
#pragma unroll
        for (int i = 0; i < NODES; i++) {
            const double q = s.w[i] * inv_w * 4611686018427387904.0;   // 2^62
            st.fix.w[i] = fix62(min(__double2ull_rn(q), (1ull << 62) - 1ull) << 2);
        }
        const double c = sc * wmax * 8.673617379884035e-19;            // 2^-60
        st.cg = c * exp(s.aa * s.aa);
        st.ck = c * s.aa;
    } else {
#pragma unroll
        for (int i = 0; i < NODES; i++)
            st.w[i] = s.w[i];
    }
    if (!careful) {
        far_coefficients64(s.w, u1, s.aa, vmp, st.A);
        tiles = sc > 0.0 && st.A[0] > 0.0;
#pragma unroll
        for (int r = 1; r < T64_R; r++)
            tiles = tiles && st.A[r] >= 0.0;
        if (!(lp.tautail > 0.0)) {
            vsure = __int_as_float(0x7f800000);
        } else if (tiles) {
            // y = (vmp/V)^2 where the wing equals tautail, by Newton's method
            // from above (the polynomial is increasing and convex)
            const double yt = lp.tautail / (sc * st.A[0] * (np > 1 ? (double)(np - 1) : 1.0));
            if (yt < 1.0 && yt > 1e-30) {
                float c[T64_R];
                const double inv0 = 1.0 / st.A[0];
#pragma unroll
                for (int r = 0; r < T64_R; r++)
                    c[r] = (float)(st.A[r] * inv0);
                const float t = (float)yt;
                float y = t;
#pragma unroll 1
                for (int it = 0; it < 4; it++) {
                    float h = c[T64_R - 1], d = (float)T64_R * c[T64_R - 1];
#pragma unroll
                    for (int r = T64_R - 2; r >= 0; r--) {
                        h = fmaf(h, y, c[r]);
                        d = fmaf(d, y, (float)(r + 1) * c[r]);
                    }
                    y -= (h * y - t) / d;
                }
                vsure = y > 0.f ? 0.999f * (float)vmp * rsqrtf(y) : 0.f;
            } else if (yt <= 1e-30) {
                vsure = 1e14f;
            }
        }
    }
    st.vsure = vsure;
    st.flags = np | (careful ? S64_CAREFUL : 0) | (tiles ? S64_TILES : 0) |
               (fix ? S64_FIX : 0);
    st.pad = 0;
    return true;
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

// cos(pi j / 32), j = 0 .. 63 (Chebyshev nodes and their transform)
__shared__ double s_cos64[64];

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

// A pair's node sum times scale at velocity v from the line centre (all lanes
// call it).
__device__ __forceinline__ double inner64(const Stage64 &st, const Rows64 &rows, double v)
{
    const double V = v * st.inv_b;
    const double av = fabs(V);
    const double vmp = st.vmp;
    if (__all_sync(0xffffffffu, av >= vmp)) {
        const double q = vmp / av, y = q * q;
        double s;
        if (__all_sync(0xffffffffu, av >= 4.0 * vmp)) {
            s = st.A[6];
#pragma unroll
            for (int r = 5; r >= 0; r--)
                s = fma(s, y, st.A[r]);
        } else {
            s = 0.0;
            if (!__all_sync(0xffffffffu, av >= 2.0 * vmp)) {
                s = st.A[15];
#pragma unroll
                for (int r = 14; r >= 11; r--)
                    s = fma(s, y, st.A[r]);
            }
#pragma unroll
            for (int r = 10; r >= 0; r--)
                s = fma(s, y, st.A[r]);
        }
        return st.scale * (s * y);
    }
    if (st.flags & S64_FIX) {
        // V to 2^-53: the product's rounding error is added back
        const double lo = fma(v, st.inv_lo, fma(v, st.inv_b, -V));
        const int64_t vi = __double2ll_rn(V * 9007199254740992.0) +
                           __double2ll_rn(lo * 9007199254740992.0);
        int64_t sg, sk;
        int eg, ek;
        fix_node_sums(st.fix, vi, rows, s_pow2, sg, eg, sk, ek);
        return fma(exp_down(st.cg, eg), __ll2double_rn(sg),
                   exp_down(st.ck, ek) * __ll2double_rn(sk));
    }
    const double aa = st.aa, u1 = st.u1;
    double total = 0.0;
#pragma unroll 1
    for (int i = 0; i < NODES; i++)
        total = fma(voigt_f64(fma((double)(i - 3), u1, -V), aa), st.w[i], total);
    return st.scale * total;
}

// The pair's optical depth at a low pixel edge vlow (velocity from the line
// centre), tau_kern_outer's rule.
__device__ __forceinline__ double outer64(const Stage64 &st, const Rows64 &rows, double vlow,
                                          double bintov)
{
    const double vhigh = __dadd_rn(vlow, bintov);
    const int np = st.flags & S64_NP;
    if (np == 1)
        return inner64(st, rows, __dmul_rn(0.5, __dadd_rn(vhigh, vlow)));
    const double dv = (vhigh - vlow) / (np - 1);
    double total = 0.0;
#pragma unroll 1
    for (int i = 0; i < np; i++) {
        const double v = i == np - 1 ? vhigh : __dadd_rn(__dmul_rn((double)i, dv), vlow);
        const double f = inner64(st, rows, v);
        total = (i == 0 || i == np - 1) ? fma(0.5, f, total) : total + f;
    }
    return total;
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
    const double zd = st.zd, vel = st.vel;
    const int w0 = tl.w0;
    const bool tiles = w0 > 0 && (st.flags & S64_TILES);
    int kmp = 0, ksure = 0;
    if (tiles) {
        const float vk = (float)(bintov * st.inv_b);
        kmp = (int)fminf((float)st.vmp / vk * 1.000001f + 2.f, 1e9f);
        ksure = (int)fminf(st.vsure / vk - 2.f, 1e9f);
    }
    for (int dir = 0; dir < 2; dir++) {
        int c0 = dir == 0 ? st.j0 : -st.j0;
        if (dir == 1 && st.j0 == 0)
            c0 = -nbins;
        int limit = dir == 0 ? nbins : 0;
        int k = 0;
        while (k < half) {
            int c = c0 + k;
            if (c >= limit) {   // the window wraps to the other end of the row
                c0 -= nbins;
                c -= nbins;
            }
            int len = 32;
            if (tiles) {
                // first place a tile of the smallest width may start
                const int ts = (max(c, c0 + max(kmp, T64_DIST * w0)) + w0 - 1) & -w0;
                const int e = min(limit, c0 + min(half, ksure));
                if (ts == c && c + w0 <= e) {
                    // runs of tiles: widths going up with the distance, then
                    // down towards e
                    int rn[T64_RUNS], rc[T64_RUNS];
                    int top = 0, cur = c, total = 0;
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
                        // going down: level T64_RUNS - 1 - r, when reached
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
                        total += rn[r];
                    for (int base = 0; base < total * T64_M; base += 32) {
                        const int it = base + lane;
                        const bool on = it < total * T64_M;
                        int t = on ? it / T64_M : 0;
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
                        const int w = w0 << (2 * l);
                        // node m of the tile, pixels from its lowest bin
                        const double x = fma(0.5 * (double)w, 1.0 + s_cos64[2 * m + 1], -0.5);
                        const int kt = ct - c0;
                        const double off = (double)(dir == 0 ? kt : -kt - w) + x;
                        const double vlow = fma(off, bintov, fma(zd, bintov, -vel));
                        const double v = outer64(st, rows, vlow, bintov);
                        if (on) {
                            const int tile = dir == 0 ? ct / w : -(ct / w) - 1;
                            const int first = l == 0 ? tl.first[0]
                                                     : (l == 1 ? tl.first[1] : tl.first[2]);
                            accumulate<double, 0>(a.dev_err, v, first + tile * T64_M + m, S, tlo,
                                                  thi, bad);
                        }
                    }
                    k = cur - c0;
                    continue;
                }
                if (ts > c)
                    len = min(len, ts - c);
            }
            len = min(len, limit - c);
            const int koff = dir == 0 ? k + lane : -1 - k - lane;
            const double vlow = __dsub_rn(__dmul_rn(zd + (double)koff, bintov), vel);
            const double v = outer64(st, rows, vlow, bintov);
            const bool valid = lane < len && k + lane < half;
            const unsigned m = __ballot_sync(0xffffffffu, valid && v < tautail);
            const int last = m ? (__ffs(m) - 1) : 31;
            if (valid && lane <= last)
                accumulate<double, 0>(a.dev_err, v,
                                      dir == 0 ? c + lane : -(c + lane) - 1, S, lo, hi, bad);
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
    if (lane < n) {
        const PairInput in = load_pair(a.p, a.pl, cb + lane, axis, true, a.dev_err);
        if (!stage64_setup(a.lp, in, stage[lane]))
            stage[lane].flags = S64_SKIP;
    }
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
