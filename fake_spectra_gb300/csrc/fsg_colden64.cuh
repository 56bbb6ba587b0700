// Column-density deposit, FP64 form (included by fsg_deposit.cu inside its
// anonymous namespace, before fsg_fast64.cuh).
//
// Values as kern_frac<double> (absorption.cpp:53-115): the pixels inside the
// kernel support with 1 - q^2 >= 2^-8 at both ends go through
// fix_spline_sum (integer arithmetic; the pixel edges are the reference's
// rounded doubles, taken into integers), the rest - the clipped end pixels,
// pairs that graze the support, the top hat and Voronoi cells - through the
// reference's unfused double arithmetic.  Near the support's edge 1 - q
// cancels and only the same double operations give the reference's tails.
// Per warp: one lane per pair sets up a chunk; the interior pixels of each
// pair go 32 per step; the remaining pixels of the whole chunk are dealt out
// evenly to the lanes, so the FP64 work runs in full warps.
// Measured (GB300): 3600 sightlines x 6691 pixels of a 256^3 snapshot, 1.0e7
// pairs of about 75 pixels: deposit 590 ms with 9 FP64 nodes at every pixel, 70
// ms so (integer instructions of the interior nodes, then the FP64 pixels).

constexpr int C64_THREADS = 512;
constexpr int C64_CHUNK = 32;

struct __align__(16) StageC64 {
    double pos1, zlow;       // particle position; first pixel
    double zrange, dr2;
    double inv_h;            // 2^62 / h
    double dens;
    uint64_t B;              // dr2 / h^2, units of 2^-64
    float smooth;
    int j0, kmax;            // bin of the first pixel; last pixel
    int ilo, ihi;            // interior pixels [ilo, ihi] (empty: ihi < ilo)
    int pad;
};
static_assert(sizeof(StageC64) == 80, "StageC64 is five 16-byte words");

// Pixels left to the FP64 form: [0, ilo) and (ihi, kmax].
__device__ __forceinline__ int edge_count64(const StageC64 &st)
{
    return st.ihi < st.ilo ? st.kmax + 1 : st.ilo + st.kmax - st.ihi;
}
__device__ __forceinline__ int edge_pixel64(const StageC64 &st, int i)
{
    return st.ihi < st.ilo || i < st.ilo ? i : i - st.ilo + st.ihi + 1;
}

// False for a pair that misses the sightline (kmax = -1); ok = false for a
// window beyond the limit.
__device__ __forceinline__ bool stagec64_setup(const LineParams &lp, const PairInput &in,
                                               double btk, StageC64 &st, bool &ok)
{
    Colden c;
    ok = true;
    st.kmax = -1;
    st.ilo = 0;
    st.ihi = -1;
    if (!c.setup(lp, in, btk))
        return false;
    if (!c.ok) {
        ok = false;
        return false;
    }
    st.pos1 = c.pos1;
    st.zlow = (double)c.zlow;
    st.zrange = c.zrange;
    st.dr2 = c.dr2;
    st.dens = c.dens;
    st.smooth = in.smooth;
    st.j0 = wrap_bin(c.zlow, lp.nbins);
    st.kmax = (int)c.kmax;
    st.inv_h = 0.0;
    st.B = 0;
    st.pad = 0;
    if ((lp.kernel == SPH_CUBIC || lp.kernel == SPH_QUINTIC) && btk > 0.0) {
        const double h2 = c.smooth * c.smooth;
        const double l2 = 0.99609375 * h2 - c.dr2;   // (1 - 2^-8) h^2 - dr2
        if (l2 > 0.0 && h2 < 1e200 && h2 > 1e-200) {
            const double zl = sqrt(l2) * (1.0 - 1e-9);
            const double a = ceil((c.pos1 - zl) / btk - st.zlow + 1e-6);
            const double b = floor((c.pos1 + zl) / btk - st.zlow - 1e-6) - 1.0;
            const int ilo = (int)fmax(a, 0.0), ihi = (int)fmin(b, (double)st.kmax);
            if (b >= a && ihi >= ilo) {
                st.ilo = ilo;
                st.ihi = ihi;
                st.inv_h = 4611686018427387904.0 / c.smooth;
                st.B = __double2ull_rn(c.dr2 / h2 * 18446744073709551616.0);
            }
        }
    }
    return true;
}

// kern_frac of interior pixel k.
__device__ __forceinline__ double colden64_interior(const StageC64 &st, int kernel, double btk,
                                                    int k)
{
    const double plow = __dsub_rn(__dmul_rn(btk, st.zlow + (double)k), st.pos1);
    const double phigh = __dadd_rn(plow, btk);
    int e;
    const bool cubic = kernel == SPH_CUBIC;
    const int64_t sum = fix_spline_sum(cubic, __double2ll_rn(plow * st.inv_h),
                                       __double2ll_rn(phigh * st.inv_h), st.B, e);
    const double norm = cubic ? 32. / 4 / PI_D : 9. / 40 / PI_D * 243.0;
    const int sh = 59 + 3 + (cubic ? 3 : 5) * e;   // 2^-59, the node spacing's 1/8, 2^-3e
    return (phigh - plow) * norm * exp_down(__ll2double_rn(sum), sh);
}

// kern_frac of any pixel k in the reference's double arithmetic.
__device__ __forceinline__ double colden64_direct(const StageC64 &st, int kernel, double btk,
                                                  int k)
{
    const double plow = __dsub_rn(__dmul_rn(btk, st.zlow + (double)k), st.pos1);
    return kern_frac<double>(kernel, plow, __dadd_rn(plow, btk), (double)st.smooth, st.dr2,
                             st.zrange);
}

// Deals the FP64 pixels of a staged chunk of n pairs to the lanes: f(pair,
// pixel) for each, whole warp.
template <class F>
__device__ __forceinline__ void for_each_edge64(const StageC64 *stage, int n, int lane, F f)
{
    // at most 32 (2^26 + 1) pixels: fits unsigned
    unsigned incl = lane < n ? (unsigned)edge_count64(stage[lane]) : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += v;
    }
    const unsigned total = __shfl_sync(0xffffffffu, incl, 31);
    for (unsigned base = 0; base < total; base += 32) {
        const unsigned it = base + lane;
        // the pair of item it: the number of pairs whose items end at or before it
        int p = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned end = __shfl_sync(0xffffffffu, incl, p + o - 1);
            if (end <= it)
                p += o;
        }
        const unsigned start = __shfl_sync(0xffffffffu, incl, p > 0 ? p - 1 : 0);
        if (it < total) {
            const StageC64 &st = stage[p];
            f(p, edge_pixel64(st, (int)(it - (p > 0 ? start : 0u))));
        }
    }
}

__device__ __forceinline__ int col_bin(int j0, int k, int nbins)
{
    return (int)(((unsigned)j0 + (unsigned)k) % (unsigned)nbins);
}

// One chunk of pairs [cb, cb + n) of a sightline, whole warp.
__device__ __forceinline__ void deposit_colden64(const DepositArgs &a, int axis, long long cb,
                                                 int n, int S, unsigned long long *lo,
                                                 unsigned long long *hi, int *bad,
                                                 StageC64 *stage, double btk, int lane)
{
    const int nbins = a.lp.nbins, kernel = a.lp.kernel;
    if (lane < n) {
        const PairInput in = load_pair(a.p, a.pl, cb + lane, axis, false, a.dev_err);
        bool ok;
        stagec64_setup(a.lp, in, btk, stage[lane], ok);
        if (!ok) {
            atomicOr(a.dev_err, (unsigned)DEVERR_WINDOW_LIMIT);
            *bad = 1;
        }
    }
    __syncwarp();
    for (int q = 0; q < n; q++) {
        const StageC64 &st = stage[q];
        for (int k = st.ilo + lane; k <= st.ihi; k += 32)
            accumulate<double, 0>(a.dev_err,
                                  __dmul_rn(st.dens, colden64_interior(st, kernel, btk, k)),
                                  col_bin(st.j0, k, nbins), S, lo, hi, bad);
    }
    for_each_edge64(stage, n, lane, [&](int p, int k) {
        const StageC64 &st = stage[p];
        accumulate<double, 0>(a.dev_err, __dmul_rn(st.dens, colden64_direct(st, kernel, btk, k)),
                              col_bin(st.j0, k, nbins), S, lo, hi, bad);
    });
    __syncwarp();
}
