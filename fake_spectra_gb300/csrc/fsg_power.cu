// 1-D flux power spectrum (fake_spectra/fluxstatistics.py:53-110) with the
// project's own discrete Fourier transforms: in shared memory and 64-bit fixed
// point for lengths that fit, else FP64 passes over global memory.
//
// The reference takes np.fft.rfft of d_F = exp(-s tau) / <F> - 1 along each
// sightline and sums |rfft|^2 / npix^2 over sightlines.  Here two sightlines a
// and b go through one complex transform of z = d_a + i d_b: with Z the
// transform of z, A and B those of d_a and d_b,
//     A_k = (Z_k + conj Z_{N-k}) / 2,   B_k = (Z_k - conj Z_{N-k}) / (2i),
// and by the parallelogram law |A_k|^2 + |B_k|^2 = (|Z_k|^2 + |Z_{N-k}|^2) / 2,
// so the pair's power needs no separation step and the work per sightline is
// half a complex transform, for every length N.
//
// Transforms: the self-sorting Stockham form of the mixed-radix Cooley-Tukey
// algorithm (one pass per radix, as formulated for GPUs by Govindaraju et al.,
// "High performance discrete Fourier transforms on graphics processors", SC
// 2008), radices 16/8/4/2 in registers and odd radices up to 63 by the direct
// DFT with the symmetric pairing of j and R - j (cos and sin sums over half the
// terms).  A length with a prime factor above 63 uses Bluestein's chirp-z
// algorithm over a 7-smooth length M >= 2N - 1: X_k = w_k (a * b)_k with
// w_n = exp(-i pi n^2 / N), a_n = z_n w_n, b_n = conj w_n, the circular
// convolution as conj(FFT(conj(FFT(a) FFT(b)))) / M; |w_k| = 1, so the power is
// |FFT(conj(FFT(a) FFT(b)))_k|^2 / M^2.
//
// GB300 runs FP64 at 1/64 of the FP32 rate, and the FP64 passes are bound by it
// (the reference's test tolerance of 1e-10 relative leaves no room for FP32
// arithmetic): they keep every table (twiddles, cos/sin of the odd radices)
// precomputed, and the odd-radix DFT costs about R FMAs per point.  They serve
// rows too long for shared memory (and, once per length, the chirp filter).  Sums
// over sightlines go in a fixed order: fixed segments of pairs, each summed in
// order, then the segments in order.
#include "fsg_dft_fix.cuh"
#include "fsg_fexp.cuh"
#include "fsg_internal.cuh"

namespace fsg {

namespace {

constexpr int PASS_THREADS = 256;
constexpr int POWER_SEGMENTS = 64;   // fixed: the summation order does not depend on the GPU

__device__ __forceinline__ double2 cadd(double2 a, double2 b)
{
    return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b)
{
    return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// -i a
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }

// exp(-i pi E / 8) a, E in 0..15 known at compile time.
template <int E>
__device__ __forceinline__ double2 rot16(double2 a)
{
    constexpr double H = 0.70710678118654752440;    // cos(pi/4)
    constexpr double C1 = 0.92387953251128675613;   // cos(pi/8)
    constexpr double S1 = 0.38268343236508977173;   // sin(pi/8)
    if constexpr (E == 0)
        return a;
    else if constexpr (E == 4)
        return mul_mi(a);
    else if constexpr (E == 8)
        return make_double2(-a.x, -a.y);
    else if constexpr (E == 2)
        return make_double2(H * (a.x + a.y), H * (a.y - a.x));
    else if constexpr (E == 6)
        return make_double2(H * (a.y - a.x), -H * (a.x + a.y));
    else if constexpr (E == 1)
        return cmul(a, make_double2(C1, -S1));
    else if constexpr (E == 3)
        return cmul(a, make_double2(S1, -C1));
    else if constexpr (E == 9)
        return cmul(a, make_double2(-C1, S1));
    else
        static_assert(E == 0, "rotation not used by the 8- and 16-point DFTs");
}

__device__ __forceinline__ void dft2(double2 &a, double2 &b)
{
    const double2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

// In-place forward DFT of 4 points, natural order.
__device__ __forceinline__ void dft4(double2 &x0, double2 &x1, double2 &x2, double2 &x3)
{
    const double2 t0 = cadd(x0, x2), t1 = csub(x0, x2);
    const double2 t2 = cadd(x1, x3), t3 = mul_mi(csub(x1, x3));
    x0 = cadd(t0, t2);
    x2 = csub(t0, t2);
    x1 = cadd(t1, t3);
    x3 = csub(t1, t3);
}

// Forward DFT of R points held in registers, natural order in and out.  R = 8
// and 16 split as R1 x R2 (R1 = 4): n = R2 n1 + n2, k = k1 + R1 k2: R2 DFTs of 4
// on the stride-R2 subsequences, the twiddles exp(-2 pi i n2 k1 / R), then 4
// DFTs of R2 across them.
template <int R>
__device__ __forceinline__ void dft(double2 (&v)[R]);

template <>
__device__ __forceinline__ void dft<2>(double2 (&v)[2])
{
    dft2(v[0], v[1]);
}

template <>
__device__ __forceinline__ void dft<4>(double2 (&v)[4])
{
    dft4(v[0], v[1], v[2], v[3]);
}

template <int K1, int N2, int R>
__device__ __forceinline__ double2 twid(double2 a)
{
    return rot16<(16 / R) * N2 * K1>(a);
}

template <>
__device__ __forceinline__ void dft<8>(double2 (&v)[8])
{
    // n = 2 n1 + n2
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    // y[n2][k1] sits at v[2 k1 + n2]
    v[3] = twid<1, 1, 8>(v[3]);
    v[5] = twid<2, 1, 8>(v[5]);
    v[7] = twid<3, 1, 8>(v[7]);
    double2 o[8];
    o[0] = cadd(v[0], v[1]);
    o[4] = csub(v[0], v[1]);
    o[1] = cadd(v[2], v[3]);
    o[5] = csub(v[2], v[3]);
    o[2] = cadd(v[4], v[5]);
    o[6] = csub(v[4], v[5]);
    o[3] = cadd(v[6], v[7]);
    o[7] = csub(v[6], v[7]);
#pragma unroll
    for (int i = 0; i < 8; i++)
        v[i] = o[i];
}

template <>
__device__ __forceinline__ void dft<16>(double2 (&v)[16])
{
    // n = 4 n1 + n2: after the first DFTs y[n2][k1] sits at v[4 k1 + n2]
    dft4(v[0], v[4], v[8], v[12]);
    dft4(v[1], v[5], v[9], v[13]);
    dft4(v[2], v[6], v[10], v[14]);
    dft4(v[3], v[7], v[11], v[15]);
    v[5] = twid<1, 1, 16>(v[5]);
    v[9] = twid<2, 1, 16>(v[9]);
    v[13] = twid<3, 1, 16>(v[13]);
    v[6] = twid<1, 2, 16>(v[6]);
    v[10] = twid<2, 2, 16>(v[10]);
    v[14] = twid<3, 2, 16>(v[14]);
    v[7] = twid<1, 3, 16>(v[7]);
    v[11] = twid<2, 3, 16>(v[11]);
    v[15] = twid<3, 3, 16>(v[15]);
    // X[k1 + 4 k2] = DFT4 over n2 of y[n2][k1]
    dft4(v[0], v[1], v[2], v[3]);
    dft4(v[4], v[5], v[6], v[7]);
    dft4(v[8], v[9], v[10], v[11]);
    dft4(v[12], v[13], v[14], v[15]);
    double2 o[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++)
            o[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int i = 0; i < 16; i++)
        v[i] = o[i];
}

// One Stockham pass of radix R (power of two) over `rows` transforms of length
// L: butterfly j of a row reads in[j + r L/R], applies exp(-2 pi i k r / (ns R))
// (k = j mod ns; table tw[k R + r]), and writes out[(j - k) R + k + r ns].
template <int R>
__global__ void __launch_bounds__(PASS_THREADS)
    pass_pow2_kernel(const double2 *__restrict__ in, double2 *__restrict__ out,
                     const double2 *__restrict__ tw, unsigned L, unsigned ns, unsigned total)
{
    const unsigned nb = L / R;
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < total; f += stride) {
        const unsigned p = f / nb, j = f - p * nb;
        const unsigned k = j % ns;
        const double2 *src = in + (size_t)p * L + j;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            v[r] = src[(size_t)r * nb];
        if (ns > 1) {
            const double2 *t = tw + (size_t)k * R;
#pragma unroll
            for (int r = 1; r < R; r++)
                v[r] = cmul(v[r], __ldg(t + r));
        }
        dft<R>(v);
        double2 *dst = out + (size_t)p * L + (size_t)(j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++)
            dst[(size_t)r * ns] = v[r];
    }
}

// One Stockham pass of odd radix R (3 <= R <= 63): G = PASS_THREADS / R
// butterflies per block.  The twiddled inputs v_r go to shared memory, then
// a_q = v_q + v_{R-q} and b_q = v_q - v_{R-q} (q = 1..h, h = (R-1)/2), then
// thread (g, m) forms C = sum_q a_q cos(2 pi q m / R), S = sum_q b_q
// sin(2 pi q m / R) and writes X_m = v_0 + C - i S and X_{R-m} = v_0 + C + i S
// (m = 0: X_0 = v_0 + sum a_q).  cs[t] = (cos, sin)(2 pi t / R).
__global__ void __launch_bounds__(PASS_THREADS)
    pass_odd_kernel(const double2 *__restrict__ in, double2 *__restrict__ out,
                    const double2 *__restrict__ tw, const double2 *__restrict__ cs, unsigned L,
                    unsigned ns, int R, unsigned total)
{
    __shared__ double2 sv[PASS_THREADS];
    __shared__ double2 sab[PASS_THREADS];
    __shared__ double2 scs[64];
    const int h = (R - 1) >> 1;
    const int G = PASS_THREADS / R;
    const unsigned nb = L / R;
    const unsigned f0 = blockIdx.x * (unsigned)G;
    const int t = threadIdx.x;
    if (t < R)
        scs[t] = cs[t];
    if (t < G * R) {
        const int g = t / R, r = t - g * R;
        const unsigned f = f0 + g;
        double2 v = make_double2(0.0, 0.0);
        if (f < total) {
            const unsigned p = f / nb, j = f - p * nb;
            v = in[(size_t)p * L + j + (size_t)r * nb];
            if (ns > 1 && r > 0)
                v = cmul(v, __ldg(tw + (size_t)(j % ns) * R + r));
        }
        sv[g * R + r] = v;
    }
    __syncthreads();
    if (t < G * h) {
        const int g = t / h, q = t - g * h + 1;
        const double2 x = sv[g * R + q], y = sv[g * R + R - q];
        sab[g * 2 * h + q - 1] = cadd(x, y);
        sab[g * 2 * h + h + q - 1] = csub(x, y);
    }
    __syncthreads();
    if (t < G * (h + 1)) {
        const int g = t / (h + 1), m = t - g * (h + 1);
        const unsigned f = f0 + g;
        if (f < total) {
            const unsigned p = f / nb, j = f - p * nb;
            const unsigned k = j % ns;
            double2 *dst = out + (size_t)p * L + (size_t)(j - k) * R + k;
            const double2 v0 = sv[g * R];
            const double2 *a = sab + g * 2 * h, *b = a + h;
            // m = 0 runs the same loop (cos 0 = 1, sin 0 = 0: C = sum a_q,
            // S = 0), so the warp does not split on it
            double2 C = make_double2(0.0, 0.0), S = make_double2(0.0, 0.0);
            int idx = 0;
            for (int q = 0; q < h; q++) {
                idx += m;
                idx -= idx >= R ? R : 0;
                const double c = scs[idx].x, s = scs[idx].y;
                C.x = fma(a[q].x, c, C.x);
                C.y = fma(a[q].y, c, C.y);
                S.x = fma(b[q].x, s, S.x);
                S.y = fma(b[q].y, s, S.y);
            }
            const double re = v0.x + C.x, im = v0.y + C.y;
            dst[(size_t)m * ns] = make_double2(re + S.y, im - S.x);
            if (m > 0)
                dst[(size_t)(R - m) * ns] = make_double2(re - S.y, im + S.x);
        }
    }
}

// (cos, sin)(pi x) for x = 2 m / d with the angle reduced to (-pi, pi].
__device__ __forceinline__ double2 unit_root(long long m, long long d)
{
    m %= d;
    if (m < 0)
        m += d;
    if (2 * m > d)
        m -= d;
    double s, c;
    sincospi(2.0 * (double)m / (double)d, &s, &c);
    return make_double2(c, s);
}

// tw[k R + r] = exp(-2 pi i k r / (ns R)), k < ns, r < R
__global__ void twiddle_kernel(double2 *tw, unsigned ns, int R)
{
    const unsigned n = ns * (unsigned)R;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned k = i / R, r = i - k * R;
        const double2 w = unit_root(-(long long)k * r, (long long)n);
        tw[i] = w;
    }
}

// cs[t] = (cos, sin)(2 pi t / R)
__global__ void odd_table_kernel(double2 *cs, int R)
{
    const int t = threadIdx.x;
    if (t < R)
        cs[t] = unit_root(t, R);
}

// w[n] = exp(-i pi n^2 / N) (n^2 reduced mod 2N in integers)
__global__ void chirp_kernel(double2 *w, unsigned N)
{
    for (unsigned n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        const unsigned long long q = ((unsigned long long)n * n) % (2ull * N);
        w[n] = unit_root(-(long long)q, 2ll * N);
    }
}

// b[m] = conj w[m] (m < N), b[M - m] = conj w[m] (0 < m < N), 0 elsewhere
__global__ void chirp_filter_kernel(const double2 *w, unsigned N, unsigned M, double2 *b)
{
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        double2 v = make_double2(0.0, 0.0);
        if (i < N)
            v = make_double2(w[i].x, -w[i].y);
        else if (i > M - N)
            v = make_double2(w[M - i].x, -w[M - i].y);
        b[i] = v;
    }
}

// z[p][n] = (d_{2p}[n] + i d_{2p+1}[n]) (times w[n] for Bluestein; 0 for
// n >= N), d = exp(-scale tau) inv_mean - 1; a missing second row counts as 0.
__global__ void power_pack_kernel(const double *__restrict__ tau, unsigned rows, unsigned N,
                                  unsigned L, double scale, double inv_mean,
                                  const double2 *__restrict__ chirp,
                                  const uint64_t *__restrict__ etab, double2 *__restrict__ z,
                                  unsigned total)
{
    const ExpScale es = exp_scale(-scale);
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const unsigned p = i / L, n = i - p * L;
        double2 v = make_double2(0.0, 0.0);
        if (n < N) {
            const size_t ra = 2 * (size_t)p;
            v.x = fma(fexp(tau[ra * N + n], -scale, es, etab), inv_mean, -1.0);
            if (ra + 1 < rows)
                v.y = fma(fexp(tau[(ra + 1) * N + n], -scale, es, etab), inv_mean, -1.0);
            if (chirp)
                v = cmul(v, chirp[n]);
        }
        z[i] = v;
    }
}

// a[p][m] = conj(a[p][m] bhat[m])
__global__ void filter_conj_kernel(double2 *a, const double2 *__restrict__ bhat, unsigned L,
                                   unsigned total)
{
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const double2 v = cmul(a[i], bhat[i % L]);
        a[i] = make_double2(v.x, -v.y);
    }
}

// partial[s][k] = sum over the pairs of segment s, in order, of
// |Z_k|^2 + |Z_{(N-k) mod N}|^2.
__global__ void power_partial_kernel(const double2 *__restrict__ Z, unsigned pairs, unsigned L,
                                     unsigned N, unsigned nk, double *partial)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nk)
        return;
    const unsigned s = blockIdx.y;
    const unsigned p0 = (unsigned)((unsigned long long)pairs * s / POWER_SEGMENTS);
    const unsigned p1 = (unsigned)((unsigned long long)pairs * (s + 1) / POWER_SEGMENTS);
    const unsigned k2 = k == 0 ? 0 : N - k;
    double sum = 0.0;
#pragma unroll 4
    for (unsigned p = p0; p < p1; p++) {
        const double2 a = Z[(size_t)p * L + k], b = Z[(size_t)p * L + k2];
        sum += fma(a.x, a.x, a.y * a.y) + fma(b.x, b.x, b.y * b.y);
    }
    partial[(size_t)s * nk + k] = sum;
}

// power[k] += factor * sum over segments (in order) of partial[s][k]
__global__ void power_combine_kernel(const double *partial, unsigned nk, int segments,
                                     double factor, double *power)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nk)
        return;
    double sum = 0.0;
    for (int s = 0; s < segments; s++)
        sum += partial[(size_t)s * nk + k];
    power[k] += factor * sum;
}

// ------------------------------------------------- transforms in shared memory
// Lengths up to FUSED_MAX: a block keeps `batch` sightline pairs in shared memory
// from the optical depth to |Z_k|^2, in the fixed-point arithmetic of
// fsg_dft_fix.cuh; global memory holds tau, the tables and one partial sum per
// block.  Bluestein's two transforms meet in the digit-reversed order the first
// leaves, so neither reorders, and the last pass of the one, the filter and the
// first pass of the other run on the same R points in registers.
//
// 3600 sightlines x 6691 pixels (length 13440, 10 passes of 16 bytes per point
// read and written in global memory and about 116 FP64 operations per point):
// 6.6 ms with the FP64 passes and exponential below, 1.9 ms so.
constexpr int FUSED_THREADS = 512;
constexpr int FUSED_BLOCKS = 152;    // fixed: the summation order does not depend on the GPU
constexpr int FUSED_BATCH = 64;
constexpr size_t FUSED_SMEM = 227 * 1024 - 2048;   // dynamic; the rest holds the row sums
constexpr int FUSED_MAX = (int)((FUSED_SMEM - sizeof(uint64_t) * EXP_TABLE) / sizeof(FixC));

struct FusedArgs {
    const double *tau;
    long long rows;
    unsigned N, L;
    int npass, batch;
    FusedPass pass[FUSED_PASSES];
    const FixW *tw, *chirp, *filter;   // chirp, filter: null for a direct transform
    const unsigned *pos;               // direct: position of frequency k
    const uint64_t *etab;
    double scale, inv_mean;
    int shift;                         // divisions by 2 of all passes
    double *partial;
};

enum { PASS_DIF, PASS_DIT, PASS_FILTER };

template <int R, int KIND>
__device__ __forceinline__ void fused_butterflies(FixC *x, const FixW *tab, unsigned total,
                                                  unsigned m, unsigned L, int e)
{
    for (unsigned f = threadIdx.x; f < total / R; f += FUSED_THREADS) {
        if constexpr (KIND == PASS_DIF)
            dif_butterfly<R>(x, tab, f, m, e);
        else if constexpr (KIND == PASS_DIT)
            dit_butterfly<R>(x, tab, f, m, e);
        else
            filter_butterfly<R>(x, tab, f, L, e);
    }
    __syncthreads();
}

template <int KIND>
__device__ __forceinline__ void fused_pass(FixC *x, const FixW *tab, unsigned total, int R,
                                           unsigned m, unsigned L, int e)
{
    switch (R) {
    case 2: fused_butterflies<2, KIND>(x, tab, total, m, L, e); break;
    case 3: fused_butterflies<3, KIND>(x, tab, total, m, L, e); break;
    case 4: fused_butterflies<4, KIND>(x, tab, total, m, L, e); break;
    case 5: fused_butterflies<5, KIND>(x, tab, total, m, L, e); break;
    case 7: fused_butterflies<7, KIND>(x, tab, total, m, L, e); break;
    case 8: fused_butterflies<8, KIND>(x, tab, total, m, L, e); break;
    default: fused_butterflies<16, KIND>(x, tab, total, m, L, e);
    }
}

__global__ void __launch_bounds__(FUSED_THREADS, 1) power_fused_kernel(FusedArgs a)
{
    extern __shared__ __align__(16) unsigned char fraw[];
    uint64_t *etab = reinterpret_cast<uint64_t *>(fraw);
    FixC *x = reinterpret_cast<FixC *>(fraw + sizeof(uint64_t) * EXP_TABLE);
    __shared__ unsigned long long row_sq[FUSED_BATCH];
    __shared__ int top;
    constexpr int NW = FUSED_THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < EXP_TABLE; k += FUSED_THREADS)
        etab[k] = a.etab[k];
    const ExpScale es = exp_scale(-a.scale);
    const unsigned N = a.N, L = a.L, nk = N / 2 + 1;
    const long long pairs = (a.rows + 1) / 2;
    const long long nbatch = (pairs + a.batch - 1) / a.batch;
    const long long b0 = nbatch * blockIdx.x / gridDim.x, b1 = nbatch * (blockIdx.x + 1) / gridDim.x;
    double *partial = a.partial + (size_t)blockIdx.x * nk;
    for (long long b = b0; b < b1; b++) {
        const long long p0 = b * a.batch;
        const int cnt = (int)(pairs - p0 < a.batch ? pairs - p0 : a.batch);
        if (threadIdx.x < FUSED_BATCH)
            row_sq[threadIdx.x] = 0ull;
        if (threadIdx.x == 0)
            top = 0;
        __syncthreads();
        // d = exp(-scale tau) inv_mean - 1 of both sightlines as doubles; a warp
        // takes one of `parts` stretches of a pair
        const int parts = (NW + cnt - 1) / cnt;
        const unsigned len = ((N + parts - 1) / parts + 31) & ~31u;
        int hmax = 0;
        for (int u = warp; u < cnt * parts; u += NW) {
            const int p = u / parts;
            const unsigned n0 = (u - p * parts) * len, n1 = n0 + len < N ? n0 + len : N;
            const double *ta = a.tau + 2 * (size_t)(p0 + p) * N;
            const bool both = 2 * (p0 + p) + 1 < a.rows;
            double2 *z = reinterpret_cast<double2 *>(x + (size_t)p * L);
            for (unsigned n = n0 + lane; n < n1; n += 32) {
                double2 d = make_double2(0.0, 0.0);
                d.x = fma(fexp(ta[n], -a.scale, es, etab), a.inv_mean, -1.0);
                if (both)
                    d.y = fma(fexp(ta[N + n], -a.scale, es, etab), a.inv_mean, -1.0);
                z[n] = d;
                hmax = max(hmax, max(__double2hiint(d.x) & 0x7FFFFFFF,
                                     __double2hiint(d.y) & 0x7FFFFFFF));
            }
        }
        hmax = __reduce_max_sync(0xffffffffu, hmax);
        if (lane == 0)
            atomicMax(&top, hmax);
        __syncthreads();
        // sums of squares per pair, rounded up, in units of 2^(2 (emax - 21)) of the
        // largest value's exponent
        const int hi = top, ehi = hi >> 20, emax = ehi - 1022;
        for (int u = warp; u < cnt * parts; u += NW) {
            const int p = u / parts;
            const unsigned n0 = (u - p * parts) * len, n1 = n0 + len < N ? n0 + len : N;
            const int2 *z = reinterpret_cast<const int2 *>(x + (size_t)p * L);
            unsigned long long sq = 0;
            for (unsigned n = n0 + lane; n < n1; n += 32)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int h = z[2 * n + c].y & 0x7FFFFFFF;
                    const unsigned q = ((((unsigned)h & 0xFFFFFu) | 0x100000u) >>
                                        min(31, ehi - (h >> 20))) + 1u;
                    sq += (unsigned long long)q * q;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if (lane == 0)
                atomicAdd(&row_sq[p], sq);
        }
        __syncthreads();
        unsigned long long sq = 1;
        for (int p = 0; p < cnt; p++)
            sq = row_sq[p] > sq ? row_sq[p] : sq;
        // the largest power of two that keeps |z|_2 below 2^60.8 (the bound that the
        // radix-16 butterflies and fixc_mul allow): 2^121.6 = 1.515 2^121
        const int l2 = 63 - __clzll((long long)sq);
        const bool high = ((sq << (63 - l2)) >> 32) > 3253500928ull;   // 1.515 2^31
        int sh = ((high ? 120 : 121) - l2) / 2 + 21 - emax;
        if (hi == 0)
            sh = 0;
        const bool bad = ehi == 0x7FF;       // an infinity or NaN: every power is NaN
        // the same in fixed point, times the chirp
        for (unsigned i = threadIdx.x; i < (unsigned)cnt * L; i += FUSED_THREADS) {
            const unsigned n = i % L;
            FixC v = {0, 0};
            if (n < N && !bad) {
                const double2 d = reinterpret_cast<const double2 *>(x)[i];
                if (a.chirp)
                    v = fixc_mul({fix_from_double(d.x, sh + 2), fix_from_double(d.y, sh + 2)},
                                 a.chirp[n], 2, 0);
                else
                    v = {fix_from_double(d.x, sh), fix_from_double(d.y, sh)};
            }
            x[i] = v;
        }
        __syncthreads();
        const unsigned total = (unsigned)cnt * L;
        const int last = a.npass - 1;
        for (int i = 0; i < (a.filter ? last : a.npass); i++)
            fused_pass<PASS_DIF>(x, a.tw + a.pass[i].tw, total, a.pass[i].radix, a.pass[i].m, L,
                                 a.pass[i].e_dif);
        if (a.filter) {
            fused_pass<PASS_FILTER>(x, a.filter, total, a.pass[last].radix, 1, L,
                                    a.pass[last].e_dif);
            for (int i = last - 1; i >= 0; i--)
                fused_pass<PASS_DIT>(x, a.tw + a.pass[i].tw, total, a.pass[i].radix,
                                     a.pass[i].m, L, a.pass[i].e_dit);
        }
        // |Z_k|^2 + |Z_(N-k)|^2; values that square to infinity anyway need no exponent
        // above 900
        const int ex = min(a.shift - sh, 900);
        for (unsigned k = threadIdx.x; k < nk; k += FUSED_THREADS) {
            const unsigned k2 = k == 0 ? 0 : N - k;
            const unsigned i1 = a.pos ? a.pos[k] : k, i2 = a.pos ? a.pos[k2] : k2;
            double sum = b == b0 ? 0.0 : partial[k];
            for (int p = 0; p < cnt; p++) {
                const FixC u = x[(size_t)p * L + i1], v = x[(size_t)p * L + i2];
                const double ux = fix_to_double(u.x, ex), uy = fix_to_double(u.y, ex);
                const double vx = fix_to_double(v.x, ex), vy = fix_to_double(v.y, ex);
                sum += fma(ux, ux, uy * uy) + fma(vx, vx, vy * vy);
            }
            partial[k] = bad ? __longlong_as_double(0x7FF8000000000000ll) : sum;
        }
        __syncthreads();
    }
}

// tw[(q - 1) m + j] = exp(-2 pi i j q / (m R))
__global__ void fused_twiddle_kernel(FixW *tw, unsigned m, int R)
{
    const unsigned n = (R - 1) * m;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned q = i / m + 1, j = i - (q - 1) * m;
        const double2 w = unit_root(-(long long)j * q, (long long)m * R);
        tw[i] = {fix_v62(w.x), fix_v62(w.y)};
    }
}

// largest modulus of b, rounded up (one block)
__global__ void fused_filter_max_kernel(const double2 *b, unsigned M, double *out)
{
    __shared__ unsigned long long top;
    if (threadIdx.x == 0)
        top = 0ull;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < M; i += blockDim.x)
        atomicMax(&top, (unsigned long long)__double_as_longlong(
                            fma(b[i].x, b[i].x, b[i].y * b[i].y)));
    __syncthreads();
    if (threadIdx.x == 0)
        *out = sqrt(__longlong_as_double((long long)top)) * (1.0 + 1e-14);
}

// The chirp, and the filter over its largest modulus in the order the first
// transform leaves.
__global__ void fused_filter_kernel(FusedArgs a, const double2 *w, const double2 *bhat,
                                    const double *top, FixW *chirp, FixW *filter)
{
    const double inv = 1.0 / *top;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < a.L; i += gridDim.x * blockDim.x) {
        if (i < a.N)
            chirp[i] = {fix_v62(w[i].x), fix_v62(w[i].y)};
        unsigned rest = i, k = 0, mul = 1;
        for (int p = 0; p < a.npass; p++) {
            const unsigned d = rest / a.pass[p].m;
            rest -= d * a.pass[p].m;
            k += d * mul;
            mul *= a.pass[p].radix;
        }
        filter[i] = {fix_v62(bhat[k].x * inv), fix_v62(bhat[k].y * inv)};
    }
}

std::vector<long long> prime_factors(long long n)
{
    std::vector<long long> f;
    for (long long p = 2; p * p <= n; p++)
        while (n % p == 0) {
            f.push_back(p);
            n /= p;
        }
    if (n > 1)
        f.push_back(n);
    return f;
}

// smallest 2^a 3^b 5^c 7^d >= m
long long smooth7_at_least(long long m)
{
    long long best = -1;
    for (long long a = 1; a < 2 * m; a *= 2)
        for (long long b = a; b < 2 * m; b *= 3)
            for (long long c = b; c < 2 * m; c *= 5)
                for (long long d = c; d < 2 * m; d *= 7)
                    if (d >= m && (best < 0 || d < best))
                        best = d;
    return best;
}

unsigned grid_for(unsigned long long n, int threads)
{
    const unsigned long long b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : (b > 65535ull * 32 ? 65535ull * 32 : b));
}

// Runs the plan's passes on `rows` transforms in x (scratch y); returns the
// buffer that holds the result.
double2 *run_passes(const PowerPlan &pl, const double2 *tables, double2 *x, double2 *y,
                    unsigned rows, cudaStream_t s, int &launches)
{
    const unsigned L = (unsigned)pl.len;
    for (const PowerPass &ps : pl.passes) {
        const unsigned total = rows * (L / ps.radix);
        const double2 *tw = tables + ps.tw_off;
        const unsigned ns = (unsigned)ps.ns;
        switch (ps.radix) {
        case 2:
            pass_pow2_kernel<2><<<grid_for(total, PASS_THREADS), PASS_THREADS, 0, s>>>(
                x, y, tw, L, ns, total);
            break;
        case 4:
            pass_pow2_kernel<4><<<grid_for(total, PASS_THREADS), PASS_THREADS, 0, s>>>(
                x, y, tw, L, ns, total);
            break;
        case 8:
            pass_pow2_kernel<8><<<grid_for(total, PASS_THREADS), PASS_THREADS, 0, s>>>(
                x, y, tw, L, ns, total);
            break;
        case 16:
            pass_pow2_kernel<16><<<grid_for(total, PASS_THREADS), PASS_THREADS, 0, s>>>(
                x, y, tw, L, ns, total);
            break;
        default: {
            const unsigned G = PASS_THREADS / ps.radix;
            const unsigned blocks = (total + G - 1) / G;
            pass_odd_kernel<<<blocks, PASS_THREADS, 0, s>>>(x, y, tw, tables + ps.cs_off, L, ns,
                                                           ps.radix, total);
        }
        }
        launches++;
        std::swap(x, y);
    }
    return x;
}

}  // namespace

namespace {

// Passes of a fused transform of length len (7-smooth): powers of two first (the
// last pass, over adjacent points, is free of bank conflicts for an odd radix);
// divisions by 2 so that after combining m points at least sqrt(m) is divided out,
// 1 or 2 per pass.  Returns an estimate of the instructions per point, 0 when no
// such plan exists.
int fused_passes(long long len, bool bluestein, std::vector<FusedPass> &ps)
{
    std::vector<int> radix;
    int twos = 0;
    for (long long p : prime_factors(len)) {
        if (p == 2)
            twos++;
        else if (p <= 7)
            radix.push_back((int)p);
        else
            return 0;
    }
    std::vector<int> order;
    if (twos % 4 == 1 && twos > 4) {       // 8 x 4 rather than 16 x 2
        order = {8, 4};
        twos -= 5;
    } else if (twos % 4) {
        order = {1 << twos % 4};
        twos -= twos % 4;
    }
    order.insert(order.begin(), twos / 4, 16);
    order.insert(order.end(), radix.begin(), radix.end());
    if (order.size() > FUSED_PASSES)
        return 0;
    ps.clear();
    int cost = 0;
    unsigned m = (unsigned)len, tw = 0;
    for (int r : order) {
        m /= r;
        FusedPass p;
        p.radix = r;
        p.m = m;
        p.tw = tw;
        if (m > 1)
            tw += (r - 1) * m;
        ps.push_back(p);
        // instructions per point of the butterfly and its twiddles, and of the
        // loads, stores and indices
        cost += 25 + (r == 2 ? 30 : r == 3 ? 53 : r == 4 ? 45 : r == 5 ? 68 : r == 7 ? 100
                                                              : r == 8 ? 61 : 80);
    }
    const auto divisions = [](double half_bits, int done) {
        const int e = (int)std::ceil(half_bits - 1e-9) - done;
        return e < 1 ? 1 : e;
    };
    double bits = 0.0;
    int done = 0;
    for (FusedPass &p : ps) {
        bits += 0.5 * std::log2((double)p.radix);
        if (p.m > 1 || bluestein)
            done += p.e_dif = divisions(bits, done);
        if (p.e_dif > 2)
            return 0;
    }
    bits = 0.0;
    done = 0;
    for (size_t i = ps.size(); bluestein && i-- > 0;) {
        if (ps[i].m > 1)
            done += ps[i].e_dit = divisions(bits, done);
        if (ps[i].e_dit > 2)
            return 0;
        bits += 0.5 * std::log2((double)ps[i].radix);
    }
    return bluestein ? 2 * cost : cost;
}

bool smooth7(long long n)
{
    for (int p : {2, 3, 5, 7})
        while (n % p == 0)
            n /= p;
    return n == 1;
}

// The fused plan of npix pixels, if there is one: the length itself when it is
// 7-smooth, else the cheapest Bluestein length.
bool fused_plan(long long npix, PowerPlan &pl)
{
    pl.bluestein = !smooth7(npix);
    if (!pl.bluestein) {
        pl.len = npix;
        return npix <= FUSED_MAX && (npix == 1 || fused_passes(npix, false, pl.fused) > 0);
    }
    long long best = 0;
    for (long long len = 2 * npix - 1; len <= FUSED_MAX && len < 4 * npix; len++) {
        std::vector<FusedPass> ps;
        const int c = smooth7(len) ? fused_passes(len, true, ps) : 0;
        if (c > 0 && (best == 0 || c * len < best)) {
            best = c * len;
            pl.len = len;
            pl.fused = ps;
        }
    }
    return best > 0;
}

FusedArgs fused_args(const PowerPlan &pl, const void *tables)
{
    FusedArgs a{};
    a.N = (unsigned)pl.npix;
    a.L = (unsigned)pl.len;
    a.npass = (int)pl.fused.size();
    for (int i = 0; i < a.npass; i++) {
        a.pass[i] = pl.fused[i];
        a.shift += a.pass[i].e_dif + a.pass[i].e_dit;
    }
    // twiddles, then the chirp and the filter, or the positions
    a.tw = (const FixW *)tables;
    const FixW *rest = a.tw + pl.len * (pl.fused.empty() ? 0 : 2);
    if (pl.bluestein) {
        a.filter = rest;
        a.chirp = rest + pl.len;
    } else {
        a.pos = (const unsigned *)rest;
    }
    return a;
}

}  // namespace

PowerPlan power_plan(long long npix)
{
    PowerPlan pl;
    pl.npix = npix;
    pl.in_smem = fused_plan(npix, pl);
    if (pl.in_smem && !pl.bluestein) {
        return pl;
    }
    if (!pl.in_smem) {
        pl.fused.clear();
        const std::vector<long long> f = prime_factors(npix);
        long long pmax = 1;
        for (long long p : f)
            pmax = p > pmax ? p : pmax;
        pl.bluestein = pmax > POWER_MAX_ODD_RADIX;
        pl.len = pl.bluestein ? smooth7_at_least(2 * npix - 1) : npix;
    }
    // passes of the FP64 transform (fused: of the chirp filter only)
    std::vector<long long> g = prime_factors(pl.len);
    int twos = 0;
    std::vector<int> radix;
    for (long long p : g)
        if (p == 2)
            twos++;
        else
            radix.push_back((int)p);
    std::vector<int> order;
    for (; twos >= 4; twos -= 4)
        order.push_back(16);
    if (twos)
        order.push_back(1 << twos);
    order.insert(order.end(), radix.begin(), radix.end());
    long long ns = 1, off = 0;
    for (int r : order) {
        PowerPass ps;
        ps.radix = r;
        ps.ns = ns;
        ps.tw_off = off;
        off += ns * r;
        ps.cs_off = -1;
        if (r & 1) {
            ps.cs_off = off;
            off += r;
        }
        pl.passes.push_back(ps);
        ns *= r;
    }
    pl.table_len = off;
    return pl;
}

int power_plan_tables(const PowerPlan &pl, double2 *tables, double2 *chirp, double2 *bhat,
                      double2 *scratch, cudaStream_t s)
{
    int launches = 0;
    for (const PowerPass &ps : pl.passes) {
        if (ps.ns > 1) {
            twiddle_kernel<<<grid_for((unsigned long long)ps.ns * ps.radix, 256), 256, 0, s>>>(
                tables + ps.tw_off, (unsigned)ps.ns, ps.radix);
            launches++;
        }
        if (ps.cs_off >= 0) {
            odd_table_kernel<<<1, 64, 0, s>>>(tables + ps.cs_off, ps.radix);
            launches++;
        }
    }
    if (pl.bluestein) {
        const unsigned N = (unsigned)pl.npix, M = (unsigned)pl.len;
        chirp_kernel<<<grid_for(N, 256), 256, 0, s>>>(chirp, N);
        chirp_filter_kernel<<<grid_for(M, 256), 256, 0, s>>>(chirp, N, M, scratch);
        launches += 2;
        const double2 *r = run_passes(pl, tables, scratch, bhat, 1, s, launches);
        if (r != bhat) {
            cudaMemcpyAsync(bhat, r, sizeof(double2) * M, cudaMemcpyDeviceToDevice, s);
        }
    }
    return launches;
}

size_t power_fused_bytes(const PowerPlan &pl)
{
    if (!pl.in_smem)
        return 0;
    return sizeof(FixW) * (size_t)pl.len * 4 + sizeof(unsigned) * (size_t)pl.npix + 64;
}

// Twiddles (fewer than 2 len), chirp and filter or positions; the filter's largest
// modulus comes back in pl.filter_max (the stream is synchronised).
int power_fused_tables(PowerPlan &pl, const double2 *chirp, const double2 *bhat, void *tables,
                       cudaStream_t s)
{
    int launches = 0;
    const FusedArgs a = fused_args(pl, tables);
    for (const FusedPass &p : pl.fused)
        if (p.m > 1) {
            const unsigned n = (p.radix - 1) * p.m;
            fused_twiddle_kernel<<<grid_for(n, 256), 256, 0, s>>>(
                const_cast<FixW *>(a.tw) + p.tw, p.m, p.radix);
            launches++;
        }
    pl.filter_max = 1.0;
    std::vector<unsigned> pos;
    if (pl.bluestein) {
        double *top = (double *)const_cast<FixW *>(a.filter + 2 * pl.len);
        fused_filter_max_kernel<<<1, 1024, 0, s>>>(bhat, a.L, top);
        fused_filter_kernel<<<grid_for(a.L, 256), 256, 0, s>>>(
            a, chirp, bhat, top, const_cast<FixW *>(a.chirp), const_cast<FixW *>(a.filter));
        launches += 2;
        cudaMemcpyAsync(&pl.filter_max, top, sizeof(double), cudaMemcpyDeviceToHost, s);
    } else {
        pos.resize((size_t)pl.npix);
        for (unsigned i = 0; i < a.N; i++) {
            unsigned rest = i, k = 0, mul = 1;
            for (int p = 0; p < a.npass; p++) {
                const unsigned d = rest / a.pass[p].m;
                rest -= d * a.pass[p].m;
                k += d * mul;
                mul *= a.pass[p].radix;
            }
            pos[k] = i;
        }
        cudaMemcpyAsync(const_cast<unsigned *>(a.pos), pos.data(), sizeof(unsigned) * pos.size(),
                        cudaMemcpyHostToDevice, s);
    }
    cudaStreamSynchronize(s);
    return launches;
}

int power_fused(const PowerPlan &pl, const void *tables, const uint64_t *etab, const double *tau,
                long long rows, double scale, double inv_mean, double vmax, double *partial,
                double *power, cudaStream_t s)
{
    FusedArgs a = fused_args(pl, tables);
    a.tau = tau;
    a.rows = rows;
    a.etab = etab;
    a.scale = scale;
    a.inv_mean = inv_mean;
    a.partial = partial;
    // short rows: as many pairs per block as fit, but no fewer blocks than SMs
    const long long pairs = (rows + 1) / 2;
    long long batch = std::min<long long>(FUSED_MAX / pl.len, FUSED_BATCH);
    batch = std::min(batch, (pairs + FUSED_BLOCKS - 1) / FUSED_BLOCKS);
    a.batch = (int)std::max(1ll, batch);
    const long long nbatch = (pairs + a.batch - 1) / a.batch;
    const int blocks = (int)std::min<long long>(nbatch, FUSED_BLOCKS);
    const size_t smem = sizeof(uint64_t) * EXP_TABLE + sizeof(FixC) * (size_t)a.batch * a.L;
    cudaFuncSetAttribute(power_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    power_fused_kernel<<<blocks, FUSED_THREADS, smem, s>>>(a);
    double norm = 1.0 / ((double)pl.npix * (double)pl.npix);
    if (pl.bluestein) {
        const double g = pl.filter_max / (double)pl.len;
        norm *= g * g;
    }
    const unsigned nk = a.N / 2 + 1;
    power_combine_kernel<<<(nk + 127) / 128, 128, 0, s>>>(partial, nk, blocks, 0.5 * vmax * norm,
                                                          power);
    return 2;
}

long long power_pairs_per_chunk(const PowerPlan &pl, long long nspec)
{
    const long long pairs = (nspec + 1) / 2;
    long long c = (512ll << 20) / (16 * pl.len);
    c = c < 1 ? 1 : c;
    return c < pairs ? c : pairs;
}

int power_chunk(const PowerPlan &pl, const double2 *tables, const double2 *chirp,
                const double2 *bhat, const uint64_t *etab, const double *tau, long long rows,
                double scale, double inv_mean, double vmax, double2 *a, double2 *b,
                double *partial, double *power, cudaStream_t s)
{
    int launches = 0;
    const unsigned N = (unsigned)pl.npix, L = (unsigned)pl.len;
    const unsigned pairs = (unsigned)((rows + 1) / 2);
    const unsigned total = pairs * L;
    power_pack_kernel<<<grid_for(total, 256), 256, 0, s>>>(
        tau, (unsigned)rows, N, L, scale, inv_mean, pl.bluestein ? chirp : nullptr, etab, a,
        total);
    launches++;
    double2 *r = run_passes(pl, tables, a, b, pairs, s, launches);
    double norm = 1.0 / ((double)N * (double)N);
    if (pl.bluestein) {
        filter_conj_kernel<<<grid_for(total, 256), 256, 0, s>>>(r, bhat, L, total);
        launches++;
        r = run_passes(pl, tables, r, r == a ? b : a, pairs, s, launches);
        norm /= (double)L * (double)L;
    }
    const unsigned nk = N / 2 + 1;
    power_partial_kernel<<<dim3((nk + 127) / 128, POWER_SEGMENTS), 128, 0, s>>>(r, pairs, L, N,
                                                                              nk, partial);
    power_combine_kernel<<<(nk + 127) / 128, 128, 0, s>>>(partial, nk, POWER_SEGMENTS,
                                                          0.5 * vmax * norm, power);
    launches += 2;
    return launches;
}

size_t power_partials(long long npix)
{
    return (size_t)std::max(POWER_SEGMENTS, FUSED_BLOCKS) * (npix / 2 + 1);
}

}  // namespace fsg
