// Voronoi-mesh sightline cells (kernel 2): the GPU form of
// IndexTable::assign_cells (fake_spectra/index_table.cpp:152-223).
//
// A sightline is sampled at N = int(box / 0.1) points x_i = (i + 1/2) box/N.
// Each point belongs to the nearest of the sightline's particles (periodic
// 3-D distance in double, the first in ascending particle order on a tie, as
// the reference's strict '<' over its std::map gives).  The reference walks
// the points in order; the cell of point 0 may wrap around the box, and the
// walk stops at the first point past box/2 that belongs to it again.  Here:
//   1. the cell of point 0 (first_cell_kernel),
//   2. the stop point: the first such point past box/2 (wrap_point_kernel),
//   3. first/last/count of the points of every cell before the stop point
//      (cell_extent_kernel),
//   4. each cell's float segment [left, right], rounded as the reference's
//      float array is, with the contiguity the reference asserts checked by
//      the count (cell_segment_kernel).
// The nearest-cell search works on blocks of VOR_POINTS consecutive points.  A
// cell's distance changes by at most w over a stretch of half-length w, so only
// cells with (distance at the middle, along the sightline) - w within the least
// upper bound over all cells can own a point: a few of the sightline's hundreds.
// Each point then takes the float minimum over those, and the reference's
// double distance decides only among cells within the float error bound of it.
// Ties go to the smaller particle index, which is the reference's order, so the
// pair lists need no order of their own.
// Measured (GB300, the whole FP64 optical-depth call): 100 sightlines x 200000
// points, 700 cells each: 39.2 ms with every point against every cell and the
// pairs sorted on the host, 2.5 ms so.
#include "fsg_internal.cuh"

namespace fsg {

namespace {

constexpr double RESO = 0.1;   // index_table.h:8
constexpr int VOR_THREADS = 256;
constexpr int VOR_PER = 4;                           // points per thread
constexpr int VOR_POINTS = VOR_THREADS * VOR_PER;    // points per block
constexpr int VOR_CAND = 512;                        // candidate cells held per block

struct VorArgs {
    const float *pos;          // [3N]
    const int *part;           // pairs by sightline, in any order
    const long long *off;      // [L+1]
    const int *axis;           // [L]
    const double *cofm;        // [3L]
    int nlos, npoint;
    double box, reso;
};

__device__ __forceinline__ double min_image(double d, double box)
{
    d = fabs(d);
    return d > box / 2. ? box - d : d;
}

__device__ __forceinline__ float min_image_f(float d, float box)
{
    d = fabsf(d);
    return d > 0.5f * box ? box - d : d;
}

struct VorShared {
    float4 cand[VOR_CAND];     // {x, y, z} and the cell's index in the list
    int ncand;
    int ubound;                // bits of the least upper bound (a non-negative float)
};

// The sightline of a block: its cells and fixed transverse coordinates.
struct VorLine {
    long long e0;
    int m, ax, i1, i2;
    double yp, zp;
    float boxf, ypf, zpf;
    __device__ __forceinline__ VorLine(const VorArgs &a, int l)
    {
        e0 = a.off[l];
        m = (int)(a.off[l + 1] - e0);
        ax = a.axis[l];
        i1 = ax % 3;
        i2 = (ax + 1) % 3;
        yp = a.cofm[3 * (size_t)l + i1];
        zp = a.cofm[3 * (size_t)l + i2];
        boxf = (float)a.box;
        ypf = (float)yp;
        zpf = (float)zp;
    }
    __device__ __forceinline__ float3 cell(const VorArgs &a, int k) const
    {
        const float *p = &a.pos[3 * (size_t)__ldg(&a.part[e0 + k])];
        return make_float3(__ldg(p + ax - 1), __ldg(p + i1), __ldg(p + i2));
    }
    // float distance of a cell from the point x, the part along the sightline changed
    // by shift (to zero at least; NaN stays NaN).  The image of a cell outside the box
    // has a negative distance, whose magnitude counts.
    __device__ __forceinline__ float dist(float3 q, float x, float shift) const
    {
        float dx = fabsf(min_image_f(q.x - x, boxf)) + shift;
        dx = dx < 0.f ? 0.f : dx;
        const float dy = min_image_f(q.y - ypf, boxf), dz = min_image_f(q.z - zpf, boxf);
        return sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    }
    __device__ __forceinline__ float margin(float d) const { return 1e-6f * boxf + 1e-5f * d; }
    __device__ __forceinline__ double dist64(const VorArgs &a, float3 q, double x) const
    {
        const double ddx = min_image((double)q.x - x, a.box);
        const double ddy = min_image((double)q.y - yp, a.box);
        const double ddz = min_image((double)q.z - zp, a.box);
        return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)),
                                    __dmul_rn(ddz, ddz)));
    }
};

// Cells that can be nearest to a point within w of xm along the sightline, to
// sh.cand (whole block; sh.ncand > VOR_CAND: more than it holds).
__device__ void gather_candidates(const VorArgs &a, const VorLine &L, float xm, float w,
                                  VorShared &sh)
{
    if (threadIdx.x == 0) {
        sh.ncand = 0;
        sh.ubound = 0x7f7fffff;
    }
    __syncthreads();
    float u = 3.4e38f;
    for (int k = threadIdx.x; k < L.m; k += blockDim.x)
        u = fminf(u, L.dist(L.cell(a, k), xm, w));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
    if ((threadIdx.x & 31) == 0)
        atomicMin(&sh.ubound, __float_as_int(u));
    __syncthreads();
    const float ub = __int_as_float(sh.ubound);
    const float lim = ub + 2.f * L.margin(ub);
    for (int k = threadIdx.x; k < L.m; k += blockDim.x) {
        const float3 q = L.cell(a, k);
        // NaN distances stay in: the comparisons of nearest_cell never pick them
        if (!(L.dist(q, xm, -w) > lim)) {
            const int i = atomicAdd(&sh.ncand, 1);
            if (i < VOR_CAND)
                sh.cand[i] = make_float4(q.x, q.y, q.z, __int_as_float(k));
        }
    }
    __syncthreads();
}

// Cell (index within the sightline's list) nearest to the point x.
__device__ int nearest_cell(const VorArgs &a, const VorLine &L, double x, const VorShared &sh)
{
    const float xf = (float)x;
    const bool held = sh.ncand <= VOR_CAND;
    const int n = held ? sh.ncand : L.m;
    const auto get = [&](int i, int &k) {
        if (!held) {
            k = i;
            return L.cell(a, i);
        }
        const float4 c = sh.cand[i];
        k = __float_as_int(c.w);
        return make_float3(c.x, c.y, c.z);
    };
    float best_f = 3.4e38f;
    int k1 = 0;
    for (int i = 0; i < n; i++) {
        int k;
        const float3 q = get(i, k);
        const float d = L.dist(q, xf, 0.f);
        if (d < best_f) {
            best_f = d;
            k1 = k;
        }
    }
    const float lim = best_f + L.margin(best_f);
    int within = 0;
    for (int i = 0; i < n; i++) {
        int k;
        within += L.dist(get(i, k), xf, 0.f) > lim ? 0 : 1;
    }
    if (within == 1 && best_f < 0.9f * L.boxf)
        return k1;
    // the reference's double distance on the cells within the float error
    double best = a.box;
    int best_k = -1, best_p = 0;
    for (int i = 0; i < n; i++) {
        int k;
        const float3 q = get(i, k);
        if (L.dist(q, xf, 0.f) > lim)
            continue;
        const double d = L.dist64(a, q, x);
        if (d <= best) {
            const int p = __ldg(&a.part[L.e0 + k]);
            if (d < best || (best_k >= 0 && p < best_p)) {
                best = d;
                best_k = k;
                best_p = p;
            }
        }
    }
    if (best_k < 0) {   // no cell nearer than the box: the first in particle order
        for (int k = 0; k < L.m; k++) {
            const int p = __ldg(&a.part[L.e0 + k]);
            if (best_k < 0 || p < best_p) {
                best_k = k;
                best_p = p;
            }
        }
    }
    return best_k;
}

__device__ __forceinline__ double point_x(const VorArgs &a, int i) { return (i + 0.5) * a.reso; }

// The block's points [i0, i0 + VOR_POINTS) of the sightline.
__device__ __forceinline__ void gather_block(const VorArgs &a, const VorLine &L, int i0,
                                             VorShared &sh)
{
    const double xa = point_x(a, i0), xb = point_x(a, min(i0 + VOR_POINTS, a.npoint) - 1);
    gather_candidates(a, L, (float)(0.5 * (xa + xb)), (float)(0.5 * (xb - xa)), sh);
}

__global__ void __launch_bounds__(VOR_THREADS) first_cell_kernel(VorArgs a, int line0, int *c0)
{
    __shared__ VorShared sh;
    const int l = line0 + blockIdx.y;
    if (a.off[l + 1] == a.off[l])
        return;
    const VorLine L(a, l);
    gather_candidates(a, L, (float)point_x(a, 0), 0.f, sh);
    if (threadIdx.x == 0)
        c0[l] = nearest_cell(a, L, point_x(a, 0), sh);
}

__global__ void __launch_bounds__(VOR_THREADS) wrap_point_kernel(VorArgs a, int line0,
                                                                 const int *c0, int *istar)
{
    __shared__ VorShared sh;
    const int l = line0 + blockIdx.y;
    if (a.off[l + 1] == a.off[l])
        return;
    const int i0 = blockIdx.x * VOR_POINTS;
    const double lo = a.box / 2. + 0.5 * a.reso;
    if (!(point_x(a, min(i0 + VOR_POINTS, a.npoint) - 1) > lo))
        return;
    const VorLine L(a, l);
    gather_block(a, L, i0, sh);
    for (int i = i0 + threadIdx.x; i < min(i0 + VOR_POINTS, a.npoint); i += VOR_THREADS) {
        const double x = point_x(a, i);
        if (x > lo && nearest_cell(a, L, x, sh) == c0[l])
            atomicMin(&istar[l], i);
    }
}

__global__ void __launch_bounds__(VOR_THREADS) cell_extent_kernel(VorArgs a, int line0,
                                                                  const int *istar, int *first,
                                                                  int *last, int *cnt)
{
    __shared__ VorShared sh;
    const int l = line0 + blockIdx.y;
    if (a.off[l + 1] == a.off[l])
        return;
    const int i0 = blockIdx.x * VOR_POINTS;
    const int i1 = min(i0 + VOR_POINTS, min(a.npoint, istar[l]));
    if (i0 >= i1)
        return;
    const VorLine L(a, l);
    gather_block(a, L, i0, sh);
    // whole-warp trips; the lanes of a warp that share a cell add to it together
    for (int b = i0 + (threadIdx.x & ~31); b < i1; b += VOR_THREADS) {
        const int i = b + (threadIdx.x & 31);
        const int k = i < i1 ? nearest_cell(a, L, point_x(a, i), sh) : -1;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k >= 0 && (threadIdx.x & 31) == __ffs(same) - 1) {
            atomicMin(&first[L.e0 + k], i);
            atomicMax(&last[L.e0 + k], b + 31 - __clz(same));
            atomicAdd(&cnt[L.e0 + k], __popc(same));
        }
    }
}

// The float segment of every cell (a block per sightline).
__global__ void cell_segment_kernel(VorArgs a, int line0, const int *c0, const int *istar,
                                    const int *first, const int *last, const int *cnt,
                                    float2 *seg, unsigned *dev_err)
{
    const int l = line0 + blockIdx.x;
    const long long e0 = a.off[l], e1 = a.off[l + 1];
    for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        float left, right;
        if (cnt[e] == 0) {
            left = right = (float)(3 * a.box);
        } else {
            if (cnt[e] != last[e] - first[e] + 1)
                atomicOr(dev_err, (unsigned)DEVERR_VORONOI_CELL);   // the reference exits here
            left = (float)point_x(a, first[e]);
            right = (float)point_x(a, last[e]);
        }
        if ((int)(e - e0) == c0[l] && istar[l] < a.npoint) {   // the first cell wraps round
            left = (float)point_x(a, istar[l]);
            right = (float)((double)right + a.box);
        }
        seg[e] = make_float2((float)((double)left - 0.5 * a.reso),
                             (float)((double)right + 0.5 * a.reso));
    }
}

__global__ void init_cells_kernel(int *first, int *last, int *cnt, long long npairs, int *c0,
                                  int *istar, int nlos, int npoint)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < npairs) {
        first[i] = 0x7fffffff;
        last[i] = -1;
        cnt[i] = 0;
    }
    if (i < nlos) {
        c0[i] = 0;
        istar[i] = npoint;
    }
}

unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

long long voronoi_scratch_ints(long long npairs, int nlos)
{
    return 3 * npairs + 2 * (long long)nlos;
}

void launch_voronoi_cells(const float *pos, const int *part, const long long *off,
                          const int *axis, const double *cofm, int nlos, long long npairs,
                          double box, int *scratch, float2 *seg, unsigned *dev_err,
                          cudaStream_t s)
{
    if (nlos <= 0 || npairs <= 0)
        return;
    VorArgs a;
    a.pos = pos;
    a.part = part;
    a.off = off;
    a.axis = axis;
    a.cofm = cofm;
    a.nlos = nlos;
    a.npoint = (int)(box / RESO);
    a.box = box;
    a.reso = box / a.npoint;
    int *first = scratch, *last = first + npairs, *cnt = last + npairs;
    int *c0 = cnt + npairs, *istar = c0 + nlos;
    init_cells_kernel<<<blocks_for(std::max(npairs, (long long)nlos), 256), 256, 0, s>>>(
        first, last, cnt, npairs, c0, istar, nlos, a.npoint);
    const unsigned px = blocks_for(a.npoint, VOR_POINTS);
    for (int l0 = 0; l0 < nlos; l0 += 65535) {
        const unsigned ny = (unsigned)std::min(65535, nlos - l0);
        first_cell_kernel<<<dim3(1, ny), VOR_THREADS, 0, s>>>(a, l0, c0);
        wrap_point_kernel<<<dim3(px, ny), VOR_THREADS, 0, s>>>(a, l0, c0, istar);
        cell_extent_kernel<<<dim3(px, ny), VOR_THREADS, 0, s>>>(a, l0, istar, first, last, cnt);
        cell_segment_kernel<<<ny, VOR_THREADS, 0, s>>>(a, l0, c0, istar, first, last, cnt, seg,
                                                       dev_err);
    }
}

}  // namespace fsg
