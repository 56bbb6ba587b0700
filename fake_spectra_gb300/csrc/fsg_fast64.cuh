// Kernel skeleton of the FP64 deposits (included by fsg_deposit.cu inside its
// anonymous namespace): sightlines from a queue, 128-bit accumulators in
// shared memory (or global memory for very long rows), chunks of pairs dealt to
// the warps, and optionally a thread-block cluster per sightline, whose blocks
// sum their accumulators through distributed shared memory.

__device__ __forceinline__ unsigned cluster_size()
{
    unsigned n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Barrier of every thread of the cluster (release / acquire).
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this block's shared object in the block of rank r.
template <class T>
__device__ __forceinline__ T *cluster_map(T *p, unsigned r)
{
    unsigned long long out;
    asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"((unsigned long long)p), "r"(r));
    return reinterpret_cast<T *>(out);
}

// Sum over the cluster's blocks of a 128-bit accumulator word, as a double.
__device__ __forceinline__ double cluster_fixed(unsigned long long *lo, unsigned long long *hi,
                                                unsigned nc, int S)
{
    unsigned long long l = lo[0], h = hi[0];
    if (nc > 1) {
        l = 0ull;
        h = 0ull;
        for (unsigned r = 0; r < nc; r++) {
            const unsigned long long x = *cluster_map(lo, r);
            h += *cluster_map(hi, r);
            l += x;
            h += l < x ? 1ull : 0ull;
        }
    }
    return from_fixed(l, h, S);
}

// Clenshaw sum of the M Chebyshev coefficients c at t in [-1, 1].
__device__ __forceinline__ double clenshaw64(const double *c, double t)
{
    double b1 = 0.0, b2 = 0.0;
    const double t2 = 2.0 * t;
#pragma unroll
    for (int k = T64_M - 1; k >= 1; k--) {
        const double b = fma(t2, b1, c[k] - b2);
        b2 = b1;
        b1 = b;
    }
    return fma(t, b1, c[0] - b2);
}

// Node values of `ntiles` tiles to Chebyshev coefficients, in place (half a
// warp per tile, whole block).
__device__ __forceinline__ void nodes_to_coefs64(double *node, int ntiles)
{
    static_assert(T64_M == 16, "half a warp per tile; s_cos64 has 64 entries");
    const int k = threadIdx.x & 15;
    const int per = blockDim.x / 16;
    for (int t0 = 0; t0 < ntiles; t0 += per) {
        const int t = t0 + threadIdx.x / 16;
        double *f = node + (size_t)t * T64_M;
        double s = 0.0;
        if (t < ntiles) {
#pragma unroll
            for (int m = 0; m < T64_M; m++)
                s = fma(f[m], s_cos64[(k * (2 * m + 1)) & 63], s);
            s *= k == 0 ? 1.0 / T64_M : 2.0 / T64_M;
        }
        __syncwarp();
        if (t < ntiles)
            f[k] = s;
        __syncwarp();
    }
}

template <bool TAU>
__global__ void __launch_bounds__(TAU ? T64_THREADS : C64_THREADS, 1) fast64_kernel(DepositArgs a)
{
    using Stage = typename std::conditional<TAU, Stage64, StageC64>::type;
    extern __shared__ __align__(16) unsigned long long smem[];
    __shared__ BoundScratch red;
    __shared__ int s_bad;
    __shared__ unsigned s_ticket, s_chunk;
    const int nbins = a.lp.nbins;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nc = cluster_size(), rank = cluster_rank();
    const double bintov = a.lp.vbox / nbins;
    const double btk = a.lp.vbox / nbins / a.lp.velfac;
    const Tiles64 tl = tiles64_layout(a.tiles, nbins);
    // dynamic shared memory: [accumulators lo, hi (smem_mode)] [tile nodes lo, hi] [stage]
    // [K table]
    unsigned long long *tlo = smem + (a.smem_mode ? 2 * (size_t)nbins : 0);
    unsigned long long *thi = tlo + tl.nodes;
    Stage *stage = reinterpret_cast<Stage *>(smem + (a.smem_mode ? 2 * (size_t)nbins : 0) +
                                             2 * (size_t)tl.nodes) + warp * a.chunk;
    for (int j = threadIdx.x; TAU && j < 64; j += blockDim.x) {
        s_cos64[j] = cospi((double)j / 32.0);
        s_pow2[j] = d_fix_pow2[j];
    }
    Rows64 rows{d_fix_rows, 0};
    if (TAU && a.table_off) {
        int4 *dst = reinterpret_cast<int4 *>(reinterpret_cast<char *>(smem) + a.table_off);
        const int4 *src = reinterpret_cast<const int4 *>(d_fix_rows);
        for (int j = threadIdx.x; j < 4 * FSG_FIX_ROWS; j += blockDim.x)
            dst[j ^ ((j >> 3) & 3)] = src[j];
        rows = Rows64{reinterpret_cast<const FixRow *>(dst), 3};
    }
    const unsigned first = blockIdx.x / nc;
    unsigned ticket = first;
    for (;;) {
        if (a.persistent) {
            // the cluster's first block draws the next sightline
            if (rank == 0 && threadIdx.x == 0) {
                const unsigned t = atomicAdd(a.ticket, 1u);
                for (unsigned r = 0; r < nc; r++)
                    *cluster_map(&s_ticket, r) = t;
            }
            cluster_sync();
            ticket = s_ticket;
        }
        if (ticket >= (unsigned)a.nlos)
            break;
        const int line = a.line_order[ticket];
        const int axis = a.t.axis[line];
        const long long e0 = a.pl.off[line], e1 = a.pl.off[line + 1];
        const auto bound = [&](long long e) {
            const PairInput in = load_pair(a.p, a.pl, e, axis, TAU, a.dev_err);
            return TAU ? tau_pair_bound(a.lp, in) : colden_pair_bound(a.lp, in, btk);
        };
        const double B = order_free_bound(e0, e1, bound, bound, &red);
        unsigned long long *lo, *hi;
        if (a.smem_mode) {
            lo = smem;
            hi = smem + nbins;
        } else {
            lo = a.gacc + (size_t)line * 2 * nbins;
            hi = lo + nbins;
        }
        for (int j = threadIdx.x; j < nbins; j += blockDim.x) {
            lo[j] = 0ull;
            hi[j] = 0ull;
        }
        for (int j = threadIdx.x; j < tl.nodes; j += blockDim.x) {
            tlo[j] = 0ull;
            thi[j] = 0ull;
        }
        if (threadIdx.x == 0) {
            s_chunk = 0u;
            s_bad = !isfinite(B);
        }
        cluster_sync();
        const bool live = isfinite(B) && B > 0.0;
        const int S = live ? 124 - ilogb(B) : 0;
        if (live) {
            unsigned *counter = cluster_map(&s_chunk, 0);
            for (;;) {
                unsigned c = 0;
                if (lane == 0)
                    c = atomicAdd(counter, 1u);
                c = __shfl_sync(0xffffffffu, c, 0);
                const long long cb = e0 + (long long)c * a.chunk;
                if (cb >= e1)
                    break;
                const int n = (int)min((long long)a.chunk, e1 - cb);
                if constexpr (TAU)
                    deposit_tau64(a, tl, rows, axis, cb, n, S, lo, hi, tlo, thi, &s_bad, stage,
                                  bintov, lane);
                else
                    deposit_colden64(a, axis, cb, n, S, lo, hi, &s_bad, stage, btk, lane);
            }
        }
        cluster_sync();
        bool bad = s_bad != 0;
        for (unsigned r = 0; r < nc && !bad; r++)
            bad = *cluster_map(&s_bad, r) != 0;
        if (bad) {
            if (rank == 0 && threadIdx.x == 0)
                a.bad_lines[atomicAdd(a.n_bad, 1)] = line;
        } else if (live) {
            double *row = a.out + (size_t)line * nbins;
            double *node = reinterpret_cast<double *>(tlo);
            if (tl.nodes > 0) {
                // node sums as doubles: each block forms its share for all blocks
                for (int j = rank * blockDim.x + threadIdx.x; j < tl.nodes;
                     j += nc * blockDim.x) {
                    const double v = cluster_fixed(tlo + j, thi + j, nc, S);
                    if (nc == 1)
                        node[j] = v;
                    else
                        for (unsigned r = 0; r < nc; r++)
                            *cluster_map(node + j, r) = v;
                }
                cluster_sync();
                // from the widest tiles down: coefficients, added at the nodes
                // of the four tiles below
                for (int l = T64_LEVELS - 1; l >= 0; l--) {
                    const int nt = nbins / (tl.w0 << (2 * l));
                    double *nd = node + tl.first[l];
                    nodes_to_coefs64(nd, nt);
                    __syncthreads();
                    if (l > 0) {
                        double *down = node + tl.first[l - 1];
                        for (int j = threadIdx.x; j < nt * 4 * T64_M; j += blockDim.x) {
                            const int child = j / T64_M, m = j % T64_M;
                            const double t = fma(0.25, s_cos64[2 * m + 1],
                                                 0.5 * (double)(child & 3) - 0.75);
                            down[j] += clenshaw64(nd + (size_t)(child >> 2) * T64_M, t);
                        }
                        __syncthreads();
                    }
                }
            }
            const int covered = tl.w0 > 0 ? nbins / tl.w0 * tl.w0 : 0;
            const double inv_w = tl.w0 > 0 ? 2.0 / tl.w0 : 0.0;
            for (int j = rank * blockDim.x + threadIdx.x; j < nbins; j += nc * blockDim.x) {
                double v = cluster_fixed(lo + j, hi + j, nc, S);
                if (j < covered)
                    v += clenshaw64(node + (size_t)(j / tl.w0) * T64_M,
                                    fma((double)(j & (tl.w0 - 1)) + 0.5, inv_w, -1.0));
                row[j] = v;
            }
        }
        // no block clears or leaves its accumulators while another reads them
        cluster_sync();
        if (!a.persistent)
            break;
    }
}
