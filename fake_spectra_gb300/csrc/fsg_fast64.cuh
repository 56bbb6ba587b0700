// Kernel skeleton of the FP64 deposits (included by fsg_deposit.cu inside its
// anonymous namespace): sightlines from a queue, 128-bit accumulators in
// shared memory (or global memory for very long rows), chunks of pairs dealt to
// the warps.
//
// Pair costs differ by orders of magnitude and sightlines are often few, so a
// block that finds the queue empty helps: it takes chunks from the sightline
// with the most left, adds them in its own accumulators and then adds those
// into the sightline's words in global memory.  The block whose chunks complete
// the sightline writes the row.  Sums are integers, so the bits do not depend
// on who did what.  (Without help 72 sightlines through a clumpy 128^3 snapshot
// left the SMs idle for 69% of the kernel, and 37% with a cluster of four
// blocks per sightline.)

// The sightline with the most chunks left per block working on it, or -1 (whole
// block).  Waits a while for sightlines whose bound is still being formed: at
// most SPLIT_POLLS polls, after which the block leaves (the owners need no help).
constexpr int SPLIT_POLLS = 4096;
__device__ int pick_line(const DepositArgs &a, const SplitState &sp, unsigned min_left,
                         unsigned long long *s_best)
{
    for (int poll = 0; poll < SPLIT_POLLS; poll++) {
        const bool all = share_all_open(sp, a.nlos);
        __syncthreads();
        if (threadIdx.x == 0)
            *s_best = 0ull;
        __syncthreads();
        for (int i = threadIdx.x; i < a.nlos; i += blockDim.x) {
            const int l = a.line_order[i];
            if (!share_ready(sp, i))
                continue;
            const long long n = (a.pl.off[l + 1] - a.pl.off[l] + a.chunk - 1) / a.chunk;
            const long long left = n - (long long)share_load(&sp.next[i]);
            if (left < (long long)min_left)
                continue;
            const long long blocks = 1 + (long long)share_load(&sp.active[i]);
            const unsigned score = (unsigned)min(left * 16 / blocks, 0x7fffffffll);
            atomicMax(s_best, ((unsigned long long)score << 32) | (unsigned)(i + 1));
        }
        __syncthreads();
        const unsigned long long b = *s_best;
        if (b) {
            const int i = (int)(unsigned)b - 1;
            if (threadIdx.x == 0)
                atomicAdd(&sp.active[i], 1u);
            return i;
        }
        if (__syncthreads_and(all))
            return -1;
        __nanosleep(500);
    }
    return -1;
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
    __shared__ unsigned long long s_best;
    __shared__ int s_bad;
    __shared__ unsigned s_ticket, s_chunk, s_mine, s_last;
    const int nbins = a.lp.nbins;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double bintov = a.lp.vbox / nbins;
    const double btk = a.lp.vbox / nbins / a.lp.velfac;
    const Tiles64 tl = tiles64_layout(a.tiles, nbins);
    const bool split = a.split_ws != nullptr;
    const SplitState sp = split_state(a.split_ws, a.nlos, nbins, tl.nodes);
    // dynamic shared memory: [accumulators lo, hi (smem_mode)] [tile nodes lo, hi] [stage]
    // [K table]
    unsigned long long *tlo = smem + (a.smem_mode ? 2 * (size_t)nbins : 0);
    unsigned long long *thi = tlo + tl.nodes;
    Stage *stage = reinterpret_cast<Stage *>(smem + (a.smem_mode ? 2 * (size_t)nbins : 0) +
                                             2 * (size_t)tl.nodes) + warp * a.chunk;
    for (int j = threadIdx.x; TAU && j < 64; j += blockDim.x) {
        s_cos64[j] = cospi((double)j / 32.0);
        if (j < T64_M)
            s_node64[j] = 0.5 + 0.5 * cospi((double)(2 * j + 1) / 32.0);
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
    for (bool first = true;; first = false) {
        // the next sightline (its place in the queue): an own one, else one to help with
        __syncthreads();
        if (threadIdx.x == 0)
            s_ticket = a.persistent ? atomicAdd(a.ticket, 1u) : (first ? blockIdx.x : 0xFFFFFFFFu);
        __syncthreads();
        int q = (int)min(s_ticket, 0x7fffffffu);
        const bool owner = q < a.nlos;
        if (!owner) {
            if (!split)
                break;
            q = pick_line(a, sp, (unsigned)(blockDim.x >> 5), &s_best);
            if (q < 0)
                break;
        }
        const int line = a.line_order[q];
        const int axis = a.t.axis[line];
        const long long e0 = a.pl.off[line], e1 = a.pl.off[line + 1];
        const unsigned nchunks = (unsigned)((e1 - e0 + a.chunk - 1) / a.chunk);
        double B;
        if (owner) {
            const auto bound = [&](long long e) {
                const PairInput in = load_pair(a.p, a.pl, e, axis, TAU, a.dev_err);
                return TAU ? tau_pair_bound(a.lp, in) : colden_pair_bound(a.lp, in, btk);
            };
            B = order_free_bound(e0, e1, bound, bound, &red);
        } else {
            B = __ldcg(&sp.B[q]);
        }
        const bool live = isfinite(B) && B > 0.0;
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
            s_mine = 0u;
            s_bad = !isfinite(B);
            if (owner && split)
                share_open(sp, q, B, live);
        }
        __syncthreads();
        const int S = live ? 124 - ilogb(B) : 0;
        if (live) {
            unsigned *counter = split ? &sp.next[q] : &s_chunk;
            unsigned mine = 0;
            for (;;) {
                unsigned c = 0;
                if (lane == 0)
                    c = atomicAdd(counter, 1u);
                c = __shfl_sync(0xffffffffu, c, 0);
                if (c >= nchunks)
                    break;
                mine++;
                const long long cb = e0 + (long long)c * a.chunk;
                const int n = (int)min((long long)a.chunk, e1 - cb);
                if constexpr (TAU)
                    deposit_tau64(a, tl, rows, axis, cb, n, S, lo, hi, tlo, thi, &s_bad, stage,
                                  bintov, lane);
                else
                    deposit_colden64(a, axis, cb, n, S, lo, hi, &s_bad, stage, btk, lane);
            }
            if (lane == 0 && mine)
                atomicAdd(&s_mine, mine);
        }
        __syncthreads();
        bool bad = s_bad != 0;
        if (live && split && s_mine != nchunks) {
            // a shared sightline: this block's sums go to its words in global
            // memory, and the block that completes it takes them back
            const unsigned mine = s_mine;
            if (mine == 0u)
                continue;
            unsigned long long *g = sp.acc + (size_t)q * sp.words;
            const auto merge = [&](unsigned long long *l, unsigned long long *h, size_t at, int n) {
                for (int j = threadIdx.x; j < n; j += blockDim.x)
                    if (l[j] | h[j])
                        fixed_add(g + at, g + at + n, j, l[j], h[j]);
            };
            merge(lo, hi, 0, nbins);
            merge(tlo, thi, 2 * (size_t)nbins, tl.nodes);
            if (threadIdx.x == 0 && bad)
                atomicOr(&sp.bad[q], 1u);
            __syncthreads();
            if (threadIdx.x == 0)
                s_last = share_done(sp, q, mine, nchunks);
            __syncthreads();
            if (!s_last)
                continue;
            for (int j = threadIdx.x; j < nbins; j += blockDim.x) {
                lo[j] = __ldcg(g + j);
                hi[j] = __ldcg(g + nbins + j);
            }
            for (int j = threadIdx.x; j < tl.nodes; j += blockDim.x) {
                tlo[j] = __ldcg(g + 2 * (size_t)nbins + j);
                thi[j] = __ldcg(g + 2 * (size_t)nbins + tl.nodes + j);
            }
            bad = __ldcg(&sp.bad[q]) != 0u;
            __syncthreads();
        }
        if (bad) {
            if (threadIdx.x == 0)
                a.bad_lines[atomicAdd(a.n_bad, 1)] = line;
        } else if (live) {
            double *row = a.out + (size_t)line * nbins;
            double *node = reinterpret_cast<double *>(tlo);
            if (tl.nodes > 0) {
                for (int j = threadIdx.x; j < tl.nodes; j += blockDim.x)
                    node[j] = from_fixed(tlo[j], thi[j], S);
                __syncthreads();
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
            for (int j = threadIdx.x; j < nbins; j += blockDim.x) {
                double v = from_fixed(lo[j], hi[j], S);
                if (j < covered)
                    v += clenshaw64(node + (size_t)(j / tl.w0) * T64_M,
                                    fma((double)(j & (tl.w0 - 1)) + 0.5, inv_w, -1.0));
                row[j] = v;
            }
        }
        if (!a.persistent)
            break;
    }
}
