// Sightlines shared between blocks: the per-launch state and the hand-over of a
// sightline from its owner to the blocks that help, and back.
//
// The owner stores the bound of the sightline's total and then publishes the
// sightline (share_open); a helper that has seen it published (share_ready) reads
// that bound, which fixes the unit of its integer sums.  Every block adds its
// sums to the sightline's words and then counts its chunks as done (share_done);
// the block whose chunks complete the sightline reads the words.  Both steps are a
// release on the one side and an acquire on the other, at the scope of the GPU: a
// plain load of the flag leaves the load of the bound free to come first.  One
// thread takes each step for its block, between block barriers that order the
// other threads' accesses with it.
#pragma once

#include <stddef.h>

#ifdef __CUDACC__
#define FSG_HD __host__ __device__ __forceinline__
#else
#define FSG_HD inline
#endif

namespace fsg {

// Zeroed before the launch.
struct SplitState {
    unsigned *next, *done;   // [nlos] chunks taken, chunks whose sums are in acc
    unsigned *ready;         // [nlos] B is set and chunks may be taken
    unsigned *active;        // [nlos] blocks that have joined (a hint)
    unsigned *bad;           // [nlos] a contribution was not finite
    unsigned *started;       // sightlines that are ready or need no chunks
    double *B;               // [nlos] bound of the sightline total
    unsigned long long *acc;     // [nlos][2 (nbins + nodes)]
    size_t words;            // 2 (nbins + nodes)
};

inline size_t split_bytes(int nlos, int nbins, int nodes)
{
    return 64 + (size_t)nlos * (5 * sizeof(unsigned) + sizeof(double) + 4 +
                                sizeof(unsigned long long) * 2 * ((size_t)nbins + nodes));
}

FSG_HD SplitState split_state(void *ws, int nlos, int nbins, int nodes)
{
    SplitState st;
    st.words = 2 * ((size_t)nbins + nodes);
    unsigned char *p = (unsigned char *)ws;
    st.acc = (unsigned long long *)p;
    p += sizeof(unsigned long long) * st.words * nlos;
    st.B = (double *)p;
    p += sizeof(double) * nlos;
    unsigned *u = (unsigned *)p;
    st.next = u;
    st.done = u + nlos;
    st.ready = u + 2 * (size_t)nlos;
    st.active = u + 3 * (size_t)nlos;
    st.bad = u + 4 * (size_t)nlos;
    st.started = u + 5 * (size_t)nlos;
    return st;
}

// The value of a word that another block may be writing; share_acquire: and what
// that block wrote before it.
FSG_HD unsigned share_load(const unsigned *p)
{
#ifdef __CUDA_ARCH__
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
#else
    return __atomic_load_n(p, __ATOMIC_RELAXED);
#endif
}

FSG_HD unsigned share_acquire(const unsigned *p)
{
#ifdef __CUDA_ARCH__
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
#else
    return __atomic_load_n(p, __ATOMIC_ACQUIRE);
#endif
}

// *p += n, after everything this block wrote before; the old value, and what the
// blocks that added before wrote.
FSG_HD unsigned share_add(unsigned *p, unsigned n)
{
#ifdef __CUDA_ARCH__
    unsigned v;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;"
                 : "=r"(v) : "l"(p), "r"(n) : "memory");
    return v;
#else
    return __atomic_fetch_add(p, n, __ATOMIC_ACQ_REL);
#endif
}

// The owner of sightline q publishes its bound (one thread).
FSG_HD void share_open(const SplitState &sp, int q, double B, bool live)
{
    sp.B[q] = B;
    if (live)
        share_add(&sp.ready[q], 1u);
    share_add(sp.started, 1u);
}

// Whether sightline q may be helped; then its bound may be read.
FSG_HD bool share_ready(const SplitState &sp, int q) { return share_acquire(&sp.ready[q]) != 0u; }

// Whether every sightline has been opened: the flags of those that need help are set.
FSG_HD bool share_all_open(const SplitState &sp, int nlos)
{
    return share_acquire(sp.started) >= (unsigned)nlos;
}

// Counts `mine` chunks of sightline q as done (one thread, after the block's sums
// are in its words); true for the block that completes it.
FSG_HD bool share_done(const SplitState &sp, int q, unsigned mine, unsigned nchunks)
{
    return share_add(&sp.done[q], mine) + mine == nchunks;
}

}  // namespace fsg
