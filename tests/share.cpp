/* Test helper (compiled by tests/test_share.py, with the thread sanitizer): the
 * hand-over of shared sightlines (fsg_share.cuh) with a host thread for every
 * block.  Arguments: threads, sightlines, chunks per sightline.  Prints the
 * total of every sightline, as the block that completes it reads it. */
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "fsg_share.cuh"

using namespace fsg;

static unsigned add(unsigned *p) { return __atomic_fetch_add(p, 1u, __ATOMIC_RELAXED); }

int main(int argc, char **argv)
{
    const int nthreads = atoi(argv[1]), nlos = atoi(argv[2]);
    const unsigned nchunks = (unsigned)atoi(argv[3]);
    std::vector<unsigned long long> ws(split_bytes(nlos, 2, 1) / 8 + 1, 0ull);
    const SplitState sp = split_state(ws.data(), nlos, 2, 1);
    std::vector<double> total(nlos, -1.0);
    unsigned ticket = 0;
    int here = 0;
    auto block = [&]() {
        // all at once, and slow enough that every thread finds something to help with
        __atomic_fetch_add(&here, 1, __ATOMIC_RELAXED);
        while (__atomic_load_n(&here, __ATOMIC_RELAXED) < nthreads)
            std::this_thread::yield();
        for (;;) {
            int q = (int)add(&ticket);
            const bool owner = q < nlos;
            if (!owner) {
                q = -1;
                for (bool all = false; q < 0 && !all;) {
                    all = share_all_open(sp, nlos);
                    for (int i = 0; i < nlos && q < 0; i++)
                        if (share_ready(sp, i) && share_load(&sp.next[i]) < nchunks)
                            q = i;
                }
                if (q < 0)
                    return;
            }
            double B = 3.0 + q;
            if (owner)
                share_open(sp, q, B, true);
            else
                B = sp.B[q];
            unsigned mine = 0;
            unsigned long long sum = 0;
            for (; add(&sp.next[q]) < nchunks; mine++) {
                sum += (unsigned long long)B;
                std::this_thread::yield();
            }
            if (mine == 0)
                continue;
            __atomic_fetch_add(sp.acc + (size_t)q * sp.words, sum, __ATOMIC_RELAXED);
            if (mine > 1)
                __atomic_fetch_or(&sp.bad[q], 2u, __ATOMIC_RELAXED);
            if (share_done(sp, q, mine, nchunks))
                total[q] = (double)sp.acc[(size_t)q * sp.words] + 0.25 * (sp.bad[q] & 1u);
        }
    };
    std::vector<std::thread> pool;
    for (int i = 0; i < nthreads; i++)
        pool.emplace_back(block);
    for (auto &t : pool)
        t.join();
    for (double t : total)
        printf("%.17g\n", t);
    return 0;
}
