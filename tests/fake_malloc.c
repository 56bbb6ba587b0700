/* Test helper (preloaded by tests/test_gpu_split_memory.py): a cudaMalloc that answers
 * "out of memory" (2) for requests above a limit, or for the next few requests. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdint.h>

static size_t limit = SIZE_MAX;
static int next_fail, failed;

void fake_malloc_limit(size_t n) { limit = n; }
void fake_malloc_fail_next(int n) { next_fail = n; }
int fake_malloc_failed(void) { return failed; }

int cudaMalloc(void **p, size_t n)
{
    static int (*real)(void **, size_t);
    if (n > limit || next_fail > 0) {
        next_fail -= next_fail > 0;
        failed++;
        return 2;
    }
    if (!real) {
        void *rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
        real = rt ? (int (*)(void **, size_t))dlsym(rt, "cudaMalloc") : 0;
        if (!real)
            return 999;
    }
    return real(p, n);
}
