/* cudaMalloc that refuses allocations once a budget of calls is used up.  Loaded
 * before libcudart, it stands in front of the runtime's; negative: no limit. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static long left = -1;

void cuda_budget(long calls) { left = calls; }

int cudaMalloc(void **p, size_t n)
{
    static int (*real)(void **, size_t);
    if (left == 0) {
        *p = NULL;
        return 2;   /* cudaErrorMemoryAllocation */
    }
    if (!real)
        real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), "cudaMalloc");
    if (left > 0)
        --left;
    return real(p, n);
}
