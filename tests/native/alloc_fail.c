/* alloc_fail.c -- preloaded: the next n calls of cudaMalloc fail (cudaErrorMemoryAllocation) without reaching the
 * runtime */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

static int left;
void alloc_fail_next(int n) { left = n; }

int cudaMalloc(void **p, size_t n) {
    static int (*real)(void **, size_t);
    if (left > 0) {
        left--;
        return 2;
    }
    if (!real) {  /* (the runtime comes in with the engine's library, out of RTLD_NEXT's sight) */
        void *rt = dlopen("libcudart.so.13", RTLD_NOW | RTLD_NOLOAD);
        if (rt) real = (int (*)(void **, size_t))dlsym(rt, "cudaMalloc");
    }
    return real ? real(p, n) : 999;
}
