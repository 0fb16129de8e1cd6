/* Preloaded before the CUDA runtime: the n-th cudaMalloc from now on answers "out of memory" without
 * reaching the driver.  failing_malloc_arm(0) turns it off. */
#include <dlfcn.h>
#include <stddef.h>

static int left = 0;

void failing_malloc_arm(int n) { left = n; }

int cudaMalloc(void** p, size_t bytes)
{
    static int (*real)(void**, size_t) = NULL;
    if (left > 0 && --left == 0) return 2;      /* cudaErrorMemoryAllocation */
    if (!real)                                  /* the runtime that the library has loaded, not in the global scope */
    {
        void* runtime = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
        if (runtime) real = (int (*)(void**, size_t))dlsym(runtime, "cudaMalloc");
    }
    return real ? real(p, bytes) : 999;         /* cudaErrorUnknown */
}
