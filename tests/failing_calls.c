/* Stands in front of the CUDA runtime of a test's child process: the n-th kernel launch, or the n-th device allocation, after
 * fail_launch(n) or fail_allocation(n) is not made and reports an error, as one that the runtime refuses does. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>

typedef struct { unsigned x, y, z; } dim3_t;
static int launches, allocations, launch_to_fail = -1, allocation_to_fail = -1, pending;

static void *next(const char *name) {
    void *runtime = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    return dlsym(runtime, name);
}
void fail_launch(int n) { launches = 0; launch_to_fail = n; }
void fail_allocation(int n) { allocations = 0; allocation_to_fail = n; }
int launches_made(void) { return launches; }
int allocations_made(void) { return allocations; }

int cudaLaunchKernel(const void *f, dim3_t grid, dim3_t block, void **args, size_t shared, void *stream) {
    if (launches++ == launch_to_fail) return pending = 701;      /* cudaErrorLaunchOutOfResources */
    return ((int (*)(const void *, dim3_t, dim3_t, void **, size_t, void *))next("cudaLaunchKernel"))(f, grid, block, args, shared, stream);
}
int cudaMalloc(void **p, size_t bytes) {
    if (allocations++ == allocation_to_fail) return pending = 2;      /* cudaErrorMemoryAllocation */
    return ((int (*)(void **, size_t))next("cudaMalloc"))(p, bytes);
}
int cudaGetLastError(void) {
    const int e = pending;
    pending = 0;
    return e ? e : ((int (*)(void))next("cudaGetLastError"))();
}
int cudaPeekAtLastError(void) { return pending ? pending : ((int (*)(void))next("cudaPeekAtLastError"))(); }
