/* Stands between the library and the CUDA runtime (LD_PRELOAD), for tests of
 * what the host code does when a call fails, and of what it asks for.
 *   CGB_SHIM_FAIL_BYTES=n  the first cudaMalloc of exactly n bytes fails
 *   CGB_SHIM_ATTR_LOG=path the number of every device attribute asked for is
 *                          appended to this file, one per line */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>

static void* runtime_symbol(const char* name) {
    void* lib = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    return lib ? dlsym(lib, name) : NULL;
}

int cudaMalloc(void** p, size_t bytes) {
    static int (*real)(void**, size_t);
    static int failed;
    const char* e = getenv("CGB_SHIM_FAIL_BYTES");
    if (!real) real = (int (*)(void**, size_t))runtime_symbol("cudaMalloc");
    if (!failed && e && bytes == strtoull(e, NULL, 10)) {
        failed = 1;
        return 2; /* cudaErrorMemoryAllocation */
    }
    return real(p, bytes);
}

int cudaDeviceGetAttribute(int* value, int attr, int device) {
    static int (*real)(int*, int, int);
    const char* path = getenv("CGB_SHIM_ATTR_LOG");
    if (!real) real = (int (*)(int*, int, int))runtime_symbol("cudaDeviceGetAttribute");
    if (path) {
        FILE* f = fopen(path, "a");
        if (f) {
            fprintf(f, "%d\n", attr);
            fclose(f);
        }
    }
    return real(value, attr, device);
}
