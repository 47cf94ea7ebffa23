/* Stands between the library and the CUDA runtime (LD_PRELOAD), for tests of
 * what the host code does when a call fails, and of what it asks for.
 *   CGB_SHIM_FAIL_BYTES=n  the first cudaMalloc of exactly n bytes fails
 *   CGB_SHIM_REUSE=1       a block below 16 MiB that is freed is handed out
 *                          again, to the next request of up to 16 times its size
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

enum { kBlocks = 4096, kSpare = 16 };
static struct { void* p; size_t room; int freed; } blocks[kBlocks];
static int n_blocks;

int cudaMalloc(void** p, size_t bytes) {
    static int (*real)(void**, size_t);
    static int failed;
    const char* e = getenv("CGB_SHIM_FAIL_BYTES");
    if (!real) real = (int (*)(void**, size_t))runtime_symbol("cudaMalloc");
    if (!failed && e && bytes == strtoull(e, NULL, 10)) {
        failed = 1;
        return 2; /* cudaErrorMemoryAllocation */
    }
    if (!getenv("CGB_SHIM_REUSE") || bytes >= 16u << 20) return real(p, bytes);
    int last = -1;
    for (int i = 0; i < n_blocks; ++i)
        if (blocks[i].room >= bytes && blocks[i].freed && (last < 0 || blocks[i].freed > blocks[last].freed)) last = i;
    if (last < 0) {
        if (n_blocks == kBlocks) return real(p, bytes);
        int rc = real(&blocks[n_blocks].p, bytes * kSpare);
        if (rc) return rc;
        blocks[n_blocks].room = bytes * kSpare;
        last = n_blocks++;
    }
    blocks[last].freed = 0;
    *p = blocks[last].p;
    return 0;
}

int cudaFree(void* p) {
    static int (*real)(void*);
    static int clock;
    if (!real) real = (int (*)(void*))runtime_symbol("cudaFree");
    for (int i = 0; p && i < n_blocks; ++i)
        if (blocks[i].p == p) {
            blocks[i].freed = ++clock;
            return 0;
        }
    return real(p);
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
