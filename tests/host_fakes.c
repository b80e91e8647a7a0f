/* A CUDA runtime on host memory for tests of the C host layer: device memory is
 * malloc'd, streams run at once, and page-locked ranges are a table that a test
 * can extend (fake_register).  A copy whose host side is partly registered is
 * refused, as the runtime's documentation has it.  A test's unit includes the C
 * file that it looks at and this one; tests/host_build.py adds stubs that return 0
 * for whatever is still missing. */
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

enum { FAKE_RANGES = 64 };
static struct FakeRange {
    uintptr_t first, end;
} fake_ranges[FAKE_RANGES]; /* page-locked host memory */
int fake_host_alloc_fails;  /* page-locking answers cudaErrorMemoryAllocation */
int fake_last_error;        /* what cudaGetLastError will return and clear */

__attribute__((visibility("default"))) void fake_register(const void* at, size_t bytes) {
    for (int k = 0; k < FAKE_RANGES; ++k)
        if (fake_ranges[k].end == 0) {
            fake_ranges[k].first = (uintptr_t)at;
            fake_ranges[k].end = (uintptr_t)at + bytes;
            return;
        }
    abort();
}

__attribute__((visibility("default"))) void fake_unregister(const void* at) {
    for (int k = 0; k < FAKE_RANGES; ++k)
        if (fake_ranges[k].end != 0 && fake_ranges[k].first == (uintptr_t)at)
            memset(&fake_ranges[k], 0, sizeof(fake_ranges[k]));
}

static int fake_locked(uintptr_t at) {
    for (int k = 0; k < FAKE_RANGES; ++k)
        if (at >= fake_ranges[k].first && at < fake_ranges[k].end) return 1;
    return 0;
}

/* Page-locked bytes among [at, at + bytes), in steps of 8 and at the last one. */
static int fake_mixed(const void* at, size_t bytes) {
    const int first = fake_locked((uintptr_t)at);
    for (size_t k = 0; k < bytes; k += 8)
        if (fake_locked((uintptr_t)at + k) != first) return 1;
    return bytes > 0 && fake_locked((uintptr_t)at + bytes - 1) != first;
}

/* Whether a kernel could reach [at, at + bytes) as doubles: mapped 4 KiB pages. */
static int fake_reachable(const void* at, size_t bytes) {
    if ((uintptr_t)at % sizeof(double) != 0) return 0;
    for (uintptr_t page = (uintptr_t)at & ~(uintptr_t)4095; page < (uintptr_t)at + bytes;
         page += 4096) {
        int any = 0;
        for (uintptr_t p = page; p < page + 4096; p += 8) any |= fake_locked(p);
        if (!any) return 0;
    }
    return 1;
}

static cudaError_t fake_fail(cudaError_t code) {
    fake_last_error = (int)code;
    return code;
}

cudaError_t cudaGetLastError(void) {
    const cudaError_t code = (cudaError_t)fake_last_error;
    fake_last_error = 0;
    return code;
}
const char* cudaGetErrorString(cudaError_t code) { return code == cudaSuccess ? "none" : "fake error"; }

cudaError_t cudaGetDeviceCount(int* count) {
    *count = 1;
    return cudaSuccess;
}
#undef cudaGetDeviceProperties
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int device) {
    memset(p, 0, sizeof(*p));
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp* p, int device) {
    return cudaGetDeviceProperties(p, device);
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
    *p = calloc(1, bytes + 1);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned flags) {
    if (fake_host_alloc_fails) return fake_fail(cudaErrorMemoryAllocation);
    if (posix_memalign(p, 4096, bytes) != 0) abort();
    fake_register(*p, bytes);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) {
    *p = calloc(1, bytes + 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    fake_unregister(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** device, void* host, unsigned flags) {
    *device = host;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* at, const void* p) {
    memset(at, 0, sizeof(*at));
    at->type = fake_locked((uintptr_t)p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    at->hostPointer = (void*)p;
    at->devicePointer = at->type == cudaMemoryTypeHost ? (void*)p : NULL;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t bytes, enum cudaMemcpyKind kind) {
    if (kind == cudaMemcpyHostToDevice && fake_mixed(from, bytes)) return fake_fail(cudaErrorInvalidValue);
    if (kind == cudaMemcpyDeviceToHost && fake_mixed(to, bytes)) return fake_fail(cudaErrorInvalidValue);
    memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, enum cudaMemcpyKind kind,
                            cudaStream_t stream) {
    return cudaMemcpy(to, from, bytes, kind);
}
cudaError_t cudaMemset(void* to, int value, size_t bytes) {
    memset(to, value, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* to, int value, size_t bytes, cudaStream_t stream) {
    return cudaMemset(to, value, bytes);
}
