// The CUDA runtime calls of copystage.cpp, faked: what fails is set by the
// test, and the last error is kept as the runtime keeps it (a call that
// succeeds leaves it alone).
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../moldy_b200/csrc/copystage.h"

static cudaError_t g_last = cudaSuccess;
static bool g_no_pinned = false, g_unknown_pointer = false, g_dst_pinned = false;
static int g_copies = 0;

static cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}

extern "C" {
cudaError_t cudaGetLastError() { cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (g_no_pinned) return ret(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)0x1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    if (g_unknown_pointer) return ret(cudaErrorInvalidValue);
    a->type = g_dst_pinned ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    ++g_copies;
    return cudaSuccess;
}
}

#define EXPECT(c)                                                     \
    do {                                                              \
        if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } \
    } while (0)

int main() {
    const size_t sizes[] = {0, 8, 65536, 65537, moldy::kStageBytes, moldy::kStageBytes + 1, 5 * moldy::kStageBytes + 123};
    for (int opened = 0; opened < 2; ++opened)
        for (int pinned = 0; pinned < 2; ++pinned)
            for (int unknown = 0; unknown < 2; ++unknown)
                for (size_t n : sizes) {
                    g_dst_pinned = pinned; g_unknown_pointer = unknown;
                    moldy::CopyStage c;
                    if (opened) EXPECT(c.open(100) == cudaSuccess);
                    std::vector<unsigned char> a(n + 1), b(n + 1, 0);
                    for (size_t k = 0; k < n; ++k) a[k] = (unsigned char)(k * 31 + 7);
                    a[n] = 0;
                    EXPECT(c.out(b.data(), a.data(), n, nullptr) == cudaSuccess);
                    EXPECT(a == b);
                    EXPECT(cudaPeekAtLastError() == cudaSuccess);
                }
    g_dst_pinned = g_unknown_pointer = false;
    // a launch that failed before the copy: handed on, nothing copied
    for (int opened = 0; opened < 2; ++opened) {
        moldy::CopyStage c;
        if (opened) EXPECT(c.open(100) == cudaSuccess);
        unsigned char x[8] = {1}, y[8] = {2};
        g_last = cudaErrorInvalidConfiguration;
        EXPECT(c.out(y, x, 8, nullptr) == cudaErrorInvalidConfiguration);
        EXPECT(y[0] == 2);
        g_last = cudaSuccess;
    }
    // no pinned memory: the copy goes without, and no error is left behind
    {
        moldy::CopyStage c;
        g_no_pinned = true;
        EXPECT(c.open(100) != cudaSuccess);
        EXPECT(cudaPeekAtLastError() == cudaSuccess);
        std::vector<unsigned char> a(300000, 3), b(300000, 0);
        g_dst_pinned = true;
        EXPECT(c.out(b.data(), a.data(), a.size(), nullptr) == cudaSuccess && a == b);
        EXPECT(cudaPeekAtLastError() == cudaSuccess);
        g_no_pinned = false;
        EXPECT(c.open(100) == cudaSuccess && c.head && c.piece);
        // an error of an earlier call is not lost by opening
        moldy::CopyStage q;
        g_last = cudaErrorInvalidConfiguration;
        (void)q.open(100);
        EXPECT(cudaPeekAtLastError() == cudaErrorInvalidConfiguration);
    }
    std::printf("ok\n");
    return 0;
}
