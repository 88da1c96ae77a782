// csrc/host_pull.cu on the host, over a fake of the runtime calls it makes
// (tests/test_host_pull.py): copies of several sizes with nothing failing, and
// with the n-th thread's start failing in either of the two ways it can.
#include <errno.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <new>
#include <vector>

#include "host_pull.cu"

static std::atomic<int> fail_new{-1}, fail_thread{-1};  // calls until one fails (-1: none)
static bool due(std::atomic<int>& n) { return n.load() >= 0 && n.fetch_sub(1) == 0; }

void* operator new(size_t n) {
    if (due(fail_new)) throw std::bad_alloc();
    if (void* p = malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

extern "C" int __real_pthread_create(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
extern "C" int __wrap_pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    return due(fail_thread) ? EAGAIN : __real_pthread_create(t, a, f, x);
}

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    return memcpy(dst, src, n), cudaSuccess;
}
}

// One copy with the given call failing; false if its bytes or status are wrong.
static bool copies(vof::HostPull* h, size_t bytes, int nth_new, int nth_thread) {
    std::vector<unsigned char> src(bytes), dst(bytes, 0);
    for (size_t q = 0; q < bytes; ++q) src[q] = (unsigned char)(q * 2654435761u >> 13);
    fail_new = nth_new;
    fail_thread = nth_thread;
    const cudaError_t e = vof::host_pull(h, dst.data(), src.data(), bytes, nullptr);
    fail_new = fail_thread = -1;
    return e == cudaSuccess && src == dst;
}

int main() {
    vof::HostPull h = {};
    const size_t sizes[] = {(4u << 20) - 8, 4u << 20, (4u << 20) + 8, (5u << 20) + 12345, 16u << 20};
    int bad = 0;
    for (size_t n : sizes) {
        bad += !copies(&h, n, -1, -1);
        for (int f = 0; f < vof::PULL_THREADS; ++f) bad += !copies(&h, n, f, -1) + !copies(&h, n, -1, f);
    }
    vof::host_pull_destroy(&h);
    printf("%d wrong\n", bad);
    return bad != 0;
}
