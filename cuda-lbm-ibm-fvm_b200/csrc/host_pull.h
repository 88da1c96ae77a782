// host_pull.h -- device to pageable host copies through pinned chunks and several threads (host_pull.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace vof {

constexpr int PULL_THREADS = 8;
constexpr size_t PULL_CHUNK = 256 << 10;  // bytes a thread copies at a time (two chunks each in flight)

// What the copies of one context keep; zero-initialised, filled by the first large copy.
struct HostPull {
    char* pinned;  // PULL_THREADS x 2 chunks
    cudaStream_t stream[PULL_THREADS];
    cudaEvent_t ready, done[PULL_THREADS][2];
    bool made;
};

// Copy `bytes` contiguous bytes of the current device (src) to host memory
// after the work on s; returns when they are there.
cudaError_t host_pull(HostPull* h, void* dst, const void* src, size_t bytes, cudaStream_t s);
void host_pull_destroy(HostPull* h);

}  // namespace vof
