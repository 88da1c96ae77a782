// jacobi_cluster.h -- all Jacobi sweeps of a small grid in one launch (jacobi_cluster.cu).
#pragma once
#include <cuda_runtime.h>

#include "vof_device.cuh"

namespace vof {

// Whether `iters` sweeps of a grid fit one cluster and are enough of them.
bool jacobi_cluster_fits(const Geom& g, int iters);

// `iters` (1 or more) Jacobi sweeps from p[src] with rhs into the interior of
// p[src] (iters even) or of the other of the two buffers (odd), whose ghost
// cells are read as the sweeps' ping-pong reads them and left as they are.
cudaError_t jacobi_cluster_launch(const Geom& g, float* const p[2], int src, const float* rhs, int iters,
                                  cudaStream_t s);

// Query the device's largest cluster (once per device).
cudaError_t jacobi_cluster_configure();

}  // namespace vof
