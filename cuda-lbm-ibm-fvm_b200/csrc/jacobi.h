// jacobi.h -- one Jacobi sweep per launch (jacobi.cu).
#pragma once
#include <cuda_runtime.h>

#include "vof_device.cuh"

namespace vof {

// One Jacobi sweep from pin (and rhs) into the interior of pout (a different
// buffer; its ghost cells are left as they are), two cells per thread, the
// wall and last planes peeled out of the z march.
cudaError_t jacobi_peel_launch(const Geom& g, const float* pin, const float* rhs, float* pout, cudaStream_t s);

// z chunk of a launch of bx blocks per chunk whose resident blocks number
// `wave`: the longest chunk whose last wave of blocks is 85 % full or more,
// else the one that fills it best.
int wave_kchunk(int nz, int bx, int wave);

// Query the kernel's occupancy (once per device).
cudaError_t jacobi_configure();

}  // namespace vof
