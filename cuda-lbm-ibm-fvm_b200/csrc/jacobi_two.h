// jacobi_two.h -- two Jacobi sweeps per launch (jacobi_two.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "jacobi_two_plan.h"
#include "vof_device.cuh"

namespace vof {

// What the launches on one set of buffers need, made once: the tiling and the
// TMA descriptors of the three pressure buffers and of the right-hand side.
struct J2Tables {
    J2Plan plan;
    CUtensorMap map[4];
};

// Fill t for the buffers field[0 .. 2] (pressure) and field[3] (right-hand
// side), and set the right-hand side's padding columns (beyond the ghosts; no
// other kernel reads them) to a value in the fast division's range.
cudaError_t jacobi_two_prepare(const Geom& g, float* const field[4], J2Tables* t, cudaStream_t s);

// Two Jacobi sweeps from pressure buffer `in` (pin) into the interior of pout,
// another buffer.  A copy that does not land in time sets DEV_TMA_TIMEOUT in
// *status.
cudaError_t jacobi_two_launch(const Geom& g, const J2Tables& t, int in, const float* pin, float* pout, int* status,
                              cudaStream_t s);

// Raise the kernel's shared-memory ceiling (once per device).
cudaError_t jacobi_two_configure();

}  // namespace vof
