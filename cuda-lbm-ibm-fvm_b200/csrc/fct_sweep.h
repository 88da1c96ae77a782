// fct_sweep.h -- one fused FCT sweep of the volume fraction (fct_sweep.cu).
#pragma once
#include <cuda_runtime.h>

#include "vof_device.cuh"

namespace vof {

// Enqueue the sweep along `axis` (0 = x, 1 = y, 2 = z) on stream s with the
// face velocity `vel` of that axis: reads Fin, writes Fout, another buffer (its
// interior cells; final_sweep: the last sweep of the step, which also applies
// the final clamp and the F boundary conditions, so every ghost cell too).
// On a non-final sweep Fout's ghost cells must already hold finite values (the
// next sweep reads them only through wall-face fluxes of zero velocity).
cudaError_t fct_launch_to(const Geom& g, int axis, bool final_sweep, const float* Fin, float* Fout, const float* vel,
                          cudaStream_t s);

// Whether a sweep takes lines of n cells.
bool fct_supported(int n);

}  // namespace vof
