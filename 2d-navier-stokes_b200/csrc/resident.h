// resident.h -- launch interface of the resident small-grid kernel (resident.cu).
#pragma once
#include "resident.cuh"

namespace ns2d {

// Set-up of the kernels of grid size n on the current device; false when the
// size has none or the device cannot run them.
bool resident_setup(int n, bool fp32);
template <typename Real>
cudaError_t resident_launch(int n, int scheme, const ResArgs<Real>& a, cudaStream_t s);

}  // namespace ns2d
