// xy phase of the NS step on small planes: y-inverse of the six fields,
// x-inverse, cross product, x-forward and y-forward in one CTA per xy plane
// (host interface; kernels in sns_plane.cu).
#pragma once

#include <cuda_runtime.h>

namespace sns {

// Whether a CTA can hold the six fields' plane of stored rows of nx values.
bool plane_supported(int nx, int ny, int prec);
// The xy phase of nz planes in place on U[0..5]: U[0..2] = y- and x-transformed
// cross product (U[3..5] are left as they were).  real: half-spectrum rows.
int plane_run(void* const U[6], int nx, int ny, int nz, int prec, bool real, cudaStream_t s);

}  // namespace sns
