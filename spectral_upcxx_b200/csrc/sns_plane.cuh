// xy phase of the NS step on small planes: y-inverse of the six fields,
// x-inverse, cross product, x-forward and y-forward in one CTA per xy plane
// (host interface; kernels in sns_plane.cu).
#pragma once

#include <cuda_runtime.h>

namespace sns {

// Whether a CTA can hold the six fields' plane of stored rows of nx values.
bool plane_supported(int nx, int ny, int prec);
// The xy phase of nz planes: out[0..2] = scale2 (in[0..2] x in[3..5]), both
// y- and x-inverse-transformed before and y- and x-forward-transformed after
// (out may be in[0..2]).  real: half-spectrum rows.
int plane_run(void* const in[6], void* const out[3], int nx, int ny, int nz, int prec, bool real,
              double scale2, cudaStream_t s);

}  // namespace sns
