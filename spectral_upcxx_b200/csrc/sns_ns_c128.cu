// The passes of the Navier-Stokes step in complex128.
#define SNS_NS_PASSES
#include "sns_ns_passes.cuh"

namespace sns {
SNS_NS_PASSES_OF(double)
}  // namespace sns
