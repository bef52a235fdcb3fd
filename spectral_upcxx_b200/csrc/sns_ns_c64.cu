// The passes of the Navier-Stokes step in complex64.
#define SNS_NS_PASSES
#include "sns_ns_passes.cuh"

namespace sns {
SNS_NS_PASSES_OF(float)
}  // namespace sns
