// Kernel instantiation: bulk precision double, a runtime species count of at most 8.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(double, -8)
}  // namespace ccb
