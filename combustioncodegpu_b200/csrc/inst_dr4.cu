// Kernel instantiation: bulk precision double, a runtime species count of at most 4.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(double, -4)
}  // namespace ccb
