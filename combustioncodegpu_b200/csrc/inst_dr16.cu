// Kernel instantiation: bulk precision double, a runtime species count of at most 16.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(double, -16)
}  // namespace ccb
