// Kernel instantiation: bulk precision double, a runtime species count of at most 11.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(double, -11)
}  // namespace ccb
