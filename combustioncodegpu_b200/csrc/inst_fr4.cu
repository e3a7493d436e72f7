// Kernel instantiation: bulk precision float, a runtime species count of at most 4.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(float, -4)
}  // namespace ccb
