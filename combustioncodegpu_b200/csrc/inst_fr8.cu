// Kernel instantiation: bulk precision float, a runtime species count of at most 8.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(float, -8)
}  // namespace ccb
