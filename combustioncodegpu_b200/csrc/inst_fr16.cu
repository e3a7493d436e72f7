// Kernel instantiation: bulk precision float, a runtime species count of at most 16.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(float, -16)
}  // namespace ccb
