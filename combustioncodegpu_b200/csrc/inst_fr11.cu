// Kernel instantiation: bulk precision float, a runtime species count of at most 11.
#include "launch.cuh"
namespace ccb {
CCB_INSTANTIATE(float, -11)
}  // namespace ccb
