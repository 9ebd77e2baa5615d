// Resident sweeps in the whole device, 1 plane per thread.
#include "sor_resident_launch.cuh"

namespace vb {
namespace resident {
template bool launch_planes<1, true>(Mode, int, int, const Shape&, const Args&, bool, cudaStream_t);
}
}  // namespace vb
