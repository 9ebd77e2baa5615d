// Resident sweeps in the whole device, 3 planes per thread.
#include "sor_resident_launch.cuh"

namespace vb {
namespace resident {
template bool launch_planes<3, true>(Mode, int, int, const Shape&, const Args&, bool, cudaStream_t);
}
}  // namespace vb
