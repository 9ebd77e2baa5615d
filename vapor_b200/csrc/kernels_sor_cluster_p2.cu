// Resident sweeps in one cluster, 2 planes per thread.
#include "sor_resident_launch.cuh"

namespace vb {
namespace resident {
template bool launch_planes<2, false>(Mode, int, int, const Shape&, const Args&, bool, cudaStream_t);
}
}  // namespace vb
