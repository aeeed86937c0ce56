// sph_force_lanes64_3.cu -- the FP64 force pass over the cell windows of small
// launches in 3D.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceLanes, double, 3>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
