// sph_force_lanes3.cu -- the mixed-precision force pass of small launches in 3D.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceLanes, float, 3>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
