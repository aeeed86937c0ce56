// sph_force_lanes2.cu -- the mixed-precision force pass of small launches in 2D.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceLanes, float, 2>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
