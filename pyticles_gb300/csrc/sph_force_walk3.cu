// sph_force_walk3.cu -- the mixed-precision force pass in 3D, one particle per
// thread over the cell windows.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceWalk, float, 3>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
