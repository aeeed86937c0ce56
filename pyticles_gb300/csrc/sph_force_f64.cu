// sph_force_f64.cu -- the plain FP64 force pass over the cell windows.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceWalk, double, 2>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);
template void launch_force_t<kForceWalk, double, 3>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
