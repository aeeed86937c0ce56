// sph_force_list.cu -- the force pass over the pair lists.
#include "sph_force.cuh"

namespace sph {

template void launch_force_t<kForceList, float, 2>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);
template void launch_force_t<kForceList, float, 3>(const View &, int, int, int, int, int, int, int,
                                cudaStream_t);

}  // namespace sph
