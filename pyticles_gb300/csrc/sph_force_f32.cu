// sph_force_f32.cu -- the dispatch of the force pass to its forms and the
// integrator stage pass.
#include "sph_force.cuh"

namespace sph {

#define SPH_FORM(F, R, D)                                                                     \
    extern template void launch_force_t<F, R, D>(const View &, int, int, int, int, int, int, \
                                                 int, cudaStream_t)
SPH_FORM(kForceWalk, float, 2);
SPH_FORM(kForceWalk, float, 3);
SPH_FORM(kForceList, float, 2);
SPH_FORM(kForceList, float, 3);
SPH_FORM(kForceLanes, float, 2);
SPH_FORM(kForceLanes, float, 3);
SPH_FORM(kForceLanes, double, 2);
SPH_FORM(kForceLanes, double, 3);
SPH_FORM(kForceWalk, double, 2);
SPH_FORM(kForceWalk, double, 3);
#undef SPH_FORM

void launch_force(const View &v, int precision, int kernel, int viscosity, int heat,
                  int integrator, int stage, int mode, int block, cudaStream_t s) {
    if (v.np <= 0) return;
    auto run = [&](auto fn2, auto fn3) {
        (v.dim == 2 ? fn2 : fn3)(v, kernel, viscosity, heat, integrator, stage, mode, block, s);
    };
    if (precision != SPH_MIXED) {
        if (v.n_tile > 0)
            tile_force(v, kernel, (viscosity ? 1 : 0) | (heat ? 2 : 0), integrator, stage, mode, s);
        if (v.n_walk > 0 && walk_lanes<double>(v) > 1)
            run(launch_force_t<kForceLanes, double, 2>, launch_force_t<kForceLanes, double, 3>);
        else if (v.n_walk > 0)
            run(launch_force_t<kForceWalk, double, 2>, launch_force_t<kForceWalk, double, 3>);
    } else if (v.vl_on) {
        run(launch_force_t<kForceList, float, 2>, launch_force_t<kForceList, float, 3>);
    } else if (walk_lanes<float>(v) > 1) {
        run(launch_force_t<kForceLanes, float, 2>, launch_force_t<kForceLanes, float, 3>);
    } else {
        run(launch_force_t<kForceWalk, float, 2>, launch_force_t<kForceWalk, float, 3>);
    }
}

void launch_integrate(const View &v, int precision, int integrator, int stage, cudaStream_t s,
                      int cl_only) {
    if (precision == SPH_MIXED) launch_integrate_t<float>(v, integrator, stage, s, cl_only);
    else launch_integrate_t<double>(v, integrator, stage, s, cl_only);
}

}  // namespace sph
