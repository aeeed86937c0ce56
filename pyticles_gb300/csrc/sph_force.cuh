// sph_force.cuh -- the force pass and the integrator stage:
//
//   k_force   : pressure + cohesive accelerations, Monaghan viscosity, energy
//               rate incl. conduction (forces.py:338-405, c_forces.pyx:96-111,
//               163-178, 224-237) fused with the integrator stage update
//               (integrator.py:14-103), periodic teleport (box.py:33-47) and the
//               thermostat (particles.py:450-457).
//
// Instantiated per form and dimension in sph_force_*.cu.
#pragma once

#include "sph_pairs.cuh"

namespace sph {

// Next evaluation state: positions/velocities/energy in FP64 plus packed
// cell-local copies relative to the particle's cell (binned at x0).
template <typename R, int D>
__device__ __forceinline__ void write_eval_state(const View &v, const SimDev &S, int i,
                                                 const double *x, const double *vel, double u,
                                                 double m) {
    using T4 = typename V4<R>::T;
    R xl[3] = {0, 0, 0}, vv[3] = {0, 0, 0};
    bool skin = false;
    double moved = 0.0;   // squared displacement from the pair lists' build
#pragma unroll
    for (int a = 0; a < D; ++a) {
        // relative to the cell the particle was binned in; with binning on
        // demand the step may have started from a wrapped position
        double d = x[a] - v.org[a][i];
        if (d > S.half_L[a]) d -= S.L[a];
        if (d < -S.half_L[a]) d += S.L[a];
        if (v.vl_on) {
            const float4 x0 = v.vl_x0[i];
            const double m = d - (double)(a == 0 ? x0.x : (a == 1 ? x0.y : x0.z));
            moved += m * m;
        }
        xl[a] = (R)d;
        vv[a] = (R)vel[a];
        v.xe_out[a][i] = x[a];
        v.ve_out[a][i] = vel[a];
        // the cell list finds every pair while each particle stays within its
        // cell grown by the slack
        skin |= fabs(d) > S.box_half[a];
    }
    // with pair lists: a pair can be missing from them once a particle has
    // moved half the skin
    skin |= moved > S.vl_eskin2;
    if (skin) set_err(v.err, v.err_any, v.b_sim[i], SPH_ESKIN);
    v.ue_out[i] = u;
    store_packed<R>(v.pk_pos_out, v.pk_vel_out, D == 2, i, xl, vv, (R)m);
}

// Final state of the step into A (same slot as B), with the teleport wrap.
// In rebin mode it is also the next step's start state in B and its packed
// stage-0 copies, relative to the unchanged cells (the final stage writes
// pk_*_out == buffer 0 for improved Euler and RK4); a particle past half of
// its cell slack -- with pair lists, one that has moved a quarter of the
// skin since their build -- asks for a binning before the next step.
template <typename R, int D>
__device__ __forceinline__ void write_final_state(const View &v, const SimDev &S, int i,
                                                  double *x, const double *vel, double u) {
    using T4 = typename V4<R>::T;
    R xl[3] = {0, 0, 0}, vv[3] = {0, 0, 0};
    bool far = false;
    double moved = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        double L = S.L[a];
        if (x[a] > L) x[a] = 0;
        if (x[a] < 0) x[a] = L;
        v.a_pos[a][i] = x[a];
        v.a_vel[a][i] = vel[a];
        if (v.reuse) {
            double d = x[a] - v.org[a][i];
            if (d > S.half_L[a]) d -= L;   // the wrap moved it across the box
            if (d < -S.half_L[a]) d += L;
            if (v.vl_on) {
                const float4 x0 = v.vl_x0[i];
                const double m = d - (double)(a == 0 ? x0.x : (a == 1 ? x0.y : x0.z));
                moved += m * m;
            } else {
                far |= fabs(d) > S.rebin_half[a];
            }
            xl[a] = (R)d;
            vv[a] = (R)vel[a];
            v.b_pos[a][i] = x[a];
            v.b_vel[a][i] = vel[a];
        }
    }
    v.a_u[i] = u;
    v.a_m[i] = v.b_m[i];
    v.a_id[i] = v.b_id[i];
    v.a_sim[i] = v.b_sim[i];
    if (v.reuse) {
        far |= moved > S.vl_gate2;
        v.b_u[i] = u;
        store_packed<R>(v.pk_pos_out, v.pk_vel_out, D == 2, i, xl, vv,
                        flat2<R, D> ? (R)0 : (R)v.b_m[i]);
        if (far) *v.rebin_gate = 1;
    }
}

// Integrator stage of particle i (c = xdot dt as in integrator.py:14-103)
// from its rates vdr, udr, followed on the last stage by the teleport wrap
// and the thermostat.
template <typename R, int D>
__device__ __forceinline__ void integrate_stage(const View &v, const SimDev &S, int i, int s,
                                                int stage, int integ, const R *vdr, R udr) {
    const double dt = S.dt;
    double x0[3] = {0, 0, 0}, v0[3] = {0, 0, 0}, rd[3] = {0, 0, 0}, vd[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < D; ++a) {
        x0[a] = v.b_pos[a][i];
        v0[a] = v.b_vel[a][i];
        rd[a] = v.ve_in[a][i];
        vd[a] = (double)vdr[a];
    }
    double u0 = v.b_u[i], udd = (double)udr, m = v.b_m[i];
    double x[3] = {0, 0, 0}, vel[3] = {0, 0, 0}, u;
    bool final_stage = false;
    // Euler and improved Euler in FMA form: x0 + dt f and x0 + dt/2 (f0 + f1)
    // (integrator.py:14-59 round c = f dt and (c1 + c2)/2 separately; the
    // difference is one rounding per step, far below the FP64 tolerance)
    if (integ == SPH_EULER) {
        for (int a = 0; a < D; ++a) {
            x[a] = fma(dt, rd[a], x0[a]);
            vel[a] = fma(dt, vd[a], v0[a]);
        }
        u = fma(dt, udd, u0);
        final_stage = true;
    } else if (integ == SPH_IEULER) {
        if (stage == 0) {
            for (int a = 0; a < D; ++a) {
                ((R *)v.f0v[a])[i] = vdr[a];
                x[a] = fma(dt, rd[a], x0[a]);
                vel[a] = fma(dt, vd[a], v0[a]);
            }
            ((R *)v.f0u)[i] = udr;
            u = fma(dt, udd, u0);
            write_eval_state<R, D>(v, S, i, x, vel, u, m);
        } else {
            const double hdt = S.hdt;
            for (int a = 0; a < D; ++a) {
                x[a] = fma(hdt, v0[a] + rd[a], x0[a]);
                vel[a] = fma(hdt, (double)((const R *)v.f0v[a])[i] + vd[a], v0[a]);
            }
            u = fma(hdt, (double)((const R *)v.f0u)[i] + udd, u0);
            final_stage = true;
        }
    } else {  // RK4
        double cr[3], cv[3], cu = dmul(udd, dt);
        for (int a = 0; a < D; ++a) {
            cr[a] = dmul(rd[a], dt);
            cv[a] = dmul(vd[a], dt);
        }
        if (stage == 0) {
            for (int a = 0; a < D; ++a) {
                v.acc_r[a][i] = cr[a];
                v.acc_v[a][i] = cv[a];
                x[a] = dadd(x0[a], cr[a] / 2.0);
                vel[a] = dadd(v0[a], cv[a] / 2.0);
            }
            v.acc_u[i] = cu;
            u = dadd(u0, cu / 2.0);
            write_eval_state<R, D>(v, S, i, x, vel, u, m);
        } else if (stage < 3) {
            for (int a = 0; a < D; ++a) {
                v.acc_r[a][i] = dadd(v.acc_r[a][i], dmul(2.0, cr[a]));
                v.acc_v[a][i] = dadd(v.acc_v[a][i], dmul(2.0, cv[a]));
                x[a] = stage == 1 ? dadd(x0[a], cr[a] / 2.0) : dadd(x0[a], cr[a]);
                vel[a] = stage == 1 ? dadd(v0[a], cv[a] / 2.0) : dadd(v0[a], cv[a]);
            }
            v.acc_u[i] = dadd(v.acc_u[i], dmul(2.0, cu));
            u = stage == 1 ? dadd(u0, cu / 2.0) : dadd(u0, cu);
            write_eval_state<R, D>(v, S, i, x, vel, u, m);
        } else {
            for (int a = 0; a < D; ++a) {
                x[a] = dadd(x0[a], dmul(1.0 / 6.0, dadd(v.acc_r[a][i], cr[a])));
                vel[a] = dadd(v0[a], dmul(1.0 / 6.0, dadd(v.acc_v[a][i], cv[a])));
            }
            u = dadd(u0, dmul(1.0 / 6.0, dadd(v.acc_u[i], cu)));
            final_stage = true;
        }
    }
    if (final_stage) {
        if (S.thermostat) {
            // particles.py:450-457: T <- T * target / mean(T); u <- k_B T - a rho
            R *tp = (R *)v.temp;
            double T = (double)tp[i] * v.t_scale[s];
            u = dadd(dmul(T, S.kb), -dmul(S.a, (double)((const R *)v.rho0)[i]));
            tp[i] = (R)T;
        }
        write_final_state<R, D>(v, S, i, x, vel, u);
    }
}

// Epilogue of the force passes: the rates of particle i and, with mode, its
// integrator stage.
template <typename R, int D>
__device__ __forceinline__ void force_finish(const View &v, const SimDev &S, int i, int s, int stage,
                                             int mode, int integ, const R *vdr, R udr) {
    for (int a = 0; a < D; ++a) ((R *)v.vdot[a])[i] = vdr[a];
    ((R *)v.udot)[i] = udr;
    if (!isfinite(vdr[0]) || !isfinite(udr)) set_err(v.err, v.err_any, s, SPH_ENAN);
    if (mode == 0) return;

    integrate_stage<R, D>(v, S, i, s, stage, integ, vdr, udr);
}

// VH: bit 0 viscosity, bit 1 heat flux (compile-time, so a workload without
// them carries neither their registers nor their branches).  ONE: a single
// simulation, whose constants come from the kernel parameters.
// Register caps by resident blocks of 256 threads; force of a step, us: a single
// simulation in 2D (199k particles) 324 / 337 / 294 at 4 / 5 / 6 blocks, in 3D (205k)
// 2248 / 2649 at 4 / 5.  3D at 3 blocks is 3% faster at 205k, whose last wave it fills,
// and slower elsewhere; whole step at 3 / 4: 46,656 particles 1684 / 1727, 125,000 2668 /
// 2344, 205,379 3444 / 3497, 343,000 5336 / 5309, 729,000 10154 / 9751, 1,331,000 18098 /
// 17391.  Several in 2D at 5 / 4: 24 of 16,900 944 / 935, with a cutoff of 1.5 491 / 456,
// 3 of 90,000 684 / 669.
// LIST: the pair lists (tuning.pair_scheme 2) instead of the cell windows.
// LANES: lanes per particle (for_pairs_lanes; the same bits).
template <typename R, int D, int K, int VH, bool ONE, bool LIST = false, int LANES = 1>
__device__ __forceinline__ void force_one(const View &v, int stage, int mode, int integ, int i) {
    constexpr bool visc = (VH & 1) != 0;
    constexpr bool heat = (VH & 2) != 0;
    bool active = i < v.np;
    const int ii = active ? i : v.np - 1;
    using T4 = typename V4<R>::T;
    const T4 *__restrict__ P = (const T4 *)v.pk_pos_in;
    const T4 *__restrict__ FV = (const T4 *)v.pk_fv;
    const float2 *__restrict__ FR = (const float2 *)v.pk_fv;   // 2D mixed: {p/rho^2, rho}
    const R *__restrict__ RHO = (const R *)v.rho;
    const T4 *__restrict__ Q = (const T4 *)v.pk_q;
    const int s = v.b_sim[ii];
    const SimDev &S = ONE ? v.one : v.sims[s];
    if (S.cl_on || (!LIST && S.tile_on)) {   // cluster passes, cell tiles
        if (LANES == 1) return;
        active = false;
    }
    KConst<R> ks = make_kconst<R>(S, 0);
    // the long kernel with pco_i/rho_l,i^2 + pco_j/rho_l,j^2 = -2a folded in
    KConst<R> kl = make_kconst_cohesive<R>(S);
    const SimConst<R> &sc = sconst<R>(S);
    const R hs = sc.hs, eps_h2 = sc.eps_h2;
    const R alpha_c = sc.alpha_c, beta = sc.beta;
    // own velocity, p/rho^2 and rho
    T4 fvi;
    if constexpr (flat2<R, D>) {
        const T4 p = P[ii];
        fvi = make_v4<R>(p.z, p.w, FR[ii].x, FR[ii].y);
    } else {
        fvi = FV[ii];
    }
    const R vix = fvi.x, viy = fvi.y, viz = D == 3 ? fvi.z : (R)0;
    const R fsi = D == 2 ? fvi.z : fvi.w;
    const R rhoi = D == 2 ? fvi.w : RHO[ii];
    const T4 qi = heat ? Q[ii] : make_v4<R>(0, 0, 0, 0);
    BAcc<R> ax[3], ud;
    ax[0].init(0);
    ax[1].init(0);
    ax[2].init(0);
    ud.init(0);
    auto cell_done = [&]() {
        ax[0].flush();
        ax[1].flush();
        if (D == 3) ax[2].flush();
        ud.flush();
    };
    if (LANES == 1 && !active) return;
    with_masses<R, D, (LANES > 1)>(v, s, [&](auto same) {
        const PairMass<R, D, decltype(same)::value> mass(v, ii);
        // loaded: what the pair lists fetch of j beside its position, the velocity
        // record in 3D (in 2D the position record holds the velocity).  Waiting
        // for it after the test held the 3D list pass up: 3350 us a launch at
        // 2M particles, 2920 with the load ahead of the test; the heat record
        // ahead as well made 2960, two or four entries' records at once 3110 and
        // 3970 (registers).
        auto body = [&](int j, const T4 &pj, const R *d, R rsq, auto near, auto... loaded) {
            constexpr bool NEAR = decltype(near)::value;
            const Dist<R> dd = make_dist<R>(rsq);
            const R gl = kernel_g<K, R, true>(kl, dd);   // -2a grad W_l / r
            T4 fvj;
            if constexpr (flat2<R, D>) {
                fvj.x = pj.z;
                fvj.y = pj.w;
                if constexpr (NEAR) {
                    const float2 fr = FR[j];
                    fvj.z = fr.x;
                    fvj.w = fr.y;
                }
            } else if constexpr (LIST) {
                fvj = (loaded, ...);
            } else {
                fvj = FV[j];
            }
            const R mj = mass(j, pj);
            R dvdx = fma_(fvj.y - viy, d[1], (fvj.x - vix) * d[0]);
            if (D == 3) dvdx = fma_(fvj.z - viz, d[2], dvdx);
            // beyond the short support gs = 0: the pressure and viscosity terms
            // vanish and gsum = gl bit for bit
            R gsum = gl, gs = (R)0;
            // the heat record {q/rho^2, rho}: with heat flux in 3D it also
            // carries the density the viscosity needs
            T4 qj = make_v4<R>(0, 0, 0, 0);
            if constexpr (NEAR) {
                if (heat) qj = Q[j];
                gs = kernel_g<K, R, true>(ks, dd);
                R ps = fsi + (D == 2 ? fvj.z : fvj.w);
                // Monaghan viscosity on approaching pairs within the short
                // support (beyond it gs = 0, so ps no longer enters gsum and the
                // warp skips the block when none of its pairs needs it)
                if (visc && dvdx < (R)0 && gs != (R)0) {
                    const R rhoj = D == 2 ? fvj.w : (heat ? qj.w : RHO[j]);
                    const R mu = fdiv<R>(hs * dvdx, rsq + eps_h2);
                    ps = add_div<R>((R)2 * fma_(beta * mu, mu, -(alpha_c * mu)), rhoi + rhoj, ps);
                }
                gsum = fma_(ps, gs, gl);
            }
            ax[0].madd(gsum, d[0]);
            ax[1].madd(gsum, d[1]);
            if (D == 3) ax[2].madd(gsum, d[2]);
            // twice the energy-rate term; the sum is halved once at the end
            // (scaling by 2 is exact, so the bits are those of the halved terms)
            R du = gsum * dvdx;
            if (heat && NEAR) {
                R dq = fma_(qi.y + qj.y, d[1], (qi.x + qj.x) * d[0]);
                if (D == 3) dq = fma_(qi.z + qj.z, d[2], dq);
                du = fma_((R)-2 * dq, gs, du);
            }
            ud.madd(du, mj);
        };
        PairFrame<R, D> fr;
        fr.init(S);
        if constexpr (LANES > 1)
            for_pairs_lanes<R, D, LANES, false>(v, S, fr, P, ii, P[ii], active, body,
                                                      [&](unsigned mask) {
                                                          fold_lanes<LANES>(ax[0], mask);
                                                          fold_lanes<LANES>(ax[1], mask);
                                                          if (D == 3) fold_lanes<LANES>(ax[2], mask);
                                                          fold_lanes<LANES>(ud, mask);
                                                      });
        else if constexpr (LIST)
            for_list<R, D, true>(v, S, fr, P, i, P[i], body, cell_done, [] {}, [&](int j) {
                if constexpr (flat2<R, D>) return NoRecord{};
                else return FV[j];
            });
        else
            for_pairs<R, D, D == 3, false>(v, S, fr, P, i, P[i], body, cell_done);
    });
    R vdr[3] = {ax[0].get(), ax[1].get(), ax[2].get()};
    R udr = (R)0.5 * ud.get();
    if constexpr (LANES > 1) {   // the epilogue by consecutive threads (lanes_block)
        constexpr int N = lanes_block<LANES> / LANES;   // particles of the block
        __shared__ T4 rates[N];
        __shared__ int live[N];
        if ((threadIdx.x & (LANES - 1)) == 0) {
            rates[threadIdx.x / LANES] = make_v4<R>(vdr[0], vdr[1], vdr[2], udr);
            live[threadIdx.x / LANES] = active;
        }
        __syncthreads();
        const int t = threadIdx.x, p = blockIdx.x * N + t;
        if (t >= N || !live[t]) return;
        const R vd[3] = {rates[t].x, rates[t].y, rates[t].z};
        const int sp = v.b_sim[p];
        force_finish<R, D>(v, v.sims[sp], p, sp, stage, mode, integ, vd, rates[t].w);
    } else {
        force_finish<R, D>(v, S, i, s, stage, mode, integ, vdr, udr);
    }
}

// One thread per particle; PERSIST: the resident blocks of pass_grid walk
// the particles grid-stride (the same per-particle work, the same bits).
template <typename R, int D, int K, int VH, bool ONE, bool PERSIST>
__global__ void __launch_bounds__(256, ONE && D == 2 ? 6 : 4) k_force(const __grid_constant__ View v, int stage,
                                                  int mode, int integ) {
    if constexpr (PERSIST) {
        for (int base = blockIdx.x * blockDim.x; base < v.np; base += gridDim.x * blockDim.x)
            force_one<R, D, K, VH, ONE>(v, stage, mode, integ, base + threadIdx.x);
    } else {
        force_one<R, D, K, VH, ONE>(v, stage, mode, integ, blockIdx.x * blockDim.x + threadIdx.x);
    }
}

// The force pass over the pair lists (mixed precision); a single
// simulation at SPH_VL_FORCE_BLOCKS (2D) / SPH_VL_FORCE3_BLOCKS (3D)
// resident blocks of 256 per SM.
#ifndef SPH_VL_FORCE_BLOCKS
#define SPH_VL_FORCE_BLOCKS 5
#endif
#ifndef SPH_VL_FORCE3_BLOCKS
#define SPH_VL_FORCE3_BLOCKS 4
#endif
#ifndef SPH_VL_FORCE_MULTI_BLOCKS
#define SPH_VL_FORCE_MULTI_BLOCKS 4
#endif
template <int D, int K, int VH, bool ONE>
__global__ void __launch_bounds__(256, ONE ? (D == 2 ? SPH_VL_FORCE_BLOCKS : SPH_VL_FORCE3_BLOCKS) : SPH_VL_FORCE_MULTI_BLOCKS)
    k_force_vl(const __grid_constant__ View v, int stage, int mode, int integ) {
    force_one<float, D, K, VH, ONE, true>(v, stage, mode, integ,
                                          blockIdx.x * blockDim.x + threadIdx.x);
}

// The cell windows of a small launch, LANES lanes per particle.
template <typename R, int D, int K, int VH, int LANES>
__global__ void __launch_bounds__(256)
    k_force_lanes(const __grid_constant__ View v, int stage, int mode, int integ) {
    force_one<R, D, K, VH, false, false, LANES>(
        v, stage, mode, integ, (blockIdx.x * blockDim.x + threadIdx.x) / LANES);
}

// Integrator stage from the stored rates: the epilogue of k_force as a pass
// of its own, for steps whose velocities change between the force pass and
// the update (hard collisions).
template <typename R, int D>
__global__ void __launch_bounds__(256) k_integrate(View v, int stage, int integ, int cl_only) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.np) return;
    const int s = v.b_sim[i];
    const SimDev &S = v.sims[s];
    if (!S.active || (cl_only && !S.cl_on)) return;
    R vdr[3] = {0, 0, 0};
    for (int a = 0; a < D; ++a) vdr[a] = ((const R *)v.vdot[a])[i];
    integrate_stage<R, D>(v, S, i, s, stage, integ, vdr, ((const R *)v.udot)[i]);
}

// The forms of the force pass, each instantiated in a translation unit of its
// own (sph_force_*.cu) per dimension.  The persistent form is for the
// mixed-precision pass only (see density_launch); FP64 walks (and lanes) serve the
// simulations that are too sparse for cell tiles.
enum ForceForm { kForceWalk, kForceList, kForceLanes };

template <int FORM, typename R, int D, int K, int VH, bool ONE>
void force_launch(const View &v, int stage, int mode, int integ, int block, cudaStream_t s) {
    const int grid = (v.np + block - 1) / block;
    if constexpr (FORM == kForceList) {
        k_force_vl<D, K, VH, ONE><<<grid, block, 0, s>>>(v, stage, mode, integ);
    } else if constexpr (FORM == kForceLanes) {
        if (walk_lanes<R>(v) == 32)
            k_force_lanes<R, D, K, VH, 32><<<lanes_grid<32>(v), lanes_block<32>, 0, s>>>(v, stage, mode, integ);
        else
            k_force_lanes<R, D, K, VH, 8><<<lanes_grid<8>(v), lanes_block<8>, 0, s>>>(v, stage, mode, integ);
    } else if (std::is_same<R, float>::value && v.persist) {
        auto *fn = k_force<R, D, K, VH, ONE, std::is_same<R, float>::value>;
        fn<<<pass_grid(v, fn, block), block, 0, s>>>(v, stage, mode, integ);
    } else {
        k_force<R, D, K, VH, ONE, false><<<grid, block, 0, s>>>(v, stage, mode, integ);
    }
}

template <int FORM, typename R, int D>
void launch_force_t(const View &v, int kernel, int viscosity, int heat, int integrator, int stage,
                    int mode, int block, cudaStream_t s) {
    const int vh = (viscosity ? 1 : 0) | (heat ? 2 : 0);
    // constants from the kernel parameters for a single simulation
    constexpr bool kOne = std::is_same<R, float>::value && FORM != kForceLanes;
#define SPH_FORCE(VH_)                                                                        \
    (v.one_sim && kOne                                                                        \
         ? force_launch<FORM, R, D, K, VH_, kOne>(v, stage, mode, integrator, block, s)       \
         : force_launch<FORM, R, D, K, VH_, false>(v, stage, mode, integrator, block, s))
#define SPH_FORCE_VH                                                                     \
    switch (vh) {                                                                        \
        case 0: SPH_FORCE(0); break;                                                     \
        case 1: SPH_FORCE(1); break;                                                     \
        case 2: SPH_FORCE(2); break;                                                     \
        default: SPH_FORCE(3); break;                                                    \
    }
    SPH_DISPATCH_K(kernel, SPH_FORCE_VH);
#undef SPH_FORCE_VH
#undef SPH_FORCE
}

template <typename R>
void launch_integrate_t(const View &v, int integrator, int stage, cudaStream_t s, int cl_only) {
    if (v.np <= 0) return;
    int nb = (v.np + 255) / 256;
    if (v.dim == 2) k_integrate<R, 2><<<nb, 256, 0, s>>>(v, stage, integrator, cl_only);
    else k_integrate<R, 3><<<nb, 256, 0, s>>>(v, stage, integrator, cl_only);
}

}  // namespace sph
