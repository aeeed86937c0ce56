// sph_tile.cu -- the FP64 pair passes of the cell windows by cell tiles.
//
// GB300's FP64 pipe takes a warp instruction every 16 cycles of an SM, so these
// passes are bound by their FP64 instructions and by the lanes those leave idle.
// One thread per particle that walks its own window (for_pairs) spends them on
// every candidate's test and runs its loop bodies at half of its lanes; here
//
//  * candidates are tested in packed FP32, two per instruction, as much too wide as
//    its rounding asks (fast_margin, short_support2; inside the guard band the bodies
//    ask the exact FP64 test), so that FP64 work begins with the pair;
//  * accepted candidates go through a queue in shared memory, pairs within the
//    short support from its front and the others from its back, so that the
//    bodies run with all lanes busy and the two kinds never diverge;
//  * square roots and quotients come from the hardware's approximations by
//    Newton and Goldschmidt steps, without range checks and branches.
//
// A block of four warps takes up to four rounds of one home cell.  It copies the
// particles of the cell's window into shared memory in the home cell's frame
// (the tile, at most kTileCap candidates at a time), and every warp evaluates
// one round of the cell's particles against it: four particles with eight lanes
// each; 16 or 32 lanes for the last two and the last one of a cell, and 32 for
// every particle of a small simulation (SimDev.tile_lg), which would otherwise
// leave SMs without a warp.  The lanes' sums are added in a fixed tree.
//
// The order of a particle's sum is a function of its own cell's window and of
// its simulation's size, so a simulation gives the same bits alone, in a batch
// and at any launch shape.
//
// The work items (cell, first round) are listed at binning (k_cellsort), so that
// dense cells and boxes of a few cells spread over as many blocks as they have
// work for.  The per-particle epilogues (equation of state, integrator) run
// after a block barrier, one thread per particle of the item.
//
// Measured, density / force pass in us, for_pairs -> tiles: 2D 1,024 particles
// 300 / 458 -> 21 / 25, 65,536 particles 887 / 1403 -> 352 / 495 (FP64 pipe 78 / 81%
// busy); 3D 2,197 particles 1988 / 2666 -> 110 / 172 (76 / 79%).
#include <algorithm>

#include "sph_force.cuh"
#include "sph_pack.cuh"

namespace sph {
namespace {

// Candidates held at a time: with 512 the 3D force pass of 2,197 particles took
// 215 us instead of 175 (fewer resident blocks), 2D passes the same.
constexpr int kTileCap = 256;
using TileSlot = unsigned char;
constexpr int kTileThreads = 32 * kTileRounds;

// max(x, 0) for a finite x, without the FP64 pipe
__device__ __forceinline__ double tile_pos(double x) {
    return __double2hiint(x) < 0 ? 0.0 : x;
}

// Whether rsq lies past the guard band's lower end, by the high words: the band
// is a few 1e-6 wide, and comparing costs the FP64 pipe as much as adding.
__device__ __forceinline__ bool tile_band(double rsq, double thr_lo) {
    return __double2hiint(rsq) >= __double2hiint(thr_lo);
}

// The distance of an FP64 pair, and 1/(2r) to about 2^-40.
struct TileDist {
    double r, ih;
    __device__ __forceinline__ explicit TileDist(double rsq) { r = tile_sqrt(rsq, &ih); }
};

// W / sigma of kernel K at the pair's distance.
template <int K>
__device__ __forceinline__ double tile_w(const KConst<double> &k, const TileDist &t) {
    if constexpr (K == SPH_KERNEL_LUCY) {
        const double s = tile_pos(fma(-t.r, k.inv_h, 1.0));
        return (s * s * s) * fma(-3.0, s, 4.0);
    } else if constexpr (K == SPH_KERNEL_GAUSSIAN) {
        const double q = t.r * k.inv_h;
        return exp(-(q * q));
    } else if constexpr (K == SPH_KERNEL_DEBRUN) {
        const double s = tile_pos(k.h - t.r);
        return s * s * s;
    } else {
        const double q = t.r * k.inv_h;
        if (q < 1.0) return fma(q * q, fma(0.75, q, -1.5), 1.0);
        const double s = tile_pos(2.0 - q);
        return 0.25 * s * s * s;
    }
}

// (dW/dr)/r of kernel K at the pair's distance.
template <int K>
__device__ __forceinline__ double tile_g(const KConst<double> &k, const TileDist &t) {
    if constexpr (K == SPH_KERNEL_LUCY) {
        const double s = tile_pos(fma(-t.r, k.inv_h, 1.0));
        return k.g0 * (s * s);
    } else if constexpr (K == SPH_KERNEL_GAUSSIAN) {
        const double q = t.r * k.inv_h;
        return k.g0 * k.sig * exp(-(q * q));
    } else if constexpr (K == SPH_KERNEL_DEBRUN) {
        const double s = tile_pos(k.h - t.r);
        return k.g0 * (s * s) * tile_inv(t.r, t.ih);
    } else {
        const double q = t.r * k.inv_h;
        if (q < 1.0) return k.g0 * fma(2.25, q, -3.0);
        const double s = tile_pos(2.0 - q);
        return k.g0 * (-0.75 * k.h) * (s * s) * tile_inv(t.r, t.ih);
    }
}

// ---- the tile ----

// Per-candidate arrays; Rec: what the pass needs of a candidate.
template <int D, typename Rec> struct TileMem {
    float t[D][kTileCap];                  // FP32 positions of the candidate test
    double p[D][kTileCap], mass[kTileCap];
    Rec rec;
    int j[kTileCap];                       // the candidate's B slot
    unsigned char c[kTileCap];             // its cell's place among the 32 being copied
    __device__ __forceinline__ void put(int k, const double *x, double m) {
#pragma unroll
        for (int a = 0; a < D; ++a) {
            t[a][k] = (float)x[a];
            p[a][k] = x[a];
        }
        mass[k] = m;
    }
};
// Each warp's queues of accepted candidates, one per particle of the round:
// near pairs from the front, far ones from the back.
struct TileQueue { TileSlot q[4][kTileCap]; };

// Sum over the G lanes of one particle, on every lane.
__device__ __forceinline__ void tile_tree(double &s, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
}

// ---- the passes: what the tile holds of a candidate, and the terms of a pair ----

struct NoRecord {};

// Density: rho_s and rho_l sums; the epilogue reads them back from pk_f (the
// slot it then overwrites) and the pair count from temp.
template <int D, int K> struct TileDensity {
    using Mem = TileMem<D, NoRecord>;
    static constexpr bool kFar = true;
    const View &v;
    KConst<double> ks, kl;
    double rs, rl;
    __device__ TileDensity(const View &v_, const SimDev &S) : v(v_) {
        ks = make_kconst<double>(S, 0);
        kl = make_kconst<double>(S, 1);
    }
    __device__ __forceinline__ static void load(const View &, Mem &, int, int,
                                                const double4_32a &) {}
    __device__ __forceinline__ void begin(int) { rs = rl = 0.0; }
    template <bool NEAR>
    __device__ __forceinline__ void pair(const Mem &mem, int k, const double *, double rsq) {
        const double m = mem.mass[k];
        const TileDist t(rsq);
        if constexpr (NEAR) rs = fma(m, tile_w<K>(ks, t), rs);
        rl = fma(m, tile_w<K>(kl, t), rl);
    }
    __device__ __forceinline__ void end(int i, int G, bool writes, int npairs) {
        tile_tree(rs, G);
        tile_tree(rl, G);
        if (!writes) return;
        ((double4_32a *)v.pk_f)[i] = make_v4<double>(rs, 0.0, rl, 0.0);
        ((double *)v.temp)[i] = (double)npairs;
    }
};

// Heat flux: only the short kernel enters.
template <int D, int K> struct TileHeat {
    struct Rec { double t[kTileCap], mr[kTileCap]; };   // T, m / rho
    using Mem = TileMem<D, Rec>;
    static constexpr bool kFar = false;
    const View &v;
    KConst<double> ks;
    double kappa, q[D];
    double4_32a fi;
    __device__ TileHeat(const View &v_, const SimDev &S) : v(v_) {
        ks = make_kconst<double>(S, 0);
        kappa = S.cd.kappa;
    }
    __device__ __forceinline__ static void load(const View &v, Mem &mem, int k, int j,
                                                const double4_32a &pj) {
        const double4_32a f = ((const double4_32a *)v.pk_f)[j];
        mem.rec.t[k] = f.z;   // f.w, what FP64 misses of T, is 0
        mem.rec.mr[k] = pj.w / f.y;
    }
    __device__ __forceinline__ void begin(int i) {
        fi = ((const double4_32a *)v.pk_f)[i];
        for (int a = 0; a < D; ++a) q[a] = 0.0;
    }
    template <bool NEAR>
    __device__ __forceinline__ void pair(const Mem &mem, int k, const double *d, double rsq) {
        const double g = tile_g<K>(ks, TileDist(rsq));
        const double f = mem.rec.mr[k] * (mem.rec.t[k] - fi.z) * g;
#pragma unroll
        for (int a = 0; a < D; ++a) q[a] = fma(f, d[a], q[a]);
    }
    __device__ __forceinline__ void end(int i, int G, bool writes, int) {
#pragma unroll
        for (int a = 0; a < D; ++a) tile_tree(q[a], G);
        if (!writes) return;
        const double ir2 = 1.0 / (fi.y * fi.y);
        double qq[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < D; ++a) {
            qq[a] = kappa * q[a];
            ((double *)v.q[a])[i] = qq[a];
        }
        ((double4_32a *)v.pk_q)[i] =
            make_v4<double>(qq[0] * ir2, qq[1] * ir2, qq[2] * ir2, fi.y);
    }
};

// Force, viscosity and energy rate; the terms of force_one (sph_force.cuh).
template <int D, int K, int VH> struct TileForce {
    static constexpr bool kFar = true;
    static constexpr bool visc = (VH & 1) != 0, heat = (VH & 2) != 0;
    struct Rec {
        double vel[D][kTileCap], fs[kTileCap], rho[visc ? kTileCap : 1];
        double q[heat ? D : 1][heat ? kTileCap : 1];
    };
    using Mem = TileMem<D, Rec>;
    const View &v;
    KConst<double> ks, kl;
    double hs, eps_h2, alpha_c, beta;
    double vi[D], fsi, rhoi, qi[D];
    double ax[D], ud;
    __device__ TileForce(const View &v_, const SimDev &S) : v(v_) {
        ks = make_kconst<double>(S, 0);
        kl = make_kconst_cohesive<double>(S);
        hs = S.cd.hs;
        eps_h2 = S.cd.eps_h2;
        alpha_c = S.cd.alpha_c;
        beta = S.cd.beta;
    }
    __device__ __forceinline__ static void load(const View &v, Mem &mem, int k, int j,
                                                const double4_32a &) {
        const double4_32a f = ((const double4_32a *)v.pk_fv)[j];
        mem.rec.vel[0][k] = f.x;
        mem.rec.vel[1][k] = f.y;
        if constexpr (D == 3) mem.rec.vel[2][k] = f.z;
        mem.rec.fs[k] = D == 2 ? f.z : f.w;
        if constexpr (visc) mem.rec.rho[k] = D == 2 ? f.w : ((const double *)v.rho)[j];
        if constexpr (heat) {
            const double4_32a q = ((const double4_32a *)v.pk_q)[j];
            mem.rec.q[0][k] = q.x;
            mem.rec.q[1][k] = q.y;
            if constexpr (D == 3) mem.rec.q[2][k] = q.z;
        }
    }
    __device__ __forceinline__ void begin(int i) {
        const double4_32a f = ((const double4_32a *)v.pk_fv)[i];
        vi[0] = f.x;
        vi[1] = f.y;
        if constexpr (D == 3) vi[2] = f.z;
        fsi = D == 2 ? f.z : f.w;
        rhoi = D == 2 ? f.w : ((const double *)v.rho)[i];
        if constexpr (heat) {
            const double4_32a q = ((const double4_32a *)v.pk_q)[i];
            qi[0] = q.x;
            qi[1] = q.y;
            if constexpr (D == 3) qi[2] = q.z;
        }
        for (int a = 0; a < D; ++a) ax[a] = 0.0;
        ud = 0.0;
    }
    template <bool NEAR>
    __device__ __forceinline__ void pair(const Mem &mem, int k, const double *d, double rsq) {
        const TileDist t(rsq);
        const double gl = tile_g<K>(kl, t);   // -2a grad W_l / r
        double dvdx = (mem.rec.vel[0][k] - vi[0]) * d[0];
#pragma unroll
        for (int a = 1; a < D; ++a) dvdx = fma(mem.rec.vel[a][k] - vi[a], d[a], dvdx);
        double gsum = gl, gs = 0.0;
        if constexpr (NEAR) {
            gs = tile_g<K>(ks, t);
            double ps = fsi + mem.rec.fs[k];
            if (visc && __double2hiint(dvdx) < 0) {   // approaching
                // 2 (-alpha mu + beta mu^2) / (rho_i + rho_j), mu = a / b
                const double b = rsq + eps_h2, a = hs * dvdx;
                ps += tile_div((a + a) * (beta * a - alpha_c * b),
                               b * b * (rhoi + mem.rec.rho[k]));
            }
            gsum = fma(ps, gs, gl);
        }
#pragma unroll
        for (int a = 0; a < D; ++a) ax[a] = fma(gsum, d[a], ax[a]);
        // twice the energy-rate term, halved once at the end
        double du = gsum * dvdx;
        if constexpr (heat && NEAR) {
            double dq = (qi[0] + mem.rec.q[0][k]) * d[0];
#pragma unroll
            for (int a = 1; a < D; ++a) dq = fma(qi[a] + mem.rec.q[a][k], d[a], dq);
            du = fma(-2.0 * dq, gs, du);
        }
        ud = fma(du, mem.mass[k], ud);
    }
    __device__ __forceinline__ void end(int i, int G, bool writes, int) {
#pragma unroll
        for (int a = 0; a < D; ++a) tile_tree(ax[a], G);
        tile_tree(ud, G);
        if (!writes) return;
#pragma unroll
        for (int a = 0; a < D; ++a) ((double *)v.vdot[a])[i] = ax[a];
        ((double *)v.udot)[i] = 0.5 * ud;
    }
};

// ---- the candidate test and the rounds ----

// A lane's candidates of one sub-tile: slots k0, k0 + G, ... (`steps` pairs of
// them, at most 32 candidates).  The test shifts a sign bit per candidate into
// the mask, so bit q is slot top - q G with top = k0 + (2 steps - 1) G.
__device__ __forceinline__ unsigned sign_in(unsigned mask, float t) {
    return __funnelshift_l(__float_as_uint(t), mask, 1);
}
__device__ __forceinline__ int top_bit(unsigned mask) {
    int q;
    asm("bfind.u32 %0, %1;" : "=r"(q) : "r"(mask));
    return q;
}

// Tests the lane's candidates of a sub-tile: `in` those within the cutoff and
// `near` those within the short support, both slightly too many (by 1e-6 of
// the threshold); the bodies decide the former exactly.  Only the first `sn`
// steps hold candidates that can be near.  MI: with the minimum image on
// single-cell axes.
template <int D, bool MI, typename Mem>
__device__ __forceinline__ void tile_test(const Mem &mem, int k, int G, int steps, int sn,
                                          const float *pt, const SimConst<float> &c, float thr,
                                          float thr_s, int small_mask, unsigned &in,
                                          unsigned &near) {
    in = near = 0u;
    // t = rsq - thr of candidates k and k + G, and with NEAR rsq - thr_s
    auto t_of = [&](int k, float &t0, float &t1, float &s0, float &s1, auto want_near) {
        if constexpr (MI) {
            float rsq[2] = {0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    float d = mem.t[a][k + h * G] - pt[a];
                    if (small_mask & (1 << a)) {
                        if (d > c.hL[a]) d -= c.L[a];
                        if (d < -c.hL[a]) d += c.L[a];
                    }
                    rsq[h] += d * d;
                }
            t0 = rsq[0] - thr;
            t1 = rsq[1] - thr;
            s0 = rsq[0] - thr_s;
            s1 = rsq[1] - thr_s;
        } else {
            F2 t = f2(-thr);
#pragma unroll
            for (int a = 0; a < D; ++a) {
                const F2 d = f2(mem.t[a][k], mem.t[a][k + G]) + f2(-pt[a]);
                t = fma2(d, d, t);
            }
            t0 = t.lo();
            t1 = t.hi();
            if constexpr (decltype(want_near)::value) {
                const F2 s = t + f2(thr - thr_s);
                s0 = s.lo();
                s1 = s.hi();
            }
        }
    };
    int b = 0;
#pragma unroll 2
    for (; b < sn; ++b, k += 2 * G) {
        float t0, t1, s0, s1;
        t_of(k, t0, t1, s0, s1, std::true_type{});
        in = sign_in(sign_in(in, t0), t1);
        near = sign_in(sign_in(near, s0), s1);
    }
#pragma unroll 4
    for (; b < steps; ++b, k += 2 * G) {
        float t0, t1, s0, s1;
        t_of(k, t0, t1, s0, s1, std::false_type{});
        in = sign_in(sign_in(in, t0), t1);
    }
    if (sn > 0) near <<= 2 * (steps - sn);
}

// One candidate of the lane's particle, with the exact pair test inside the
// guard band (a candidate that fails it is counted in drop).
template <bool NEAR, int D, typename Mem, typename Pass>
__device__ __forceinline__ void tile_pair(const View &v, const SimDev &S, const Mem &mem, int k,
                                          int i, const double *pi, double thr_lo, int &drop,
                                          Pass &pass) {
    double d[D], rsq = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        d[a] = mem.p[a][k] - pi[a];
        if (S.small_mask & (1 << a)) {   // minimum image on a single-cell axis
            if (d[a] > S.cd.hL[a]) d[a] -= S.cd.L[a];
            if (d[a] < -S.cd.hL[a]) d[a] += S.cd.L[a];
        }
        rsq = a == 0 ? d[a] * d[a] : fma(d[a], d[a], rsq);
    }
    if (tile_band(rsq, thr_lo) && !exact_in_set<D>(v.xe_in, &S, i, mem.j[k])) {
        ++drop;
        return;
    }
    pass.template pair<NEAR>(mem, k, d, rsq);
}

// The window of one home cell, copied into the tile piece by piece.  Every
// warp of the block keeps the same state: a lane for each of 32 window cells.
template <int D, typename Pass> struct Window {
    int base, ncw, jb, je, wc, cp;
    bool nearcap;                 // the lane's cell can hold near pairs
    double off[D];                // its frame
    int T, Tn;                    // candidates; those past Tn are not near
    int s_first, s_last, s_base;  // the home cell's: j sits at slot j - s_base

    __device__ __forceinline__ void start(const View &v, const SimDev &S, int home) {
        cp = v.cell_xyz[home];
        ncw = (2 * S.win[0] + 1) * (2 * S.win[1] + 1) * (D == 3 ? 2 * S.win[2] + 1 : 1);
        base = 0;
        jb = je = 0;
        wc = -1;
        nearcap = false;
    }
    __device__ __forceinline__ bool more() const {
        return base < ncw || __any_sync(0xffffffffu, jb < je);
    }
    // the next 32 cells of the window, a lane each
    __device__ __forceinline__ void next_cells(const View &v, const SimDev &S, float thr,
                                               float thr_s) {
        const SimConst<float> &c = S.cf;
        wc = base + (threadIdx.x & 31);
        base += 32;
        jb = je = 0;
        if (wc >= ncw) return;
        const int e0 = 2 * S.win[0] + 1, e1 = 2 * S.win[1] + 1;
        const int o[3] = {wc % e0 - S.win[0], (wc / e0) % e1 - S.win[1],
                          D == 3 ? wc / (e0 * e1) - S.win[2] : 0};
        const int cc[3] = {cp & 2047, (cp >> 11) & 2047, (cp >> 22) & 1023};
        float gap2 = 0.f;
        int lin = 0, mul = 1;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            // least distance along the axis between a particle of the home
            // cell and one of this cell, wherever the two may have drifted to
            const float gap = fabsf((float)o[a]) * c.edge[a] - 2.0f * c.ext[a];
            if (gap > 0.f) gap2 += gap * gap;
            int x = cc[a] + o[a];
            x += x < 0 ? S.nc[a] : 0;
            x -= x >= S.nc[a] ? S.nc[a] : 0;
            lin += x * mul;
            mul *= S.nc[a];
            off[a] = (double)o[a] * S.edge[a];
        }
        nearcap = !(gap2 > thr_s);
        if (gap2 > thr || !SPH_IN_BOUNDS(lin >= 0 && lin < S.ncells, v.err_any)) return;
        const int gc = S.cell_off + v.morton[S.cell_off + lin];
        if (!SPH_IN_BOUNDS(gc >= S.cell_off && gc < S.cell_off + S.ncells, v.err_any)) return;
        jb = v.cell_start[gc];
        je = v.cell_start[gc + 1];
        if (!SPH_IN_BOUNDS(jb >= 0 && jb <= je && je <= v.np, v.err_any)) jb = je = 0;
    }
    // Fills the tile with the next candidates: of each 32 cells those that can
    // hold near pairs first.  Slots are named by a lane per cell, then copied
    // by a thread per slot, so that the loads of a tile are all in flight at
    // once.
    template <typename Mem>
    __device__ __forceinline__ void fill(const View &v, const SimDev &S, Mem &mem, float thr,
                                         float thr_s) {
        const double4_32a *__restrict__ P = (const double4_32a *)v.pk_pos_in;
        const int lane = threadIdx.x & 31;
        __syncthreads();   // the last tile's readers are done
        T = Tn = s_first = s_last = 0;
        while (T < kTileCap) {
            if (!__any_sync(0xffffffffu, jb < je)) {
                if (base >= ncw) break;
                next_cells(v, S, thr, thr_s);
                continue;
            }
            const int cnt = min(je - jb, kTileCap);
            const int own = nearcap ? cnt : cnt << 16;
            int incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int tot = __shfl_sync(0xffffffffu, incl, 31), tn = tot & 0xffff;
            const int at = T + (nearcap ? (incl & 0xffff) - cnt : tn + (incl >> 16) - cnt);
            const int take = max(0, min(cnt, kTileCap - at));
            if (threadIdx.x < 32)
                for (int t = 0; t < take; ++t) {
                    mem.j[at + t] = jb + t;
                    mem.c[at + t] = (unsigned char)lane;
                }
            const unsigned mine = __ballot_sync(0xffffffffu, wc == (ncw >> 1) && take > 0);
            if (mine) {
                const int src = __ffs(mine) - 1;
                s_first = __shfl_sync(0xffffffffu, jb, src);
                s_last = s_first + __shfl_sync(0xffffffffu, take, src);
                s_base = s_first - __shfl_sync(0xffffffffu, at, src);
            }
            jb += take;
            const int T1 = min(kTileCap, T + tn + (tot >> 16));
            if (tn > 0) Tn = min(kTileCap, T + tn);
            __syncthreads();
            for (int k0 = T; k0 < T1; k0 += kTileThreads) {
                const int k = k0 + (int)threadIdx.x;
                const bool ok = k < T1;
                const int cell = ok ? mem.c[k] : 0;
                const int j = ok ? mem.j[k] : 0;
                double4_32a pj = make_v4<double>(0, 0, 0, 0);
                if (ok) {
                    pj = P[j];
                    Pass::load(v, mem, k, j, pj);
                }
                double p[D];
#pragma unroll
                for (int a = 0; a < D; ++a)
                    p[a] = (a == 0 ? pj.x : (a == 1 ? pj.y : pj.z)) +
                           __shfl_sync(0xffffffffu, off[a], cell);
                if (ok) mem.put(k, p, pj.w);
            }
            T = T1;
        }
        __syncthreads();
    }
};

// One round of the home cell: its `left` (at most 2^(5 - lg)) particles from
// `first` on, lg >= S.tile_lg lanes (log2) each, tested against the whole window.
// A warp without a round (left <= 0) helps copying.
template <int D, typename Mem, typename Pass>
__device__ __forceinline__ void tile_round(const View &v, const SimDev &S, Mem &mem,
                                           TileQueue *queue, Window<D, Pass> &win, int first,
                                           int left, Pass &pass) {
    const int lane = threadIdx.x & 31;
    // thresholds of the FP32 test, 1e-6 too wide; the bodies test exactly
    const float thr = (Pass::kFar ? S.cf.thr_hi : S.cf.thr_s) * 1.000001f;
    const float thr_s = S.cf.thr_s * 1.000001f;
    const double thr_lo = Pass::kFar ? S.cf.thr_lo : fminf(S.cf.thr_lo, S.cf.thr_s);
    const bool work = left > 0;
    const int lg = max(S.tile_lg, left > 2 ? 3 : (left == 2 ? 4 : 5)), G = 1 << lg;
    const int slot = lane >> lg, l = lane & (G - 1);
    const bool live = slot < left;
    const int i = first + (live ? slot : 0);
    const double4_32a p4 = ((const double4_32a *)v.pk_pos_in)[i];
    const double pi[3] = {p4.x, p4.y, p4.z};
    const float pt[3] = {(float)pi[0], (float)pi[1], (float)pi[2]};
    pass.begin(i);
    int npairs = 0;
    bool more;
    do {
        win.fill(v, S, mem, thr, Pass::kFar ? thr_s : 0.0f);
        more = win.more();
        if (!work) continue;
        for (int k0 = 0; k0 < win.T; k0 += 32 * G) {
            const int steps = min(16, (win.T - k0 + 2 * G - 1) >> (lg + 1));
            const int sn =
                Pass::kFar ? max(0, min(steps, (win.Tn - k0 + 2 * G - 1) >> (lg + 1))) : 0;
            unsigned in, near;
            if (S.small_mask)
                tile_test<D, true>(mem, k0 + l, G, steps, sn, pt, S.cf, thr, thr_s, S.small_mask,
                                   in, near);
            else
                tile_test<D, false>(mem, k0 + l, G, steps, sn, pt, S.cf, thr, thr_s, 0, in, near);
            if (!live) in = 0u;
            const int top = k0 + l + (2 * steps - 1) * G;
            // the test reads whole steps: slots past the tile's end hold no candidate
            // (whatever an earlier tile left there, which must name no particle)
            if (top >= win.T) {
                const int past = (top - win.T) >> lg;
                in &= past < 31 ? 0xfffffffeu << past : 0u;
            }
            // a particle is not its own neighbour
            if (i >= win.s_first && i < win.s_last) {
                const int up = top - (i - win.s_base), q = up >> lg;
                if (up >= 0 && (up & (G - 1)) == 0 && q < 2 * steps) in &= ~(1u << q);
            }
            if (!Pass::kFar) near = in;
            near &= in;
            unsigned far = in & ~near;
            int drop = 0;   // candidates of the guard band that are no pairs
            // the accepted candidates, dealt out evenly through the queue
            const int own = __popc(near) | (__popc(far) << 16);
            int incl = own;
            for (int o = 1; o < G; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o, G);
                if (l >= o) incl += y;
            }
            const int tot = __shfl_sync(0xffffffffu, incl, G - 1, G);
            int pn = (incl - own) & 0xffff, pf = kTileCap - 1 - ((incl - own) >> 16);
            TileSlot *qu = queue->q[slot];
            __syncwarp();   // the last sub-tile's readers are done
            while (near) {
                const int q = top_bit(near);
                near ^= 1u << q;
                qu[pn++] = (TileSlot)(top - (q << lg));
            }
            while (far) {
                const int q = top_bit(far);
                far ^= 1u << q;
                qu[pf--] = (TileSlot)(top - (q << lg));
            }
            __syncwarp();
            const int nn = tot & 0xffff, nf = tot >> 16;
            if (l == 0) npairs += nn + nf;
            for (int t = l; t < nn; t += G)
                tile_pair<true, D>(v, S, mem, qu[t], i, pi, thr_lo, drop, pass);
            if (Pass::kFar)
                for (int t = l; t < nf; t += G)
                    tile_pair<false, D>(v, S, mem, qu[kTileCap - 1 - t], i, pi, thr_lo, drop, pass);
            __syncwarp();
            npairs -= drop;
        }
    } while (more);
    if (!work) return;
    for (int o = G >> 1; o > 0; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    pass.end(i, G, live && l == 0, npairs);
}

// ---- kernels ----

template <typename Pass> struct TileSmem {
    typename Pass::Mem mem;
    TileQueue queue[kTileRounds];
};

// Pass over the listed items, then fin(i, s, S) once per particle of the item
// with its sums written.
template <int D, typename Pass, typename Fin>
__device__ __forceinline__ void tile_pass(const View &v, Fin fin) {
    extern __shared__ __align__(16) unsigned char tile_smem[];
    TileSmem<Pass> &sm = *(TileSmem<Pass> *)tile_smem;
    const int w = threadIdx.x >> 5, items = *v.n_items;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int cell = v.item_cell[it], r0 = v.item_round[it];
        if (!SPH_IN_BOUNDS(cell >= 0 && cell < v.ncells && r0 >= 0, v.err_any)) continue;
        const int lo = v.cell_start[cell], n = v.cell_start[cell + 1] - lo;
        if (!SPH_IN_BOUNDS(lo >= 0 && n > 0 && lo + n <= v.np, v.err_any)) continue;
        const int s = v.b_sim[lo];
        const SimDev &S = v.sims[s];
        const int slots = 32 >> S.tile_lg, first = slots * (r0 + w);
        {
            Pass pass(v, S);
            Window<D, Pass> win;
            win.start(v, S, cell);
            tile_round<D>(v, S, sm.mem, sm.queue + w, win, lo + min(first, n - 1),
                          min(n - first, slots), pass);
        }
        __syncthreads();
        const int end = min(n, slots * (r0 + kTileRounds));
        for (int k = slots * r0 + threadIdx.x; k < end; k += kTileThreads) fin(lo + k, s, S);
    }
}

// 128 registers: four resident blocks of 128 threads
template <int D, int K>
__global__ void __launch_bounds__(kTileThreads, 4)
    k_tile_density(const __grid_constant__ View v, int stage) {
    tile_pass<D, TileDensity<D, K>>(v, [&](int i, int s, const SimDev &S) {
        const double4_32a f = ((const double4_32a *)v.pk_f)[i];
        const unsigned npairs = (unsigned)((const double *)v.temp)[i];
        density_finish<double, D>(v, S, i, s, stage, f.x, f.z, npairs);
        // the candidate test drops a pair whose distance is not a number
        const double4_32a p = ((const double4_32a *)v.pk_pos_in)[i];
        if (!isfinite(p.x) || !isfinite(p.y) || (D == 3 && !isfinite(p.z)))
            set_err(v.err, v.err_any, s, SPH_ENAN);
    });
}

template <int D, int K>
__global__ void __launch_bounds__(kTileThreads, 4) k_tile_heat(const __grid_constant__ View v) {
    tile_pass<D, TileHeat<D, K>>(v, [](int, int, const SimDev &) {});
}

template <int D, int K, int VH>
__global__ void __launch_bounds__(kTileThreads, 4)
    k_tile_force(const __grid_constant__ View v, int stage, int mode, int integ) {
    tile_pass<D, TileForce<D, K, VH>>(v, [&](int i, int s, const SimDev &S) {
        double vdr[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < D; ++a) vdr[a] = ((const double *)v.vdot[a])[i];
        const double udr = ((const double *)v.udot)[i];
        if (!isfinite(vdr[0]) || !isfinite(udr)) set_err(v.err, v.err_any, s, SPH_ENAN);
        if (mode != 0) integrate_stage<double, D>(v, S, i, s, stage, integ, vdr, udr);
    });
}

// One block per item up to a few waves: the number of items is known on the
// device only, and the blocks walk them.
template <typename Pass, typename F, typename... Args>
void tile_launch(F *kernel, const View &v, cudaStream_t s, Args... args) {
    constexpr size_t smem = sizeof(TileSmem<Pass>);
    static_assert(smem <= 48 * 1024, "a block's shared memory without an opt-in");
    const int grid = std::max(1, std::min(v.items_max, 64 * device_sms()));
    kernel<<<grid, kTileThreads, smem, s>>>(v, args...);
}

// Calls f with the kernel id and the dimension as constants.
template <typename F> void tile_dispatch(const View &v, int kernel, F f) {
    auto dim = [&](auto k) {
        if (v.dim == 2) f(k, std::integral_constant<int, 2>{});
        else f(k, std::integral_constant<int, 3>{});
    };
    switch (kernel) {
        case SPH_KERNEL_GAUSSIAN: dim(std::integral_constant<int, SPH_KERNEL_GAUSSIAN>{}); break;
        case SPH_KERNEL_LUCY: dim(std::integral_constant<int, SPH_KERNEL_LUCY>{}); break;
        case SPH_KERNEL_DEBRUN: dim(std::integral_constant<int, SPH_KERNEL_DEBRUN>{}); break;
        default: dim(std::integral_constant<int, SPH_KERNEL_CUBIC>{}); break;
    }
}

}  // namespace

void tile_density(const View &v, int kernel, int stage, cudaStream_t s) {
    tile_dispatch(v, kernel, [&](auto k, auto d) {
        constexpr int K = decltype(k)::value, D = decltype(d)::value;
        tile_launch<TileDensity<D, K>>(k_tile_density<D, K>, v, s, stage);
    });
}

void tile_heat(const View &v, int kernel, cudaStream_t s) {
    tile_dispatch(v, kernel, [&](auto k, auto d) {
        constexpr int K = decltype(k)::value, D = decltype(d)::value;
        tile_launch<TileHeat<D, K>>(k_tile_heat<D, K>, v, s);
    });
}

void tile_force(const View &v, int kernel, int vh, int integ, int stage, int mode,
                cudaStream_t s) {
    tile_dispatch(v, kernel, [&](auto k, auto d) {
        constexpr int K = decltype(k)::value, D = decltype(d)::value;
        auto run = [&](auto vhc) {
            constexpr int VH = decltype(vhc)::value;
            tile_launch<TileForce<D, K, VH>>(k_tile_force<D, K, VH>, v, s, stage, mode, integ);
        };
        switch (vh) {
            case 0: run(std::integral_constant<int, 0>{}); break;
            case 1: run(std::integral_constant<int, 1>{}); break;
            case 2: run(std::integral_constant<int, 2>{}); break;
            default: run(std::integral_constant<int, 3>{}); break;
        }
    });
}

}  // namespace sph
