// sph_pairs.cuh -- shared pieces of the pair passes: the pair iteration
// (cell windows, culling, FP32 fast test with exact FP64 fallback), the
// accumulation helpers and the precision/dimension/kernel dispatch.
//
// Every pass is a gather: thread i sums over all neighbours j in the 3^dim
// cells around its own cell, so each unordered pair is evaluated from both
// sides and no atomics touch particle data.  Positions are cell-local
// (relative to the particle's cell centre), which keeps FP32 differences
// accurate; the pair-set test runs on those FP32 distances with a
// guard band and falls back to the reference's FP64 test for pairs inside
// the band, so the pair set is bit-exact.
#pragma once

#include <type_traits>

#include "sph_device.cuh"

namespace sph {

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }

// 1/x for the EOS: FP64 division in FP64 mode; in mixed mode an FP32
// reciprocal refined by one FP64 Newton step (relative error ~1e-14), which
// spares the narrow FP64 pipe a full division per particle.
template <typename R> __device__ __forceinline__ double recip64(double x);
template <> __device__ __forceinline__ double recip64<double>(double x) { return 1.0 / x; }
template <> __device__ __forceinline__ double recip64<float>(double x) {
    double r = (double)__frcp_rn((float)x);
    return r * fma(-x, r, 2.0);
}
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }

template <typename R, int D>
struct PairFrame {
    R thr_lo, thr_hi, thr_s;
    R edge[3], L[3], hL[3];
    R edge_lo[3];   // FP32: the part of the cell edge that (float)edge misses
    R ext[3];       // half extent of a cell including the allowed drift
    int small_mask;
    __device__ __forceinline__ void init(const SimDev &S) {
        const SimConst<R> &c = sconst<R>(S);
        thr_lo = c.thr_lo;
        thr_hi = c.thr_hi;
        thr_s = c.thr_s;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            edge[a] = c.edge[a];
            edge_lo[a] = c.edge_lo[a];
            L[a] = c.L[a];
            hL[a] = c.hL[a];
            ext[a] = c.ext[a];
        }
        small_mask = S.small_mask;
    }
    __device__ __forceinline__ void min_image(R *d) const {
        if (small_mask) {
#pragma unroll
            for (int a = 0; a < D; ++a)
                if (small_mask & (1 << a)) {
                    if (d[a] > hL[a]) d[a] -= L[a];
                    if (d[a] < -hL[a]) d[a] += L[a];
                }
        }
    }
};

// max(|c| - ext, 0): distance along one axis from particle i to a cell whose
// centre sits at c relative to i
template <typename R> __device__ __forceinline__ R fmaxf_(R c, R ext) {
    R a = (c < (R)0 ? -c : c) - ext;
    return a > (R)0 ? a : (R)0;
}

// One window cell of particle i (linear cell lin, offset (ox, oy, oz)): body for
// every pair of i in it, in cell order.  near_cell: the cell may hold pairs
// within the short support.  Returns whether the cell was scanned.
template <typename R, int D, bool PF, bool SELF, typename T4, typename F>
__device__ __forceinline__ bool pair_cell(const View &v, const SimDev &S,
                                          const PairFrame<R, D> &fr, const T4 *__restrict__ P,
                                          int i, const T4 &pi, const int *mort, int lin, int ox,
                                          int oy, int oz, bool near_cell, F &body) {
    if (!SPH_IN_BOUNDS(lin >= 0 && lin < S.ncells, v.err_any)) return false;
    const int gc = S.cell_off + mort[lin];
    if (!SPH_IN_BOUNDS(gc >= S.cell_off && gc < S.cell_off + S.ncells, v.err_any)) return false;
    // offset of the window cell's frame from particle i; in FP32
    // the cell edge is a hi/lo pair, so that the offset carries one
    // rounding instead of the edge's rounding times the cell count
    R ox_ = (R)ox * fr.edge[0] - pi.x;
    R oy_ = (R)oy * fr.edge[1] - pi.y;
    R oz_ = (R)0;
    if constexpr (D == 3) oz_ = (R)oz * fr.edge[2] - pi.z;
    if constexpr (std::is_same<R, float>::value) {
        ox_ = __fmaf_rn((R)ox, fr.edge_lo[0], ox_);
        oy_ = __fmaf_rn((R)oy, fr.edge_lo[1], oy_);
        if (D == 3) oz_ = __fmaf_rn((R)oz, fr.edge_lo[2], oz_);
    }
    const int jb = v.cell_start[gc], je = v.cell_start[gc + 1];
    if (!SPH_IN_BOUNDS(jb >= 0 && jb <= je && je <= v.np, v.err_any)) return false;
    auto scan = [&](auto near, auto self, auto mi) {
        T4 pn;
        if (PF) pn = P[jb < je ? jb : i];
        for (int j = jb; j < je; ++j) {
            T4 pj;
            if (PF) {
                pj = pn;
                if (j + 1 < je) pn = P[j + 1];
            }
            if (decltype(self)::value && j == i) continue;
            if (!PF) pj = P[j];
            R d[3];
            d[0] = pj.x + ox_;
            d[1] = pj.y + oy_;
            d[2] = (R)0;
            if constexpr (D == 3) d[2] = pj.z + oz_;
            if constexpr (decltype(mi)::value) fr.min_image(d);
            R rsq = fma_(d[1], d[1], d[0] * d[0]);
            if (D == 3) rsq = fma_(d[2], d[2], rsq);
            if (rsq > fr.thr_hi) continue;
            if (rsq >= fr.thr_lo && !exact_in_set<D>(v.xe_in, &S, i, j)) continue;
            body(j, pj, d, rsq, near);
        }
    };
    // the minimum image applies only on single-cell axes: the scan
    // is compiled with and without it (4.7% of the 2D density
    // pass, which otherwise tested small_mask per candidate)
    if (fr.small_mask) {
        if (SELF && ox == 0 && oy == 0 && oz == 0)
            scan(std::true_type{}, std::true_type{}, std::true_type{});
        else if (__any_sync(__activemask(), near_cell))
            scan(std::true_type{}, std::false_type{}, std::true_type{});
        else
            scan(std::false_type{}, std::false_type{}, std::true_type{});
    } else {
        if (SELF && ox == 0 && oy == 0 && oz == 0)
            scan(std::true_type{}, std::true_type{}, std::false_type{});
        else if (__any_sync(__activemask(), near_cell))
            scan(std::true_type{}, std::false_type{}, std::false_type{});
        else
            scan(std::false_type{}, std::false_type{}, std::false_type{});
    }
    return true;
}

// Iterates the pair set of particle i.  body(j, pj, d[3], rsq, near) is called
// for every j != i that passes the exact pair test, in a fixed order: neighbour
// cells in raster order (z, y, x) of their offset from i's cell, particles in
// cell order.  The order depends only on i's cell, never on which particles
// share a warp or a launch, so every particle sums its pairs identically
// whether its simulation runs alone or in a batch.
//
// Cells are (cutoff + skin)/W wide and the window spans +-W cells per axis;
// a cell whose box (grown by the allowed drift) lies beyond the cutoff from
// particle i is skipped before any of its particles is loaded.
//
// near is std::true_type unless the cell lies beyond the short kernel's
// support from every lane of the warp that visits it (a warp-uniform choice,
// so the two loop bodies never diverge); with std::false_type the body may
// drop every short-kernel term, which is exactly zero there.
//
// PF: load the next candidate's position before testing the current one
// (measured: 4-7% faster for the 3D heat and force passes, slower for the
// 2D passes and for density, where more warps already hide the latency).
//
// SELF: skip j == i, which only the home cell (offset 0) can hold, so only its
// loop tests for it.  A pass whose pair terms all carry the separation d
// (force, heat flux) may leave the test out: for j == i, d = 0 exactly and
// every kernel's gradient factor is finite at r = 0, so the terms add +0 and
// the sums keep their bits.
template <typename R, int D, bool PF = false, bool SELF = true, typename T4, typename F,
          typename G>
__device__ __forceinline__ void for_pairs(const View &v, const SimDev &S,
                                          const PairFrame<R, D> &fr, const T4 *__restrict__ P,
                                          int i, const T4 &pi, F body, G cell_done) {
    const int cp = v.cell_xyz[v.cell_b[i]];
    const int c0 = cp & 2047, c1 = (cp >> 11) & 2047, c2 = (cp >> 22) & 1023;
    const int w0 = S.win[0], w1 = S.win[1], w2 = D == 3 ? S.win[2] : 0;
    const int n0 = S.nc[0], n1 = S.nc[1], n2 = S.nc[2];
    const int *mort = v.morton + S.cell_off;
    for (int oz = -w2; oz <= w2; ++oz) {
        R dz = (R)0;
        int z = 0;
        if constexpr (D == 3) {
            dz = fmaxf_((R)oz * fr.edge[2] - pi.z, fr.ext[2]);
            z = c2 + oz;
            z += (z < 0) ? n2 : 0;
            z -= (z >= n2) ? n2 : 0;
        }
        for (int oy = -w1; oy <= w1; ++oy) {
            R dy = fmaxf_((R)oy * fr.edge[1] - pi.y, fr.ext[1]);
            R dyz = fma_(dz, dz, dy * dy);
            if (dyz > fr.thr_hi) continue;
            int y = c1 + oy;
            y += (y < 0) ? n1 : 0;
            y -= (y >= n1) ? n1 : 0;
            const int row = (z * n1 + y) * n0;
            for (int ox = -w0; ox <= w0; ++ox) {
                R dx = fmaxf_((R)ox * fr.edge[0] - pi.x, fr.ext[0]);
                const R dxyz = fma_(dx, dx, dyz);
                if (dxyz > fr.thr_hi) continue;
                int x = c0 + ox;
                x += (x < 0) ? n0 : 0;
                x -= (x >= n0) ? n0 : 0;
                if (pair_cell<R, D, PF, SELF>(v, S, fr, P, i, pi, mort, row + x, ox, oy, oz,
                                              dxyz < fr.thr_s, body))
                    cell_done();
            }
        }
    }
}

// for_pairs with G lanes per particle (G = 8 or 32 consecutive lanes, all of
// the warp's lanes calling): lane l scans the window cells l, l + G, ... and
// fold(mask) then adds the G cells' blocked sums in raster order, mask holding
// the lanes whose cell was scanned.  The terms of a cell are summed by one
// lane and the cells folded in for_pairs' order, so the sums carry for_pairs'
// bits: the launch's size may choose between the two.
template <typename R, int D, int G, bool SELF, typename T4, typename F, typename H>
__device__ __forceinline__ void for_pairs_lanes(const View &v, const SimDev &S,
                                                const PairFrame<R, D> &fr,
                                                const T4 *__restrict__ P, int i, const T4 &pi,
                                                bool active, F body, H fold) {
    const int lane = threadIdx.x & 31, l = lane & (G - 1);
    const int cp = v.cell_xyz[v.cell_b[i]];
    const int c0 = cp & 2047, c1 = (cp >> 11) & 2047, c2 = (cp >> 22) & 1023;
    const int w0 = S.win[0], w1 = S.win[1], w2 = D == 3 ? S.win[2] : 0;
    const int e0 = 2 * w0 + 1, e1 = 2 * w1 + 1;
    const int n0 = S.nc[0], n1 = S.nc[1], n2 = S.nc[2];
    const int *mort = v.morton + S.cell_off;
    const int ncw = active ? e0 * e1 * (2 * w2 + 1) : 0;
    // the particles of a warp may belong to simulations with other windows
    const int rounds = __reduce_max_sync(0xffffffffu, (ncw + G - 1) / G);
    for (int r = 0; r < rounds; ++r) {
        const int c = r * G + l;
        bool scanned = false;
        if (c < ncw) {
            const int row = c / e0, ox = c - row * e0 - w0;
            const int oy = (D == 3 ? row % e1 : row) - w1, oz = D == 3 ? row / e1 - w2 : 0;
            const R dx = fmaxf_((R)ox * fr.edge[0] - pi.x, fr.ext[0]);
            const R dy = fmaxf_((R)oy * fr.edge[1] - pi.y, fr.ext[1]);
            R dz = (R)0;
            if constexpr (D == 3) dz = fmaxf_((R)oz * fr.edge[2] - pi.z, fr.ext[2]);
            const R dyz = fma_(dz, dz, dy * dy);
            const R dxyz = fma_(dx, dx, dyz);
            if (!(dyz > fr.thr_hi) && !(dxyz > fr.thr_hi)) {
                int x = c0 + ox, y = c1 + oy, z = D == 3 ? c2 + oz : 0;
                x += x < 0 ? n0 : 0;
                x -= x >= n0 ? n0 : 0;
                y += y < 0 ? n1 : 0;
                y -= y >= n1 ? n1 : 0;
                if (D == 3) {
                    z += z < 0 ? n2 : 0;
                    z -= z >= n2 ? n2 : 0;
                }
                scanned = pair_cell<R, D, false, SELF>(v, S, fr, P, i, pi, mort,
                                                       (z * n1 + y) * n0 + x, ox, oy, oz,
                                                       dxyz < fr.thr_s, body);
            }
        }
        fold((__ballot_sync(0xffffffffu, scanned) >> (lane & ~(G - 1))) &
             (G == 32 ? 0xffffffffu : (1u << G) - 1u));
    }
}

// Adds the G lanes' blocks of a sum in lane order, on every lane: the lanes in
// mask as BAcc::flush would.
template <int G, typename R>
__device__ __forceinline__ void fold_lanes(BAcc<R> &a, unsigned mask) {
#pragma unroll 8
    for (int c = 0; c < G; ++c) {
        const R x = __shfl_sync(0xffffffffu, a.part, c, G);
        if (mask & (1u << c)) a.total.add(x);
    }
    a.part = (R)0;
}

// Window offset k - 3 of a list entry's 3-bit field k, as an exact float:
// 2^23 + k built from its bits, minus 2^23 + 3.
__device__ __forceinline__ float vl_offset(unsigned k) {
    return __fsub_rn(__int_as_float(0x4B000000 | k), 8388611.0f);
}

// Iterates the pair set of particle i from its pair list (tuning.pair_scheme
// 2; FP32): the near entries, then with FAR the far ones, each in the
// order of the build (window cells in raster order, particles in cell
// order), with the same fast test and exact FP64 fallback as for_pairs.
// body(j, pj, d, rsq, near) as in for_pairs; cell_done() folds the blocked
// sums every 16 entries.  A far entry lay beyond the short support plus the
// skin at the build, so while the lists hold it stays beyond the support:
// the far bodies drop the short-kernel terms, which are exactly zero.
//
// Entries come four to a 16-byte group (near groups from row 0 up, far
// groups from row cap/4 - 1 down, a far group's entries from its last slot
// back); the next group is loaded before the current one is evaluated, so
// that the stream of entries from HBM overlaps the arithmetic.
//
// The separation is rebuilt from the entry's window offset: d = (p_j - p_i)
// + o e + o e_lo with the cell edge as a hi/lo pair, every rounding at the
// magnitude of d.
//
// Every run fills whole groups: the build ends it with entries that name the
// particle itself three window cells away on every axis, which no pair within
// the cutoff is, so that the walk tests no entry's place.  skip() is called for
// every entry that is no pair, these among them.
//
// What the body needs of j beside its position record, load(j) fetches together
// with that record, ahead of the pair test, and body gets it as its last
// argument: most entries are pairs, so the loads are rarely wasted, and they do
// not wait for the test.
template <typename R, int D, bool FAR, typename T4, typename F, typename G, typename H,
          typename L>
__device__ __forceinline__ void for_list(const View &v, const SimDev &S,
                                         const PairFrame<R, D> &fr, const T4 *__restrict__ P,
                                         int i, const T4 &pi, F body, G cell_done, H skip, L load) {
    static_assert(std::is_same<R, float>::value, "pair lists: mixed precision");
    constexpr int kBits = vl_index_bits(D);
    const unsigned cnt = v.vl_cnt[i];
    const int nn = (int)(cnt & 0xffffu), nf = (int)(cnt >> 16);
    const long long st = v.vl_stride;
    auto one = [&](int code, auto near) {
        const int j = code & vl_index_mask(D);
        if (!SPH_IN_BOUNDS(j >= 0 && j < v.np, v.err_any)) return;
        const unsigned t = (unsigned)code >> kBits;
        const float fx = vl_offset(t & 7u);
        const float fy = vl_offset(D == 3 ? (t >> 3) & 7u : t >> 3);
        const T4 pj = P[j];
        const auto rec = load(j);
        R d[3];
        d[0] = __fmaf_rn(fx, fr.edge_lo[0], __fmaf_rn(fx, fr.edge[0], __fsub_rn(pj.x, pi.x)));
        d[1] = __fmaf_rn(fy, fr.edge_lo[1], __fmaf_rn(fy, fr.edge[1], __fsub_rn(pj.y, pi.y)));
        d[2] = (R)0;
        R rsq = fma_(d[1], d[1], d[0] * d[0]);
        if constexpr (D == 3) {
            const float fz = vl_offset(t >> 6);
            d[2] = __fmaf_rn(fz, fr.edge_lo[2], __fmaf_rn(fz, fr.edge[2], __fsub_rn(pj.z, pi.z)));
            rsq = fma_(d[2], d[2], rsq);
        }
        // one branch for the guard band and everything beyond it
        if (rsq >= fr.thr_lo && (rsq > fr.thr_hi || !exact_in_set<D>(v.xe_in, &S, i, j))) {
            skip();
            return;
        }
        body(j, pj, d, rsq, near, rec);
    };
    // the groups from pointer g, stepping `dir` rows each; slots in order
    // 0..3 (near) or 3..0 (far).  Measured on the 2D fluid: a lookahead of
    // one group is enough (two, or the group's four records loaded ahead of
    // their tests, were 3-6% slower: more registers)
    auto walk = [&](const int4 *g, long long dir, int n, auto near, auto rev) {
        const int ng = (n + 3) >> 2;
        int4 cur = ng > 0 ? *g : make_int4(0, 0, 0, 0);
        for (int k = 0; k < ng; ++k) {
            const int4 nxt = k + 1 < ng ? g[(k + 1) * dir] : cur;
            if constexpr (decltype(rev)::value) {
                one(cur.w, near);
                one(cur.z, near);
                one(cur.y, near);
                one(cur.x, near);
            } else {
                one(cur.x, near);
                one(cur.y, near);
                one(cur.z, near);
                one(cur.w, near);
            }
            if ((k & 3) == 3) cell_done();
            cur = nxt;
        }
        cell_done();
    };
    const int4 *E = (const int4 *)v.vl_ent + i;
    walk(E, st, nn, std::true_type{}, std::false_type{});
    if constexpr (FAR)
        walk(E + (long long)((v.vl_cap >> 2) - 1) * st, -st, nf, std::false_type{},
             std::true_type{});
}

// load() of a list pass that needs the position records alone.
struct NoRecord {};

// Blocks of a pair-pass launch: one thread per particle, or with v.persist
// only the blocks the device holds at once (SMs x resident blocks of this
// kernel at this block size, cached per kernel), which then walk the
// particles grid-stride.
int resident_blocks(const void *kernel, int block);
template <typename F> inline int pass_grid(const View &v, F *kernel, int block) {
    const int nb = (v.np + block - 1) / block;
    if (!v.persist) return nb;
    const int cap = resident_blocks((const void *)kernel, block);
    return nb < cap ? nb : cap;
}

// Lanes per particle of the cell-window passes, by the launch (the bits do not depend
// on it).  A small launch is bound by the latency of one thread's window, which lanes
// share; a larger one pays for lanes without a cell and for the fold.  Step, us, with
// 1 / 8 / 32 lanes, mixed precision at nine (2D) or 12 (3D, with heat flux) particles per
// cell: 2D 1,024 particles 340 / 111 / 73, 4,096 325 / 108 / 107, 16,384 352 / 185 / 247,
// 32,761 350 / 259 / 432, 65,536 375 / 432 / 816; 3D 2,197 2122 / 615 / 274, 8,000 2124 /
// 608 / 675, 32,768 2354 / 1923 / 2505, 64,000 2377 / 3041 / 4484.  With fewer particles
// in a cell the line is earlier: 2D at 0.25 28,900 115 / 106, 36,100 117 / 125, at 2.25 40,000
// 197 / 168; 3D at 0.27 27,000 407 / 370, 39,304 424 / 529, at 1.33 27,000 577 / 458, 39,304
// 596 / 676.  Windows of few cells (axes of a single cell) leave lanes idle, hence the
// limits on lane_load: one cell, which has nothing to share, 40 x 1,000 particles in 3D 2408 /
// 7515, 64 particles 90 / 95 / 106; five cells 3D 20,000 1672 / 1627, 40,000 1739 / 2555,
// 2D 20,000 200 / 167; 25 cells 3D 20,250 1592 / 1200, 36,000 1639 / 1757.
// FP64, whose pipe fills sooner (simulations too sparse for cell tiles): 2D at 0.25 1,024
// 221 / 112 / 76, 2,704 239 / 121 / 170, 4,096 243 / 120 / 202, 10,000 244 / 288 / 435; at
// 1.56 665 / 251 / 130, 676 / 259 / 311, 672 / 251 / 375, 700 / 622 / 793; 3D at 0.27 512
// 997 / 501 / 232, 2,197 1136 / 532 / 683, 4,096 1041 / 519 / 1090, 15,625 1166 / 1920 / 3584.
template <typename R> inline int walk_lanes(const View &v) {
    if (v.lane_load[0] >= 8LL * v.np) return 1;   // windows of one cell
    if (sizeof(R) == 8) return v.np <= 1536 ? 32 : (v.np <= 4096 ? 8 : 1);
    const bool dense = v.np >= (v.dim == 2 ? 2LL : 4LL) * v.ncells;
    if (v.np <= 4096 && v.lane_load[1] <= 65536) return 32;
    if (v.np <= (dense ? 40960 : 28672) && v.lane_load[0] <= (v.dim == 2 ? 52428 : 41943)) return 8;
    return 1;
}
// Threads per block, and blocks, of the passes with LANES lanes per particle.  Their
// epilogues (FP64, an instruction of which costs the pipe the same for one lane of a
// warp as for all) are done by the block's first threads, one per particle, from
// shared memory.  Density + force of a step, us, epilogue by each particle's first
// lane / so in blocks of 128 / of 256: 2D 32 lanes 4k particles 102.4 / 85.5 / 88.1,
// 1k 70.2 / 68.4 / 68.6; 8 lanes 9k 106.0 / 105.4 / 102.6, 22k 179.8 / 173.1 / 171.1; 3D
// with heat 32 lanes 1.7k 241 / 243 / 248, 8 lanes 16k 1010 / 1007 / 990.
template <int LANES> constexpr int lanes_block = LANES == 32 ? 128 : 256;
template <int LANES> inline int lanes_grid(const View &v) {
    return (int)(((long long)v.np * LANES + lanes_block<LANES> - 1) / lanes_block<LANES>);
}

// Warp-aggregated per-simulation counter update.
__device__ __forceinline__ void add_pair_count(unsigned long long *cnt, int s, unsigned c) {
    const unsigned grp = __match_any_sync(__activemask(), s);
    // a warp's counts sum below 2^32: a particle has fewer than 2^26 neighbours
    const unsigned tot = __reduce_add_sync(grp, c);
    if ((threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&cnt[s], (unsigned long long)tot);
}

// Epilogue of the density passes: the equation of state of particle i from
// the sums of its pairs' m W / sigma, and the records that the heat and force
// passes read.
template <typename R, int D>
__device__ __forceinline__ void density_finish(const View &v, const SimDev &S, int i, int s,
                                               int stage, double sum_s, double sum_l,
                                               unsigned cnt) {
    using T4 = typename V4<R>::T;
    // EOS in FP64 from the compensated sums plus the FP64 self term
    // (properties.py:77-78): the temperature T = (u + a rho)/k_B cancels
    // strongly, so rho enters it with the bits the FP32 sum carried in its
    // compensation.  p/rho^2 = k_B T / (rho (1 - b rho)); the cohesive factor
    // pco/rho_l^2 is exactly -a and needs no storage.
    double rho = S.ws0 + S.sig_s * sum_s;
    double rhol = S.wl0 + S.sig_l * sum_l;
    double T = (v.ue_in[i] + S.a * rho) * S.inv_kb;
    if (T < 0.0) T = 0.0;
    double den = rho * (1.0 - S.b * rho);
    double fs = S.kb * T * recip64<R>(den);
    double p = fs * rho * rho;
    double pco = -S.a * rhol * rhol;
    R Th = (R)T;
    ((R *)v.rho)[i] = (R)rho;
    ((R *)v.rho_l)[i] = (R)rhol;
    ((R *)v.temp)[i] = Th;
    ((R *)v.pres)[i] = (R)p;
    ((R *)v.pco)[i] = (R)pco;
    if (stage == 0) {
        ((R *)v.rho0)[i] = (R)rho;
        ((R *)v.pres0)[i] = (R)p;
        ((R *)v.pco0)[i] = (R)pco;
    }
    // {p/rho^2, rho, T_hi, T_lo}: T as a hi/lo pair so that T_j - T_i in the
    // heat pass does not lose the low bits
    ((T4 *)v.pk_f)[i] = make_v4<R>((R)fs, (R)rho, Th, (R)(T - (double)Th));
    // what the force pass reads of a neighbour beside its packed record
    if constexpr (flat2<R, D>) {
        ((float2 *)v.pk_fv)[i] = make_float2((float)fs, (float)rho);
    } else {
        const T4 vi = ((const T4 *)v.pk_vel_in)[i];
        ((T4 *)v.pk_fv)[i] = D == 2 ? make_v4<R>(vi.x, vi.y, (R)fs, (R)rho)
                                    : make_v4<R>(vi.x, vi.y, vi.z, (R)fs);
    }
    if (!isfinite((R)p) || !isfinite((R)rho) || !isfinite((R)rhol))
        set_err(v.err, v.err_any, s, SPH_ENAN);
    // the pair set of one evaluation: counted at the step's first one only
    // (the counters are cleared once per step)
    if (stage == 0) add_pair_count(v.pair_count, s, cnt);
}

// ---- dispatch ----
#define SPH_DISPATCH(PREC, DIM, KERN, ...)                                       \
    do {                                                                          \
        if (PREC == SPH_MIXED) {                                                  \
            using R = float;                                                      \
            if (DIM == 2) { constexpr int D = 2; SPH_DISPATCH_K(KERN, __VA_ARGS__); }    \
            else { constexpr int D = 3; SPH_DISPATCH_K(KERN, __VA_ARGS__); }             \
        } else {                                                                  \
            using R = double;                                                     \
            if (DIM == 2) { constexpr int D = 2; SPH_DISPATCH_K(KERN, __VA_ARGS__); }    \
            else { constexpr int D = 3; SPH_DISPATCH_K(KERN, __VA_ARGS__); }             \
        }                                                                         \
    } while (0)
#define SPH_DISPATCH_K(KERN, ...)                                                \
    switch (KERN) {                                                               \
        case SPH_KERNEL_GAUSSIAN: { constexpr int K = SPH_KERNEL_GAUSSIAN; __VA_ARGS__; break; } \
        case SPH_KERNEL_LUCY: { constexpr int K = SPH_KERNEL_LUCY; __VA_ARGS__; break; }         \
        case SPH_KERNEL_DEBRUN: { constexpr int K = SPH_KERNEL_DEBRUN; __VA_ARGS__; break; }     \
        default: { constexpr int K = SPH_KERNEL_CUBIC; __VA_ARGS__; break; }                     \
    }

}  // namespace sph
