// sph_pairs.cu -- density and heat-flux passes of one derivative evaluation,
// the thermostat reductions and the pair-set export.
//
//   k_density : rho_s, rho_l summation (self term W(0,h), no m_i:
//               properties.py:77-91), fused EOS epilogue (T from u, clamp,
//               p, pco: properties.py:38-49, spam_complete_force.py:134-152)
//   k_heat    : Fourier heat flux q_i (f_properties.py:129-130 restated)
#include <map>
#include <mutex>
#include <utility>

#include "sph_pairs.cuh"

namespace sph {

// Register caps by resident blocks of 256 threads.  A single simulation (its
// constants are kernel parameters) runs best at 6 (40 registers): density of
// a step, us, at 5 / 6 / 7 blocks 252 / 229 / 233 in 2D (199k particles) and 1625 /
// 1429 / 1446 in 3D (205k); several at 4 (391 us against 418 at 5).  3D at other sizes,
// whole step at 5 / 6: 97,336 particles 2041 / 2063, 157,464 2952 / 2977, 729,000 9822 /
// 9751, 1,331,000 17553 / 17391; at 0.6 particles per cell 125,000 593 / 641, 729,000
// 2725 / 2793.
// LIST: the pair lists (tuning.pair_scheme 2) instead of the cell windows.
// LANES: lanes per particle (for_pairs_lanes; the same bits).
template <typename R, int D, int K, bool ONE, bool LIST = false, int LANES = 1>
__device__ __forceinline__ void density_one(const View &v, int stage, int i) {
    bool active = i < v.np;
    const int ii = active ? i : v.np - 1;
    using T4 = typename V4<R>::T;
    const auto *__restrict__ P = positions<R, D>(v);
    const int s = v.b_sim[ii];
    const SimDev &S = ONE ? v.one : v.sims[s];
    if (S.cl_on || (!LIST && S.tile_on)) {   // cluster passes, cell tiles
        if (LANES == 1) return;
        active = false;
    }
    KConst<R> ks = make_kconst<R>(S, 0);
    KConst<R> kl = make_kconst<R>(S, 1);
    BAcc<R> rs, rl;
    rs.init((R)0);
    rl.init((R)0);
    unsigned cnt = 0;
    auto cell_done = [&]() {
        rs.flush();
        rl.flush();
    };
    if (LANES == 1 && !active) return;
    with_masses<R, D, (LANES > 1)>(v, s, [&](auto same) {
        const PairMass<R, D, decltype(same)::value> mass(v, ii);
        auto body = [&](int j, const auto &pj, const R *d, R rsq, auto near, auto...) {
            const Dist<R> dd = plain_dist<R>(rsq);
            const R mj = mass(j, pj);
            R w, g;
            if constexpr (decltype(near)::value) {
                kernel_wg<K, R>(ks, dd, &w, &g);
                rs.madd(mj, w);
            }
            kernel_wg<K, R>(kl, dd, &w, &g);
            rl.madd(mj, w);
            if (!LIST) ++cnt;
        };
        PairFrame<R, D> fr;
        fr.init(S);
        if constexpr (LANES > 1) {
            for_pairs_lanes<R, D, LANES, true>(v, S, fr, P, ii, P[ii], active, body,
                                                      [&](unsigned mask) {
                                                          fold_lanes<LANES>(rs, mask);
                                                          fold_lanes<LANES>(rl, mask);
                                                      });
        } else if constexpr (LIST) {
            // the entries of whole groups, less those that are no pairs
            const unsigned c = v.vl_cnt[i];
            cnt = (((c & 0xffffu) + 3) & ~3u) + (((c >> 16) + 3) & ~3u);
            for_list<R, D, true>(v, S, fr, P, i, P[i], body, cell_done, [&]() { --cnt; },
                                 [](int) { return NoRecord{}; });
        } else {
            for_pairs<R, D>(v, S, fr, P, i, P[i], body, cell_done);
        }
    });
    if constexpr (LANES > 1) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        // the epilogue by consecutive threads (lanes_block)
        constexpr int N = lanes_block<LANES> / LANES;   // particles of the block
        __shared__ double sum_s[N], sum_l[N];
        __shared__ unsigned pairs[N];
        if ((threadIdx.x & (LANES - 1)) == 0) {
            const int t = threadIdx.x / LANES;
            sum_s[t] = rs.get64();
            sum_l[t] = rl.get64();
            pairs[t] = active ? cnt : ~0u;
        }
        __syncthreads();
        const int t = threadIdx.x, p = blockIdx.x * N + t;
        if (t >= N || pairs[t] == ~0u) return;
        const int sp = v.b_sim[p];
        density_finish<R, D>(v, v.sims[sp], p, sp, stage, sum_s[t], sum_l[t], pairs[t]);
    } else {
        density_finish<R, D>(v, S, i, s, stage, rs.get64(), rl.get64(), cnt);
    }
}

// One thread per particle; PERSIST: the resident blocks of pass_grid walk
// the particles grid-stride (the same per-particle work, the same bits).
template <typename R, int D, int K, bool ONE, bool PERSIST>
__global__ void __launch_bounds__(256, ONE ? 6 : 4) k_density(const __grid_constant__ View v, int stage) {
    if constexpr (PERSIST) {
        for (int base = blockIdx.x * blockDim.x; base < v.np; base += gridDim.x * blockDim.x)
            density_one<R, D, K, ONE>(v, stage, base + threadIdx.x);
    } else {
        density_one<R, D, K, ONE>(v, stage, blockIdx.x * blockDim.x + threadIdx.x);
    }
}

// The density pass over the pair lists (mixed precision); a single
// simulation at SPH_VL_DENSITY_BLOCKS (2D) / SPH_VL_DENSITY3_BLOCKS (3D)
// resident blocks of 256 per SM, several at SPH_VL_DENSITY_MULTI_BLOCKS.
// Density of a step, us: 2D 1M particles 531 / 509 / 571 at 5 / 6 / 7 blocks;
// 3D 2M 4058 / 3997 / 4234 at 5 / 6 / 7; 24 batched simulations 263 / 256 / 260
// at 4 / 5 / 6.
#ifndef SPH_VL_DENSITY_BLOCKS
#define SPH_VL_DENSITY_BLOCKS 6
#endif
#ifndef SPH_VL_DENSITY3_BLOCKS
#define SPH_VL_DENSITY3_BLOCKS 6
#endif
#ifndef SPH_VL_DENSITY_MULTI_BLOCKS
#define SPH_VL_DENSITY_MULTI_BLOCKS 5
#endif
template <int D, int K, bool ONE>
__global__ void __launch_bounds__(256, ONE ? (D == 2 ? SPH_VL_DENSITY_BLOCKS : SPH_VL_DENSITY3_BLOCKS) : SPH_VL_DENSITY_MULTI_BLOCKS)
    k_density_vl(const __grid_constant__ View v, int stage) {
    density_one<float, D, K, ONE, true>(v, stage, blockIdx.x * blockDim.x + threadIdx.x);
}

// At most 64 registers (4 blocks of 256 per SM): 8% faster in 3D than 80.
template <typename R, int D, int K, bool ONE, bool LIST = false, int LANES = 1>
__device__ __forceinline__ void heat_one(const View &v, int i) {
    bool active = i < v.np;
    const int ii = active ? i : v.np - 1;
    using T4 = typename V4<R>::T;
    const T4 *__restrict__ P = (const T4 *)v.pk_pos_in;
    const T4 *__restrict__ F = (const T4 *)v.pk_f;
    const int s = v.b_sim[ii];
    const SimDev &S = ONE ? v.one : v.sims[s];
    if (S.cl_on || (!LIST && S.tile_on)) {   // cluster passes, cell tiles
        if (LANES == 1) return;
        active = false;
    }
    KConst<R> ks = make_kconst<R>(S, 0);
    const T4 fi = F[ii];
    const PairMass<R, D, false> mass(v, ii);
    BAcc<R> q[3];
    q[0].init(0);
    q[1].init(0);
    q[2].init(0);
    auto body = [&](int j, const T4 &pj, const R *d, R rsq, auto...) {
        R g = kernel_g<K, R, true>(ks, make_dist<R>(rsq));
        T4 fj = F[j];
        R dT = (fj.z - fi.z) + (fj.w - fi.w);
        R f = mass(j, pj) * rrcp<R>(fj.y) * dT * g;
        q[0].madd(f, d[0]);
        q[1].madd(f, d[1]);
        if (D == 3) q[2].madd(f, d[2]);
    };
    auto cell_done = [&]() {
        q[0].flush();
        q[1].flush();
        if (D == 3) q[2].flush();
    };
    if (LANES == 1 && !active) return;
    {
        PairFrame<R, D> fr;
        fr.init(S);
        // only the short kernel enters q: cells and pairs beyond its support
        // contribute exactly zero and are not visited
        fr.thr_hi = fr.thr_s;
        fr.thr_lo = fr.thr_lo < fr.thr_s ? fr.thr_lo : fr.thr_s;
        if constexpr (LANES > 1) {
            for_pairs_lanes<R, D, LANES, false>(v, S, fr, P, ii, P[ii], active, body,
                                                [&](unsigned mask) {
                                                    fold_lanes<LANES>(q[0], mask);
                                                    fold_lanes<LANES>(q[1], mask);
                                                    if (D == 3) fold_lanes<LANES>(q[2], mask);
                                                });
            if (!active || (threadIdx.x & (LANES - 1))) return;
        } else if constexpr (LIST)
            for_list<R, D, false>(v, S, fr, P, i, P[i], body, cell_done, [] {},
                                  [](int) { return NoRecord{}; });
        else for_pairs<R, D, D == 3, false>(v, S, fr, P, i, P[i], body, cell_done);
    }
    R kap = sconst<R>(S).kappa;
    R qq[3] = {kap * q[0].get(), kap * q[1].get(), kap * q[2].get()};
    R ir2 = (R)1 / (fi.y * fi.y);
    for (int a = 0; a < D; ++a) ((R *)v.q[a])[i] = qq[a];
    // {q/rho^2, rho}: the force pass's heat record, which in 3D also gives
    // it the neighbour's density
    ((T4 *)v.pk_q)[i] = make_v4<R>(qq[0] * ir2, qq[1] * ir2, qq[2] * ir2, fi.y);
}

template <typename R, int D, int K, bool ONE, bool PERSIST>
__global__ void __launch_bounds__(256, 4) k_heat(const __grid_constant__ View v) {
    if constexpr (PERSIST) {
        for (int base = blockIdx.x * blockDim.x; base < v.np; base += gridDim.x * blockDim.x)
            heat_one<R, D, K, ONE>(v, base + threadIdx.x);
    } else {
        heat_one<R, D, K, ONE>(v, blockIdx.x * blockDim.x + threadIdx.x);
    }
}

// (3D 2M particles, a step: 1230 us at 4 blocks, 1161 at 5, 1269 at 6)
template <int D, int K, bool ONE>
__global__ void __launch_bounds__(256, 5) k_heat_vl(const __grid_constant__ View v) {
    heat_one<float, D, K, ONE, true>(v, blockIdx.x * blockDim.x + threadIdx.x);
}

// The cell windows of a small launch, LANES lanes per particle: one thread per
// particle would leave most SMs without a warp (1,024 particles: 32 warps) and
// every lane with the window's whole chain.
template <typename R, int D, int K, int LANES>
__global__ void __launch_bounds__(256) k_density_lanes(const __grid_constant__ View v, int stage) {
    density_one<R, D, K, false, false, LANES>(
        v, stage, (blockIdx.x * blockDim.x + threadIdx.x) / LANES);
}
template <typename R, int D, int K, int LANES>
__global__ void __launch_bounds__(256) k_heat_lanes(const __grid_constant__ View v) {
    heat_one<R, D, K, false, false, LANES>(v, (blockIdx.x * blockDim.x + threadIdx.x) / LANES);
}

// The persistent form is instantiated for the mixed-precision passes only;
// FP64 engines launch one thread per particle whatever tuning.persistent says.
// Pair lists (v.vl_on) exist for mixed-precision engines only.
template <typename R, int D, int K, bool ONE>
void density_launch(const View &v, int stage, int block, cudaStream_t s) {
    if constexpr (std::is_same<R, float>::value) {
        if (v.vl_on) {
            k_density_vl<D, K, ONE><<<(v.np + block - 1) / block, block, 0, s>>>(v, stage);
            return;
        }
    }
    const int lanes = walk_lanes<R>(v);
    if (lanes == 32)
        k_density_lanes<R, D, K, 32><<<lanes_grid<32>(v), lanes_block<32>, 0, s>>>(v, stage);
    else if (lanes == 8)
        k_density_lanes<R, D, K, 8><<<lanes_grid<8>(v), lanes_block<8>, 0, s>>>(v, stage);
    else if (std::is_same<R, float>::value && v.persist) {
        auto *fn = k_density<R, D, K, ONE, std::is_same<R, float>::value>;
        fn<<<pass_grid(v, fn, block), block, 0, s>>>(v, stage);
    } else {
        k_density<R, D, K, ONE, false><<<(v.np + block - 1) / block, block, 0, s>>>(v, stage);
    }
}

template <typename R, int D, int K, bool ONE>
void heat_launch(const View &v, int block, cudaStream_t s) {
    if constexpr (std::is_same<R, float>::value) {
        if (v.vl_on) {
            k_heat_vl<D, K, ONE><<<(v.np + block - 1) / block, block, 0, s>>>(v);
            return;
        }
    }
    const int lanes = walk_lanes<R>(v);
    if (lanes == 32)
        k_heat_lanes<R, D, K, 32><<<lanes_grid<32>(v), lanes_block<32>, 0, s>>>(v);
    else if (lanes == 8)
        k_heat_lanes<R, D, K, 8><<<lanes_grid<8>(v), lanes_block<8>, 0, s>>>(v);
    else if (std::is_same<R, float>::value && v.persist) {
        auto *fn = k_heat<R, D, K, ONE, std::is_same<R, float>::value>;
        fn<<<pass_grid(v, fn, block), block, 0, s>>>(v);
    } else {
        k_heat<R, D, K, ONE, false><<<(v.np + block - 1) / block, block, 0, s>>>(v);
    }
}

void launch_density(const View &v, int precision, int kernel, int stage, int block,
                    cudaStream_t s) {
    if (v.np <= 0) return;
    if (precision == SPH_FP64) {
        if (v.n_tile > 0) tile_density(v, kernel, stage, s);
        if (v.n_walk == 0) return;
    }
    SPH_DISPATCH(precision, v.dim, kernel, {
        constexpr bool kOne = std::is_same<R, float>::value;
        if (v.one_sim && kOne) density_launch<R, D, K, kOne>(v, stage, block, s);
        else density_launch<R, D, K, false>(v, stage, block, s);
    });
}

void launch_heat(const View &v, int precision, int kernel, int block, cudaStream_t s) {
    if (v.np <= 0) return;
    if (precision == SPH_FP64) {
        if (v.n_tile > 0) tile_heat(v, kernel, s);
        if (v.n_walk == 0) return;
    }
    SPH_DISPATCH(precision, v.dim, kernel, {
        constexpr bool kOne = std::is_same<R, float>::value;
        if (v.one_sim && kOne) heat_launch<R, D, K, kOne>(v, block, s);
        else heat_launch<R, D, K, false>(v, block, s);
    });
}

int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

int resident_blocks(const void *kernel, int block) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, int> cache;
    std::lock_guard<std::mutex> lock(mu);
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_pair(kernel, block * 64 + dev);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int per = 0;
    const int sms = device_sms();
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, 0);
    const int cap = sms * (per > 0 ? per : 1);
    cache[key] = cap;
    return cap;
}

// ---- thermostat: per-chunk FP64 partial sums of T, then one thread per
// simulation sums its chunks in order (deterministic) ----
template <typename R>
__global__ void k_tsum_chunks(View v) {
    int c = blockIdx.x;
    int b = v.chunk_start[c], n = v.chunk_len[c];
    double x = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) x += (double)((const R *)v.temp)[b + k];
    __shared__ double sh[256];
    sh[threadIdx.x] = x;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) v.tsum_part[c] = sh[0];
}

__global__ void k_tsum_sims(View v, int nsims) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsims) return;
    SimDev &S = v.sims[s];
    if (!S.active) return;
    long long done = v.steps[s] + 1;
    v.steps[s] = done;
    if (!S.thermostat) return;
    double sum = 0.0;
    for (int c = S.chunk_first; c < S.chunk_first + S.nchunk; ++c) sum += v.tsum_part[c];
    double tav = sum / (double)S.n;
    double target = S.T0;
    if (S.ramp > 0) {
        double f = (double)done / (double)S.ramp;
        if (f > 1.0) f = 1.0;
        target = S.T0 + (S.T1 - S.T0) * f;
    }
    v.t_scale[s] = target / tav;
}

void launch_tsum(const View &v, int precision, int nsims, cudaStream_t s) {
    if (v.nchunks > 0) {
        if (precision == SPH_MIXED) k_tsum_chunks<float><<<v.nchunks, 256, 0, s>>>(v);
        else k_tsum_chunks<double><<<v.nchunks, 256, 0, s>>>(v);
    }
    k_tsum_sims<<<(nsims + 127) / 128, 128, 0, s>>>(v, nsims);
}

// ---- pair-set export (VerletList.build + NeighbourList.separations
// attributes): the same pair iteration, rows keyed by original index ----
//
// A warp per particle, a lane per window cell.  The order of a row is that of
// its partners' original indices: the warp files the partners as it finds them
// and every partner's place is the number of smaller indices in the row, counted
// by its lane from the row in L1.  16,002 particles with 58 partners each: rows
// counted in 148 us and written in 190; one thread per particle, inserting each
// partner into the row in global memory, took 2.5 and 6.4 ms (in cells 2.5 times
// as wide, which the neighbour list then asked for).
template <typename R, int D, typename F>
__device__ __forceinline__ void export_pairs(const View &v, int i, F found) {
    const SimDev &S = v.sims[v.b_sim[i]];
    using T4 = typename V4<R>::T;
    const T4 *__restrict__ P = (const T4 *)v.pk_pos_in;
    PairFrame<R, D> fr;
    fr.init(S);
    const int idi = v.b_id[i];
    for_pairs_lanes<R, D, 32, true>(
        v, S, fr, P, i, P[i], true,
        [&](int j, const T4 &, const R *, R, auto) {
            const int idj = v.b_id[j];
            if (idj > idi) found(idj, j);
        },
        [](unsigned) {});
}

// A simulation of one cell, whose window has no cells to share out: the lanes share
// the cell's particles behind i, which lie in the order of their original indices, so
// that the partners are found in the order of the row.  found(place, j); returns
// their number.  8 million pairs of 4,000 particles in device arrays: 37.9 ms by one lane
// and the count of smaller indices, 18.4 ms by a thread per particle, 8.5 ms so.
template <int D, typename F>
__device__ __forceinline__ int export_one_cell(const View &v, int i, const SimDev &S, F found) {
    const int lane = threadIdx.x & 31, je = v.cell_start[S.cell_off + 1];
    int total = 0;
    if (!SPH_IN_BOUNDS(je <= v.np, v.err_any)) return 0;
    for (int j0 = i + 1; j0 < je; j0 += 32) {
        const int j = j0 + lane;
        const bool in = j < je && exact_in_set<D>(v.xe_in, &S, i, j);
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in) found(total + __popc(mask & ((1u << lane) - 1u)), j);
        total += __popc(mask);
    }
    return total;
}

constexpr int kExportWarps = 4;

template <typename R, int D>
__global__ void __launch_bounds__(32 * kExportWarps) k_pair_rows(View v, int off, int n,
                                                                 long long *row_count) {
    const int k = blockIdx.x * kExportWarps + (threadIdx.x >> 5);
    if (k >= n) return;
    const SimDev &S = v.sims[v.b_sim[off + k]];
    int c = 0;
    if (S.ncells == 1) {
        c = export_one_cell<D>(v, off + k, S, [](int, int) {});
    } else {
        export_pairs<R, D>(v, off + k, [&](int, int) { ++c; });
        c = __reduce_add_sync(0xffffffffu, c);
    }
    if ((threadIdx.x & 31) == 0) row_count[v.b_id[off + k]] = c;
}

template <typename R, int D>
__global__ void __launch_bounds__(32 * kExportWarps)
    k_pair_write(View v, int off, int n, const long long *row_start, int2 *found,
                 long long *iap, double *drij, double *rsq, double *dv) {
    __shared__ int filed[kExportWarps];
    const int k = blockIdx.x * kExportWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= n) return;
    int &m = filed[threadIdx.x >> 5];
    const int i = off + k, idi = v.b_id[i];
    const long long base = row_start[idi];
    const SimDev &S = v.sims[v.b_sim[i]];
    auto put = [&](long long p, int idj, int j) {
        if (iap) {
            iap[2 * p] = idi;
            iap[2 * p + 1] = idj;
        }
        double r2 = 0.0;
        for (int a = 0; a < D; ++a) {
            double d = __dsub_rn(v.xe_in[a][j], v.xe_in[a][i]);
            if (d > S.half_L[a]) d = __dsub_rn(d, S.L[a]);
            if (d < -S.half_L[a]) d = __dadd_rn(d, S.L[a]);
            double sq = __dmul_rn(d, d);
            r2 = (a == 0) ? sq : __dadd_rn(r2, sq);
            if (drij) drij[p * D + a] = d;
            if (dv) dv[p * D + a] = __dsub_rn(v.ve_in[a][j], v.ve_in[a][i]);
        }
        if (rsq) rsq[p] = r2;
    };
    if (S.ncells == 1) {
        export_one_cell<D>(v, i, S, [&](int e, int j) { put(base + e, v.b_id[j], j); });
        return;
    }
    int2 *row = found + base;
    if (lane == 0) m = 0;
    __syncwarp();
    export_pairs<R, D>(v, i, [&](int idj, int j) { row[atomicAdd(&m, 1)] = make_int2(idj, j); });
    __syncwarp();
    const int total = m;
    for (int e = lane; e < total; e += 32) {
        const int2 mine = row[e];
        int rank = 0;
        for (int t = 0; t < total; ++t) rank += row[t].x < mine.x ? 1 : 0;
        put(base + rank, mine.x, mine.y);
    }
}

#define SPH_EXPORT(FN, ...)                                                              \
    do {                                                                                 \
        const int nb = (n + kExportWarps - 1) / kExportWarps, nt = 32 * kExportWarps;    \
        if (precision == SPH_MIXED) {                                                    \
            if (v.dim == 2) FN<float, 2><<<nb, nt, 0, s>>>(v, sim_off, n, __VA_ARGS__);  \
            else FN<float, 3><<<nb, nt, 0, s>>>(v, sim_off, n, __VA_ARGS__);             \
        } else {                                                                         \
            if (v.dim == 2) FN<double, 2><<<nb, nt, 0, s>>>(v, sim_off, n, __VA_ARGS__); \
            else FN<double, 3><<<nb, nt, 0, s>>>(v, sim_off, n, __VA_ARGS__);            \
        }                                                                                \
    } while (0)

void launch_pair_rows(const View &v, int precision, int sim_off, int n, long long *row_count,
                      cudaStream_t s) {
    if (n <= 0) return;
    SPH_EXPORT(k_pair_rows, row_count);
}

void launch_pair_write(const View &v, int precision, int sim_off, int n,
                       const long long *row_start, int2 *found, long long *iap, double *drij,
                       double *rsq, double *dv, cudaStream_t s) {
    if (n <= 0) return;
    SPH_EXPORT(k_pair_write, row_start, found, iap, drij, rsq, dv);
}
#undef SPH_EXPORT

// Exclusive scan of n + 1 int64 entries in place (export path only): one block,
// eight entries a thread and one barrier per 8,192.  The sums of a round lie in one of
// two buffers: a warp that writes a buffer again, two rounds later, has passed the
// barrier in between, which every reader of its old content reached after reading.
constexpr int kScan64Per = 8;
__global__ void __launch_bounds__(1024) k_scan64(long long *data, int n) {
    __shared__ long long warp_sum[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long carry = 0;
    for (int base = 0, round = 0; base <= n; base += 1024 * kScan64Per, round ^= 1) {
        const int i0 = base + threadIdx.x * kScan64Per;
        long long x[kScan64Per], sum = 0;
#pragma unroll
        for (int t = 0; t < kScan64Per; ++t) {
            x[t] = i0 + t <= n ? data[i0 + t] : 0;
            sum += x[t];
        }
        long long incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sum[round][w] = incl;
        __syncthreads();
        // every warp scans the warps' sums; the other round's are still read
        long long ws = warp_sum[round][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += y;
        }
        const long long before = __shfl_sync(0xffffffffu, ws, w > 0 ? w - 1 : 0);
        long long at = carry + (w > 0 ? before : 0) + incl - sum;
#pragma unroll
        for (int t = 0; t < kScan64Per; ++t) {
            if (i0 + t <= n) data[i0 + t] = at;
            at += x[t];
        }
        carry += __shfl_sync(0xffffffffu, ws, 31);
    }
}

void launch_scan64(long long *data, int n, cudaStream_t s) {
    k_scan64<<<1, 1024, 0, s>>>(data, n);
}

}  // namespace sph
