// sph_splat.cu -- headless SPH splash rendering of particles onto a pixel
// grid (interpolate.splash_map_2d / splash_map_3d, interpolate.py:39-149),
// replacing the GL path of SmoothParticleView.render_density
// (pview.py:483-519) with a device buffer.
//
// Each particle adds a_i m_i / rho_i W(|r_i - g|, h_i) to every pixel g of
// its pixel box [floor((r - cutoff - min)/res), floor((r + cutoff - min)/res))
// -- upper end excluded, as range() does in the reference -- whose
// minimum-imaged distance is below the cutoff.  Pixel indices wrap
// periodically; the minimum image acts on x and y with the box maxima
// (neighbours.minimum_image(dr, xmax, ymax)).  W is the 2D Lucy kernel
// (spkernel.lucy_w, spkernel.py:54-63) or, for the 3D map of particles onto
// the plane z, the 3D Lucy kernel.  FP64 throughout; contributions are added
// with atomics, so the last bits of a pixel may depend on arrival order.
#include <algorithm>
#include <cmath>

#include "sph_device.cuh"

namespace {

__device__ __forceinline__ double min_image(double d, double L) {
    if (d > L / 2.) d = d - L;
    if (d < -L / 2.) d = d + L;
    return d;
}

struct SplatArgs {
    int n, cols, nx, ny, dim3;
    int per, own;   // particles of a warp; most pixels that a lane draws by itself
    const double *r, *m, *rho, *a, *h, *x, *y;
    double z, xmin, xmax, ymin, ymax, cutoff;
    double *Z;
};

// A particle's pixel box and weights, on the lane that prepares it.
struct Splat {
    double rx, ry, dz2, coef, inv_h;
    int xa, ya, w, hgt;   // first pixel, box extents (0: nothing to draw)
};

__device__ __forceinline__ Splat splat_prepare(const SplatArgs &A, int i, double res) {
    Splat s;
    const double *r = A.r + (size_t)i * A.cols;
    s.rx = r[0];
    s.ry = r[1];
    const double dz = A.dim3 ? r[2] - A.z : 0.0;
    s.dz2 = dz * dz;
    s.xa = (int)floor((s.rx - A.cutoff - A.xmin) / res);
    s.ya = (int)floor((s.ry - A.cutoff - A.ymin) / res);
    const int xb = (int)floor((s.rx + A.cutoff - A.xmin) / res);
    const int yb = (int)floor((s.ry + A.cutoff - A.ymin) / res);
    // indices wrap once: of a box wider than the grid's three images only the
    // pixels in range are drawn, so it may end there
    s.xa = max(s.xa, -A.nx);
    s.ya = max(s.ya, -A.ny);
    s.w = max(0, min(xb, 2 * A.nx) - s.xa);
    s.hgt = max(0, min(yb, 2 * A.ny) - s.ya);
    if (A.dim3 && dz > A.cutoff) s.w = 0;
    const double pi = 3.14159265358979323846;
    const double wgt = A.a[i] * A.m[i] / A.rho[i], h = A.h[i];
    // a smoothing length that is not positive draws zeros (wgt 0), and so does one too
    // small for its powers, off the particle itself (0 times a finite norm)
    const double norm = A.dim3 ? 105.0 / (pi * 16.0 * (h * h * h)) : 5.0 / (pi * h * h);
    s.inv_h = h > 0.0 ? 1.0 / h : 0.0;
    s.coef = wgt * (h > 0.0 ? fmin(norm, 1e300) : 0.0);
    return s;
}

__device__ __forceinline__ int wrap_once(int k, int n) {
    if (k >= n) k -= n;
    if (k < 0) k += n;
    return k;
}

// d less or greater than L/2, decided by the high words but for ties: a compare
// costs the FP64 pipe as much as an addition
__device__ __forceinline__ double fast_image(double d, double L) {
    const double half = 0.5 * L;
    if ((__double2hiint(d) & 0x7fffffff) < __double2hiint(half)) return d;
    return min_image(d, L);
}
__device__ __forceinline__ bool fast_less(double x, double y) {   // squares
    const int a = __double2hiint(x) & 0x7fffffff, b = __double2hiint(y);
    return a != b ? a < b : x < y;
}

// Pixels found and not yet drawn.
struct SplatQueue {
    double rsq[64];
    int2 px[64];
    unsigned char k[64];   // the particle, as the lane that prepared it
};

// One pixel of a particle at squared distance rsq.
__device__ __forceinline__ void splat_pixel(const SplatArgs &A, int xx, int yy, double rsq,
                                            double coef, double inv_h) {
    // Lucy: q (1 + 3 s/h) (1 - s/h)^3
    double ih, t = fma(-sph::tile_sqrt(rsq, &ih), inv_h, 1.0);
    if (__double2hiint(t) < 0) t = 0.0;
    atomicAdd(&A.Z[(size_t)xx * A.ny + yy], coef * (t * t * t) * fma(-3.0, t, 4.0));
}

// Draws one found pixel per lane (the first `n` of the queue).
__device__ __forceinline__ void splat_draw(const SplatArgs &A, const SplatQueue &q, int n,
                                           const Splat &mine) {
    const int lane = threadIdx.x & 31, k = lane < n ? q.k[lane] : 0;
    const double coef = __shfl_sync(0xffffffffu, mine.coef, k);
    const double inv_h = __shfl_sync(0xffffffffu, mine.inv_h, k);
    if (lane >= n) return;
    splat_pixel(A, q.px[lane].x, q.px[lane].y, q.rsq[lane], coef, inv_h);
}

// The pixels of the lane's own particle.
__device__ __forceinline__ void splat_own(const SplatArgs &A, const Splat &s, double c2) {
    for (int col = 0; col < s.w; ++col) {
        const int xx = wrap_once(s.xa + col, A.nx);
        if (xx < 0 || xx >= A.nx) continue;
        const double dx = fast_image(s.rx - A.x[xx], A.xmax);
        for (int row = 0; row < s.hgt; ++row) {
            const int yy = wrap_once(s.ya + row, A.ny);
            if (yy < 0 || yy >= A.ny) continue;
            const double dy = fast_image(A.y[yy] - s.ry, A.ymax);
            const double rsq = dx * dx + fma(dy, dy, s.dz2);
            if (fast_less(rsq, c2)) splat_pixel(A, xx, yy, rsq, s.coef, s.inv_h);
        }
    }
}

// A warp per `per` particles: each lane prepares one (the divisions of a
// particle's box and weight are FP64 work that costs a warp the same for one
// lane), then the warp goes through them, a lane per pixel of the box; the pixels
// inside the cutoff (78% of a box) are queued across particles and drawn 32 at a
// time, so that the drawing, 13 FP64 operations a pixel and what bounds the
// kernel, has no idle lanes.  One thread per particle took 1.29 ms for 100,172
// particles on 635 x 633 pixels (94 pixels each), a lane per pixel without the
// queue 0.74 ms, this form 0.47 ms.
// Boxes of few pixels leave that form's lanes idle one particle after the other: a warp
// of such boxes alone draws them with a lane per particle, up to 36 pixels a box, fewer
// in proportion where a warp has fewer than 32 particles.  Queue / lane, us, 2D on 600^2
// pixels: 1,000,000 particles of 1.4 pixels 1055 / 227, of 13 1200 / 652, of 36 1698 /
// 1126, of 52 1961 / 2121; 20,000 (16 to a warp) of 13 63 / 59, of 36 77 / 87; 3,000 (two)
// of 6 36 / 40.
__global__ void __launch_bounds__(128) k_splat(const SplatArgs A) {
    __shared__ SplatQueue queues[4];
    SplatQueue &q = queues[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int first = (blockIdx.x * 4 + (threadIdx.x >> 5)) * A.per;
    if (first >= A.n) return;
    const double res = A.x[1] - A.x[0], c2 = A.cutoff * A.cutoff;
    const int count = min(A.per, A.n - first);
    const Splat mine = splat_prepare(A, min(first + lane, A.n - 1), res);
    if (__all_sync(0xffffffffu, mine.w <= A.own && mine.hgt <= A.own && mine.w * mine.hgt <= A.own)) {
        if (lane < count) splat_own(A, mine, c2);
        return;
    }
    int queued = 0;
    for (int k = 0; k < count; ++k) {
        const int w = __shfl_sync(0xffffffffu, mine.w, k);
        const int hgt = __shfl_sync(0xffffffffu, mine.hgt, k);
        if (w == 0 || hgt == 0) continue;
        const int xa = __shfl_sync(0xffffffffu, mine.xa, k);
        const int ya = __shfl_sync(0xffffffffu, mine.ya, k);
        const double rx = __shfl_sync(0xffffffffu, mine.rx, k);
        const double ry = __shfl_sync(0xffffffffu, mine.ry, k);
        const double dz2 = __shfl_sync(0xffffffffu, mine.dz2, k);
        // boxes of at most 32 columns and rows (the rule): each lane holds the
        // squared distance of one column and one row
        const bool small = w <= 32 && hgt <= 32;
        double dx2 = 0.0, dy2 = 0.0;
        if (small) {
            const int xx = wrap_once(xa + lane, A.nx), yy = wrap_once(ya + lane, A.ny);
            const double dx = fast_image(rx - A.x[min(max(xx, 0), A.nx - 1)], A.xmax);
            const double dy = fast_image(A.y[min(max(yy, 0), A.ny - 1)] - ry, A.ymax);
            dx2 = dx * dx;
            dy2 = fma(dy, dy, dz2);
        }
        const long long pixels = (long long)w * hgt;
        int col = lane % w, row = lane / w;
        const int dc = 32 % w, dr = 32 / w;
        for (long long p = lane; p - lane < pixels; p += 32) {
            const int xx = wrap_once(xa + col, A.nx), yy = wrap_once(ya + row, A.ny);
            const bool ok = p < pixels && xx >= 0 && xx < A.nx && yy >= 0 && yy < A.ny;
            double rsq = 0.0;
            if (small) {
                rsq = __shfl_sync(0xffffffffu, dx2, col) + __shfl_sync(0xffffffffu, dy2, row & 31);
            } else if (ok) {
                const double dx = fast_image(rx - A.x[xx], A.xmax);
                const double dy = fast_image(A.y[yy] - ry, A.ymax);
                rsq = fma(dx, dx, fma(dy, dy, dz2));
            }
            const bool in = ok && fast_less(rsq, c2);
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int at = queued + __popc(mask & ((1u << lane) - 1u));
                q.rsq[at] = rsq;
                q.px[at] = make_int2(xx, yy);
                q.k[at] = (unsigned char)k;
            }
            queued += __popc(mask);
            if (queued >= 32) {
                __syncwarp();
                splat_draw(A, q, 32, mine);
                queued -= 32;
                // the rest moves to the front
                const bool keep = lane < queued;
                const double r2 = q.rsq[32 + lane];
                const int2 px = q.px[32 + lane];
                const unsigned char kk = q.k[32 + lane];
                __syncwarp();
                if (keep) {
                    q.rsq[lane] = r2;
                    q.px[lane] = px;
                    q.k[lane] = kk;
                }
                __syncwarp();
            }
            col += dc;
            row += dr;
            if (col >= w) {
                col -= w;
                ++row;
            }
        }
    }
    __syncwarp();
    splat_draw(A, q, queued, mine);
}

}  // namespace

extern "C" int sph_splash_map(int32_t mode, int64_t n, const double *r, int32_t r_cols,
                              const double *m, const double *rho, const double *a,
                              const double *h, int32_t nx, int32_t ny, const double *x,
                              const double *y, double z, const double *bounds, double cutoff,
                              double *Z, int32_t mem, void *stream) {
    if ((mode != 2 && mode != 3) || n < 0 || nx < 2 || ny < 1 || !bounds || !Z || !x || !y)
        return SPH_EINVAL;
    if (r_cols < (mode == 3 ? 3 : 2)) return SPH_EINVAL;
    if (!(cutoff > 0)) return SPH_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    size_t npix = (size_t)nx * ny;
    // device copies of host inputs (this entry point is not on the step path)
    const double *dr = r, *dm = m, *drho = rho, *da = a, *dh = h, *dx = x, *dy = y;
    double *dZ = Z;
    double *buf = nullptr;
    if (mem == SPH_HOST) {
        size_t need = (size_t)n * (r_cols + 4) + nx + ny + npix;
        if (cudaMalloc(&buf, sizeof(double) * (need ? need : 1)) != cudaSuccess) {
            cudaGetLastError();
            return SPH_ENOMEM;
        }
        double *p = buf;
        auto up = [&](const double *src, size_t cnt) {
            cudaMemcpyAsync(p, src, sizeof(double) * cnt, cudaMemcpyHostToDevice, st);
            double *q = p;
            p += cnt;
            return (const double *)q;
        };
        dr = up(r, (size_t)n * r_cols);
        dm = up(m, n);
        drho = up(rho, n);
        da = up(a ? a : rho, n);
        dh = up(h, n);
        dx = up(x, nx);
        dy = up(y, ny);
        dZ = p;
    } else if (!a) {
        da = rho;
    }
    cudaMemsetAsync(dZ, 0, sizeof(double) * npix, st);
    if (n > 0) {
        // enough warps for eight on every SM, at most 32 particles each
        const int sms = sph::device_sms();
        const int per = (int)std::min<int64_t>(32, std::max<int64_t>(1, n / (8 * sms)));
        const SplatArgs A = {(int)n,    r_cols,    nx,        ny,        mode == 3 ? 1 : 0,
                             per,       36 * per / 32, dr,        dm,        drho,      da,
                             dh,        dx,        dy,        z,         bounds[0],
                             bounds[1], bounds[2], bounds[3], cutoff,    dZ};
        const int64_t warps = (n + per - 1) / per;
        k_splat<<<(int)((warps + 3) / 4), 128, 0, st>>>(A);
    }
    int status = SPH_OK;
    if (mem == SPH_HOST) {
        if (cudaMemcpyAsync(Z, dZ, sizeof(double) * npix, cudaMemcpyDeviceToHost, st) !=
            cudaSuccess)
            status = SPH_ECUDA;
    }
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        status = SPH_ECUDA;
    if (buf) cudaFree(buf);
    return status;
}
