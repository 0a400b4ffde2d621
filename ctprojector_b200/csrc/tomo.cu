// tomo.cu -- distance-driven tomosynthesis projector pair (z main axis,
// detector u = (1,0,0), v = (0,1,0)), sm_100a.
//
// Reference: DDFPConeBoxIntKernelXY distanceDriven3DBoxInt.cu:28-117,
// DDBPConeBoxIntCartKernelXY :170-216, PreweightBPCartKernelXY
// distanceDriven3DUtils.cu:10-31, ProjectConeToDetCart :45-56, and the 2D box
// integral IntegralBoxXY cudaMath.cu:336-404.
//
// Forward: per ray and z plane the normalised integral of the plane over the
// footprint rectangle of the cell.  Back projection (reference-parity form): per
// voxel and view the normalised integral of the length-weighted projection over
// the voxel's projected rectangle.  The per-cell ray-length weight is applied
// once in a pre-pass into the workspace.  The rectangles' two sides are
// separable, so a thread takes 8 to 32 rays (voxels) of one column and shares
// the work along y: 64 x 256 x 512 voxels, 25 views of 1024 x 512 cells of 0.25 mm,
// forward and back 4.55 -> 1.63 ms against one rectangle per thread and plane (or
// view); both kernels are bound by instruction issue and the L1.  Cells much
// finer or coarser than the pixels keep one rectangle per thread (shared_rows).
// Unlike the reference, every batch item reads its own weighted projections
// (the reference reads item 0's for all items, distanceDriven3DBoxInt.cu:257-259).
#include <cuda_runtime.h>
#include <math.h>

#include "ctp_common.cuh"

namespace ctp {

namespace {

// Exact integral of an (ny, nx) plane over the clamped rectangle.
__device__ float box2d(const float* __restrict__ p, float x1, float y1, float x2, float y2, int nx, int ny) {
    x1 = clampf(x1, 0.f, (float)nx);
    y1 = clampf(y1, 0.f, (float)ny);
    x2 = clampf(x2, 0.f, (float)nx);
    y2 = clampf(y2, 0.f, (float)ny);
    if (x2 <= x1 || y2 <= y1) return 0.f;
    int ix1 = min((int)x1, nx - 1), iy1 = min((int)y1, ny - 1);
    int ix2 = min((int)x2, nx - 1), iy2 = min((int)y2, ny - 1);
    float v = 0.f;
    for (int iy = iy1; iy <= iy2; ++iy) {
        float wy = 1.f;
        if (iy == iy1) wy -= (y1 - (float)iy1);
        if (iy == iy2) wy -= ((float)(iy2 + 1) - y2);
        const float* row = p + (size_t)iy * nx;
        float r = 0.f;
        for (int ix = ix1; ix <= ix2; ++ix) r += __ldg(row + ix);
        r -= __ldg(row + ix1) * (x1 - (float)ix1);
        r -= __ldg(row + ix2) * ((float)(ix2 + 1) - x2);
        v += r * wy;
    }
    return v;
}

// One axis of a footprint: the overlaps of [lo, hi] (clamped to [0, n]) with
// the cells i, i + 1, ... times inv (one over the unclamped width); K cells
// hold it when hi - lo <= K - 1.  Zero for an empty or reversed interval.
template <int K>
struct Taps {
    float w[K];
    int i;
};
template <int K>
__device__ __forceinline__ Taps<K> taps(double lo, double hi, float inv, int n) {
    Taps<K> t;
    const double a = fmin(fmax(lo, 0.0), (double)n), b = fmin(fmax(hi, 0.0), (double)n);
    t.i = min((int)a, n - 1);
    const float fa = (float)(a - (double)t.i), fb = (float)(b - (double)t.i);  // from cell i
#pragma unroll
    for (int k = 0; k < K; ++k)
        t.w[k] = fmaxf(fminf(fb, (float)(k + 1)) - fmaxf(fa, (float)k), 0.f) * inv;
    return t;
}

// A footprint that misses the array was clamped to cells of its border: they
// are left unread (0 x infinity is not 0).  Along a row of a table the mark
// kMissed on the first cell sends the lookup past the sums, to zeros.
constexpr int kMissed = 0x40000000;
template <int K>
__device__ __forceinline__ bool missed(const Taps<K>& t) {
    bool m = true;
#pragma unroll
    for (int k = 0; k < K; ++k) m = m && t.w[k] == 0.f;
    return m;
}
template <int K>
__device__ __forceinline__ float row_index(const Taps<K>& t) {
    return __int_as_float(missed(t) ? t.i | kMissed : t.i);
}
__device__ __forceinline__ int first_row(float index) { return __float_as_int(index) & ~kMissed; }

// A view's rays in image coordinates: source (sx, sy, sz), and the cell edges'
// position on plane z: sx + r (z - sz).
struct TomoRays {
    double sx, sy, sz, cz, ox, oy;  // ox, oy: detector centre, physical
};
__device__ __forceinline__ TomoRays tomo_rays(const float* dc, const float* sr, int view, const Grid& g) {
    TomoRays r;
    r.sx = ((double)sr[view * 3] - g.cx) / g.dx + 0.5 * g.nx;
    r.sy = ((double)sr[view * 3 + 1] - g.cy) / g.dy + 0.5 * g.ny;
    r.sz = ((double)sr[view * 3 + 2] - g.cz) / g.dz + 0.5 * g.nz;
    r.cz = ((double)dc[view * 3 + 2] - g.cz) / g.dz + 0.5 * g.nz;
    r.ox = dc[view * 3];
    r.oy = dc[view * 3 + 1];
    return r;
}
// Slopes of the two edges of cell i along one axis (lower first).
__device__ __forceinline__ void edge_slopes(double o, double cell, double i_centre, double c, double d, double half_n,
                                            double s, double depth, double& r1, double& r2) {
    const double a = (o + (i_centre - 0.5) * cell - c) / d + half_n, b = (o + (i_centre + 0.5) * cell - c) / d + half_n;
    r1 = (fmin(a, b) - s) / depth;
    r2 = (fmax(a, b) - s) / depth;
}

// One ray over wide footprints (more than 2 x 2 pixels on some plane).
__device__ __noinline__ float tomo_ray_wide(const float* __restrict__ vol, const TomoRays& R, double rx1, double rx2,
                                            double ry1, double ry2, int nx, int ny, int nz) {
    float val = 0.f;
    for (int iz = 0; iz < nz; ++iz) {
        const double dz = iz - R.sz;
        const float x1 = (float)(R.sx + rx1 * dz), x2 = (float)(R.sx + rx2 * dz);
        const float y1 = (float)(R.sy + ry1 * dz), y2 = (float)(R.sy + ry2 * dz);
        val += box2d(vol + (size_t)iz * nx * ny, x1, y1, x2, y2, nx, ny) / ((x2 - x1) * (y2 - y1));
    }
    return val;
}

constexpr int kTomoThreads = 128;
constexpr int kTomoStep = 8;  // planes (FP) or views (BP) whose row tables are built together

// Forward projection.  The footprint of a cell on a plane is a rectangle whose
// x side depends on the cell's column alone and whose y side on its row alone,
// so a thread takes one column u and VT rows v of a view.  Per plane it sums
// the image rows that its cells fall on over x (two pixels each, all loads
// independent) into its own column of shared memory, then forms each cell as
// the y-weighted sum of two of them; the rows' y weights come from a table that
// the block builds for 8 planes at a time.  Cells are finer than pixels here, so
// a row's x sum serves one to several cells.  Views with footprints above 2 x 2
// pixels (the width grows with the distance from the source, so the end plane
// farther from it bounds it) go ray by ray.
template <int VT>
__global__ void __launch_bounds__(kTomoThreads, 6) tomo_fp_kernel(float* __restrict__ prj, const float* __restrict__ img,
                                                                  const float* __restrict__ dc,
                                                                  const float* __restrict__ sr, int nview, Grid g, Det d) {
    __shared__ float4 s_row[kTomoStep][VT];          // y weights of a cell row, its first image row
    // each thread its own column: up to VT + 2 rows summed over x and two of zeros, then results
    __shared__ float s_sum[VT + 4][kTomoThreads];
    const int tid = threadIdx.x;
    const int iu = blockIdx.x * kTomoThreads + tid;
    const int v0 = blockIdx.y * VT;
    const int view = blockIdx.z % nview, b = blockIdx.z / nview;
    const TomoRays R = tomo_rays(dc, sr, view, g);
    const double cu = (double)min(iu, d.nu - 1) - d.off_u - (d.nu - 1) / 2.0;
    double rx1, rx2;
    edge_slopes(R.ox, d.du, cu, g.cx, g.dx, 0.5 * g.nx, R.sx, R.cz - R.sz, rx1, rx2);
    auto row_slopes = [&](int iv, double& r1, double& r2) {
        edge_slopes(R.oy, d.dv, (double)iv - d.off_v - (d.nv - 1) / 2.0, g.cy, g.dy, 0.5 * g.ny, R.sy, R.cz - R.sz, r1, r2);
    };
    const double dmax = fmax(fabs(0.0 - R.sz), fabs((double)(g.nz - 1) - R.sz));
    const float* vol = img + (size_t)b * g.nx * g.ny * g.nz;
    const double wide_x = fabs((double)d.du / g.dx / (R.cz - R.sz)), wide_y = fabs((double)d.dv / g.dy / (R.cz - R.sz));
    if (wide_x * dmax <= 1.0 && wide_y * dmax <= 1.0) {
        float acc[VT];
#pragma unroll
        for (int q = 0; q < VT; ++q) acc[q] = 0.f;
        s_sum[VT + 2][tid] = s_sum[VT + 3][tid] = 0.f;
        for (int z0 = 0; z0 < g.nz; z0 += kTomoStep) {
            const int nz = min(kTomoStep, g.nz - z0);
            __syncthreads();
#pragma unroll 1
            for (int i = tid; i < nz * VT; i += kTomoThreads) {
                const int z = i / VT, q = i - z * VT;
                double r1, r2;
                row_slopes(min(v0 + q, d.nv - 1), r1, r2);
                const double dz = z0 + z - R.sz;
                const Taps<2> t = taps<2>(R.sy + r1 * dz, R.sy + r2 * dz, (float)(1.0 / ((r2 - r1) * dz)), g.ny);
                s_row[z][q] = make_float4(t.w[0], t.w[1], row_index(t), 0.f);
            }
            __syncthreads();
#pragma unroll 1
            for (int z = 0; z < nz; ++z) {
                const double dz = z0 + z - R.sz;
                const Taps<2> t = taps<2>(R.sx + rx1 * dz, R.sx + rx2 * dz, __fdividef(1.f, (float)((rx2 - rx1) * dz)), g.nx);
                if (missed(t)) continue;
                const int right = t.i + 1 < g.nx ? 1 : 0;
                // image rows of the first and last cell (rows advance by at most one per cell)
                const int ra = first_row(s_row[z][0].z), rb = first_row(s_row[z][VT - 1].z);
                const int y0 = min(ra, rb), n = min(max(ra, rb) + 1 - y0, VT + 1);
                const float* col = vol + ((size_t)(z0 + z) * g.ny + y0) * g.nx + t.i;
                const int last = g.ny - 1 - y0;
#pragma unroll 8
                for (int r = 0; r <= n; ++r) {
                    const float* row = col + (size_t)min(r, last) * g.nx;
                    s_sum[r][tid] = fmaf(t.w[1], __ldg(row + right), t.w[0] * __ldg(row));
                }
#pragma unroll
                for (int k = 0; k < VT; ++k) {
                    const float4 e = s_row[z][k];
                    const int r = min(__float_as_int(e.z) - y0, VT + 2);
                    acc[k] = fmaf(e.x, s_sum[r][tid], fmaf(e.y, s_sum[r + 1][tid], acc[k]));
                }
            }
        }
#pragma unroll
        for (int k = 0; k < VT; ++k) s_sum[k][tid] = acc[k];
    } else {
#pragma unroll 1
        for (int k = 0; k < VT; ++k) {
            double ry1, ry2;
            row_slopes(min(v0 + k, d.nv - 1), ry1, ry2);
            s_sum[k][tid] = tomo_ray_wide(vol, R, rx1, rx2, ry1, ry2, g.nx, g.ny, g.nz);
        }
    }
    if (iu >= d.nu) return;
    // ray length over the plane distance
    const double du = cu * d.du + R.ox - sr[view * 3], dzp = (double)dc[view * 3 + 2] - sr[view * 3 + 2];
#pragma unroll 1
    for (int k = 0; k < VT; ++k) {
        const int iv = v0 + k;
        if (iv >= d.nv) break;
        const double dv = ((double)iv - d.off_v - (d.nv - 1) / 2.0) * d.dv + R.oy - sr[view * 3 + 1];
        const double len = sqrt(du * du + dv * dv + dzp * dzp);
        prj[(((size_t)b * nview + view) * d.nv + iv) * d.nu + iu] = s_sum[k][tid] * (float)(g.dz / fabs(dzp) * len);
    }
}

// Length-weighted projections, one cell per thread of a one-dimensional grid
// (views x batch items may exceed a grid's third dimension).
__global__ void tomo_preweight_kernel(float* __restrict__ out, const float* __restrict__ prj,
                                      const float* __restrict__ dc, const float* __restrict__ sr, int nview, Det d,
                                      float dz, unsigned blocks_u) {
    const unsigned row = blockIdx.x / blocks_u;  // of all views and batch items
    const int iu = (int)(blockIdx.x - row * blocks_u) * blockDim.x + threadIdx.x;
    if (iu >= d.nu) return;
    const int iv = (int)(row % d.nv), view = (int)(row / d.nv % nview);
    const double u = ((double)iu - d.off_u - (d.nu - 1) / 2.0) * d.du + dc[view * 3] - sr[view * 3];
    const double v = ((double)iv - d.off_v - (d.nv - 1) / 2.0) * d.dv + dc[view * 3 + 1] - sr[view * 3 + 1];
    const double h = (double)dc[view * 3 + 2] - sr[view * 3 + 2];
    const size_t i = (size_t)row * d.nu + iu;
    out[i] = prj[i] * (float)(dz / fabs(h) * sqrt(u * u + v * v + h * h));
}

// Normalised integral of a view over one voxel's wide footprint (more than 3 x 3 cells).
__device__ __noinline__ float tomo_box_wide(const float* __restrict__ pv, float u1, float u2, float v1, float v2, int nu,
                                            int nv) {
    return box2d(pv, u1, v1, u2, v2, nu, nv) / ((u2 - u1) * (v2 - v1));
}

// Back projection.  A voxel's footprint on a view is a rectangle whose u side
// depends on x (and the plane) alone and whose v side on y alone, so a thread
// takes one x and YT rows y of a plane.  Per view it sums the detector rows that
// its voxels fall on over u (up to 3 cells each, all loads independent) into
// its own column of shared memory, then forms each voxel as the v-weighted sum
// of up to three of them; the rows' v weights come from a table that the block
// builds for 8 views at a time, with the views' u mapping (affine in x).
template <int YT>
__global__ void __launch_bounds__(kTomoThreads, 5) tomo_bp_kernel(float* __restrict__ img, const float* __restrict__ wprj,
                                                                  const float* __restrict__ dc,
                                                                  const float* __restrict__ sr, int nview, Grid g, Det d) {
    constexpr int kRows = 2 * YT + 2;                 // detector rows under YT voxels of at most 2 rows
    __shared__ float4 s_row[kTomoStep][YT];           // v weights of a voxel row, its first detector row
    __shared__ double s_u[kTomoStep][2];              // u = s_u[0] + s_u[1] x
    __shared__ float s_sum[kRows + 3][kTomoThreads];  // each thread its own column: rows summed over u, three of zeros
    const int tid = threadIdx.x;
    const int ix = blockIdx.x * kTomoThreads + tid;
    const int y0 = blockIdx.y * YT;
    const int iz = blockIdx.z % g.nz, b = blockIdx.z / g.nz;
    const double x = ((double)min(ix, g.nx - 1) - (g.nx - 1) / 2.0) * g.dx + g.cx;
    const double z = ((double)iz - (g.nz - 1) / 2.0) * g.dz + g.cz;
    const float* pb = wprj + (size_t)b * nview * d.nv * d.nu;
    float acc[YT];
#pragma unroll
    for (int q = 0; q < YT; ++q) acc[q] = 0.f;
    s_sum[kRows][tid] = s_sum[kRows + 1][tid] = s_sum[kRows + 2][tid] = 0.f;
    // detector coordinate of the position p along one axis: lo + slope p
    auto mapping = [&](double S, double C, double cell, double off, int n, double r, double& c0, double& c1) {
        c1 = r / cell;
        c0 = (S - C - r * S) / cell + off + (n - 1) / 2.0;
    };
    auto magnification = [&](int view) {
        return ((double)dc[view * 3 + 2] - sr[view * 3 + 2]) / (z - sr[view * 3 + 2]);
    };
    auto voxel_y = [&](int q) { return ((double)min(y0 + q, g.ny - 1) - (g.ny - 1) / 2.0) * g.dy + g.cy; };
    const double hx = 0.5 * g.dx, hy = 0.5 * g.dy;
    for (int w0 = 0; w0 < nview; w0 += kTomoStep) {
        const int nw = min(kTomoStep, nview - w0);
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < nw * YT; i += kTomoThreads) {
            const int w = i / YT, q = i - w * YT, view = w0 + w;
            const double r = magnification(view);
            double c0, c1;
            mapping(sr[view * 3 + 1], dc[view * 3 + 1], d.dv, d.off_v, d.nv, r, c0, c1);
            const double y = voxel_y(q);
            const Taps<3> t = taps<3>(fma(c1, y - hy, c0), fma(c1, y + hy, c0), (float)(1.0 / (c1 * g.dy)), d.nv);
            s_row[w][q] = make_float4(t.w[0], t.w[1], t.w[2], row_index(t));
            if (q == 0) mapping(sr[view * 3], dc[view * 3], d.du, d.off_u, d.nu, r, s_u[w][0], s_u[w][1]);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < nw; ++w) {
            const int view = w0 + w;
            const double c0 = s_u[w][0], c1 = s_u[w][1];
            const double u1 = fma(c1, x - hx, c0), u2 = fma(c1, x + hx, c0);
            const float* pv = pb + (size_t)view * d.nv * d.nu;
            const double wu = fabs(c1 * g.dx), wv = fabs(c1 * d.du / d.dv * g.dy);
            if (wu <= 2.0 && wv <= 2.0) {
                const Taps<3> t = taps<3>(u1, u2, __fdividef(1.f, (float)(c1 * g.dx)), d.nu);
                if (missed(t)) continue;
                const int i1 = min(1, d.nu - 1 - t.i), i2 = min(2, d.nu - 1 - t.i);
                // detector rows of the first and last voxel (rows advance by at most two per voxel)
                const int ra = first_row(s_row[w][0].w), rb = first_row(s_row[w][YT - 1].w);
                const int v0 = min(ra, rb), n = min(max(ra, rb) + 3 - v0, kRows), last = d.nv - 1 - v0;
                const float* col = pv + (size_t)v0 * d.nu + t.i;
#pragma unroll 6
                for (int r = 0; r < n; ++r) {
                    const float* p = col + (size_t)min(r, last) * d.nu;
                    s_sum[r][tid] = fmaf(t.w[2], __ldg(p + i2), fmaf(t.w[1], __ldg(p + i1), t.w[0] * __ldg(p)));
                }
#pragma unroll
                for (int k = 0; k < YT; ++k) {
                    const float4 e = s_row[w][k];
                    const int r = min(__float_as_int(e.w) - v0, kRows);
                    acc[k] = fmaf(e.x, s_sum[r][tid], fmaf(e.y, s_sum[r + 1][tid], fmaf(e.z, s_sum[r + 2][tid], acc[k])));
                }
            } else {
                double m0, m1;
                mapping(sr[view * 3 + 1], dc[view * 3 + 1], d.dv, d.off_v, d.nv, magnification(view), m0, m1);
#pragma unroll 1
                for (int k = 0; k < YT; ++k) {
                    const double y = voxel_y(k);
                    s_sum[k][tid] = tomo_box_wide(pv, (float)u1, (float)u2, (float)fma(m1, y - hy, m0),
                                                  (float)fma(m1, y + hy, m0), d.nu, d.nv);
                }
#pragma unroll
                for (int k = 0; k < YT; ++k) acc[k] += s_sum[k][tid];
            }
        }
    }
    if (ix >= g.nx) return;
#pragma unroll
    for (int k = 0; k < YT; ++k) {
        if (y0 + k >= g.ny) break;
        img[(((size_t)b * g.nz + iz) * g.ny + y0 + k) * g.nx + ix] = acc[k];
    }
}

// Rows per thread: 32, or fewer while the launch has less than four blocks per
// SM (each block then re-reads more of its neighbours' rows).
int tomo_rows(size_t columns, size_t rows, size_t planes, int most) {
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int t = most; t > 8; t /= 2)
        if (((columns + kTomoThreads - 1) / kTomoThreads) * ((rows + t - 1) / t) * planes >= 4 * (size_t)sms) return t;
    return 8;
}

// One ray (FP) or voxel (BP) per thread, a rectangle per plane or view: for
// cells much finer or coarser than the pixels (shared_rows).

// The same integral when the rectangle spans at most K pixels along each axis
// (x2 - x1 <= K - 1 and y2 - y1 <= K - 1, K = 2 or 3): the pixel weights are
// the overlaps of the clamped rectangle with K consecutive columns and rows,
// straight-line code with K*K loads (indices clamped, weights 0 past the
// edge) instead of the general loops.
template <int K>
__device__ __forceinline__ float box2d_small(const float* __restrict__ p, float x1, float y1, float x2, float y2,
                                             int nx, int ny) {
    x1 = clampf(x1, 0.f, (float)nx);
    y1 = clampf(y1, 0.f, (float)ny);
    x2 = clampf(x2, 0.f, (float)nx);
    y2 = clampf(y2, 0.f, (float)ny);
    if (x2 <= x1 || y2 <= y1) return 0.f;
    const int ix = min((int)x1, nx - 1), iy = min((int)y1, ny - 1);
    float wx[K], wy[K];
    int cx[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        // overlap of [x1, x2] with column ix + k (and of [y1, y2] with row iy + k)
        wx[k] = fmaxf(fminf(x2, (float)(ix + k + 1)) - fmaxf(x1, (float)(ix + k)), 0.f);
        wy[k] = fmaxf(fminf(y2, (float)(iy + k + 1)) - fmaxf(y1, (float)(iy + k)), 0.f);
        cx[k] = min(ix + k, nx - 1);
    }
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const float* row = p + (size_t)min(iy + j, ny - 1) * nx;
        float r = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) r = fmaf(wx[k], __ldg(row + cx[k]), r);
        v = fmaf(wy[j], r, v);
    }
    return v;
}

__global__ void __launch_bounds__(256) tomo_fp_ray_kernel(float* __restrict__ prj, const float* __restrict__ img,
                                                      const float* __restrict__ dc, const float* __restrict__ sr,
                                                      int nview, Grid g, Det d) {
    int iu = blockIdx.x * 32 + (threadIdx.x & 31);
    int iv = blockIdx.y * 8 + (threadIdx.x >> 5);
    int view = blockIdx.z % nview, b = blockIdx.z / nview;
    if (iu >= d.nu || iv >= d.nv) return;
    double u = ((double)iu - d.off_u - (d.nu - 1) / 2.0) * d.du;
    double v = ((double)iv - d.off_v - (d.nv - 1) / 2.0) * d.dv;
    double C[3] = {dc[view * 3], dc[view * 3 + 1], dc[view * 3 + 2]};
    double S[3] = {sr[view * 3], sr[view * 3 + 1], sr[view * 3 + 2]};
    // image coordinates of the source and of the four cell-edge mid points
    auto ix_ = [&](double x) { return (x - g.cx) / g.dx + 0.5 * g.nx; };
    auto iy_ = [&](double y) { return (y - g.cy) / g.dy + 0.5 * g.ny; };
    auto iz_ = [&](double z) { return (z - g.cz) / g.dz + 0.5 * g.nz; };
    double sx = ix_(S[0]), sy = iy_(S[1]), sz = iz_(S[2]);
    double cz = iz_(C[2]);
    double xa = ix_(C[0] + u - d.du / 2.0), xb = ix_(C[0] + u + d.du / 2.0);
    double ya = iy_(C[1] + v - d.dv / 2.0), yb = iy_(C[1] + v + d.dv / 2.0);
    if (xa > xb) { double t = xa; xa = xb; xb = t; }
    if (ya > yb) { double t = ya; ya = yb; yb = t; }
    double rx1 = (xa - sx) / (cz - sz), rx2 = (xb - sx) / (cz - sz);
    double ry1 = (ya - sy) / (cz - sz), ry2 = (yb - sy) / (cz - sz);
    const float* vol = img + (size_t)b * g.nx * g.ny * g.nz;
    float val = 0.f;
    // footprint widths grow linearly with the distance from the source: the
    // widest is on the end plane farther from it
    const double dmax = fmax(fabs(0.0 - sz), fabs((double)(g.nz - 1) - sz));
    if (fabs(rx2 - rx1) * dmax <= 1.0 && fabs(ry2 - ry1) * dmax <= 1.0) {
        // at most 2 x 2 pixels per plane; edges in FP32 from per-ray FP32
        // coefficients (the width and the integral see the same rounded edges)
        const float fsx = (float)sx, fsy = (float)sy, fsz = (float)sz;
        const float frx1 = (float)rx1, frx2 = (float)rx2, fry1 = (float)ry1, fry2 = (float)ry2;
        for (int iz = 0; iz < g.nz; ++iz) {
            const float dz = (float)iz - fsz;
            const float x1 = fmaf(frx1, dz, fsx), x2 = fmaf(frx2, dz, fsx);
            const float y1 = fmaf(fry1, dz, fsy), y2 = fmaf(fry2, dz, fsy);
            val += __fdividef(box2d_small<2>(vol + (size_t)iz * g.nx * g.ny, x1, y1, x2, y2, g.nx, g.ny),
                              (x2 - x1) * (y2 - y1));
        }
    } else {
        for (int iz = 0; iz < g.nz; ++iz) {
            double dz = iz - sz;
            float x1 = (float)(sx + rx1 * dz), x2 = (float)(sx + rx2 * dz);
            float y1 = (float)(sy + ry1 * dz), y2 = (float)(sy + ry2 * dz);
            val += box2d(vol + (size_t)iz * g.nx * g.ny, x1, y1, x2, y2, g.nx, g.ny) / ((x2 - x1) * (y2 - y1));
        }
    }
    double D[3] = {C[0] + u, C[1] + v, C[2]};
    double L = sqrt((S[2] - D[2]) * (S[2] - D[2]) + (S[1] - D[1]) * (S[1] - D[1]) + (S[0] - D[0]) * (S[0] - D[0]));
    val *= (float)(g.dz / fabs(S[2] - D[2]) * L);
    float* o = prj + (((size_t)b * nview + view) * d.nv + iv) * d.nu + iu;
    *o = val;
}

__global__ void __launch_bounds__(256) tomo_bp_voxel_kernel(float* __restrict__ img, const float* __restrict__ wprj,
                                                      const float* __restrict__ dc, const float* __restrict__ sr,
                                                      int nview, Grid g, Det d) {
    int ix = blockIdx.x * 32 + (threadIdx.x & 31);
    int iy = blockIdx.y * 8 + (threadIdx.x >> 5);
    int iz = blockIdx.z % g.nz, b = blockIdx.z / g.nz;
    if (ix >= g.nx || iy >= g.ny) return;
    float x = ((float)ix - (g.nx - 1) / 2.0f) * g.dx + g.cx;
    float y = ((float)iy - (g.ny - 1) / 2.0f) * g.dy + g.cy;
    float z = ((float)iz - (g.nz - 1) / 2.0f) * g.dz + g.cz;
    const float* pb = wprj + (size_t)b * nview * d.nv * d.nu;
    // fast divides and reciprocals of the cell sizes (a few ulp each)
    const float idu = 1.f / d.du, idv = 1.f / d.dv;
    float val = 0.f;
    for (int view = 0; view < nview; ++view) {
        float Sx = sr[view * 3], Sy = sr[view * 3 + 1], Sz = sr[view * 3 + 2];
        float Cx = dc[view * 3], Cy = dc[view * 3 + 1], Cz = dc[view * 3 + 2];
        float r = __fdividef(Cz - Sz, z - Sz);
        float u1 = (Sx - Cx + r * (x - g.dx / 2 - Sx)) * idu + d.off_u + (d.nu - 1) / 2.0f;
        float u2 = (Sx - Cx + r * (x + g.dx / 2 - Sx)) * idu + d.off_u + (d.nu - 1) / 2.0f;
        float v1 = (Sy - Cy + r * (y - g.dy / 2 - Sy)) * idv + d.off_v + (d.nv - 1) / 2.0f;
        float v2 = (Sy - Cy + r * (y + g.dy / 2 - Sy)) * idv + d.off_v + (d.nv - 1) / 2.0f;
        const float* pv = pb + (size_t)view * d.nv * d.nu;
        const float w = fabsf(u2 - u1), h = fabsf(v2 - v1);
        float box;
        if (w <= 1.f && h <= 1.f) box = box2d_small<2>(pv, u1, v1, u2, v2, d.nu, d.nv);
        else if (w <= 2.f && h <= 2.f) box = box2d_small<3>(pv, u1, v1, u2, v2, d.nu, d.nv);
        else box = box2d(pv, u1, v1, u2, v2, d.nu, d.nv);
        val += __fdividef(box, (u2 - u1) * (v2 - v1));
    }
    float* o = img + (((size_t)b * g.nz + iz) * g.ny + iy) * g.nx + ix;
    *o = val;
}

// Whether the kernels with shared row sums take the call: cells no larger than
// the pixels (a footprint then spans at most two pixels of any plane between
// source and panel) and no smaller than 0.6 of them (a voxel at most two cells
// at magnifications to 1.2), with a margin for sizes rounded to FP32 (0.24 over
// 0.4 is 0.59999998).  Elsewhere their threads fall back to whole rectangles,
// with fewer of them in flight.  Pixels of 0.4 mm, forward and back, one rectangle
// per thread and shared rows: cells of 0.25 mm 4.55 and 1.63 ms (64 x 256 x 512
// voxels, 25 views), 0.24 mm 466 and 232 us (56 x 166 x 200, 10 views); 0.52 mm
// 221 and 336 us (18 x 127 x 273, 19 views), 0.57 mm 137 and 310 us (26 x 121 x 225,
// 9 views).
bool shared_rows(const ctp_geometry& g) {
    const double finest = 0.6 * (1 - 1e-6);
    const double u = fabs((double)g.du / g.dx), v = fabs((double)g.dv / g.dy);
    return u <= 1.0 && v <= 1.0 && u >= finest && v >= finest;
}

}  // namespace

int tomo_fp(float* prj, const float* img, const float* dc, const float* sr, const ctp_geometry& g, unsigned flags,
            cudaStream_t s) {
    (void)flags;  // the reference overwrites
    if (!shared_rows(g)) {
        tomo_fp_ray_kernel<<<dim3((unsigned)((g.nu + 31) / 32), (unsigned)((g.nv + 7) / 8),
                                  (unsigned)(g.nview * g.nbatch)),
                             256, 0, s>>>(prj, img, dc, sr, (int)g.nview, make_grid(g), make_det(g));
        return check_launch("tomo_fp_ray_kernel");
    }
    const int t = tomo_rows(g.nu, g.nv, g.nview * g.nbatch, 32);
    dim3 grid((unsigned)((g.nu + kTomoThreads - 1) / kTomoThreads), (unsigned)((g.nv + t - 1) / t),
              (unsigned)(g.nview * g.nbatch));
    auto k = t == 32 ? tomo_fp_kernel<32> : t == 16 ? tomo_fp_kernel<16> : tomo_fp_kernel<8>;
    k<<<grid, kTomoThreads, 0, s>>>(prj, img, dc, sr, (int)g.nview, make_grid(g), make_det(g));
    return check_launch("tomo_fp_kernel");
}

size_t tomo_bp_workspace(const ctp_geometry& g) { return align_up(g.nbatch * g.nview * g.nv * g.nu * sizeof(float)); }

int tomo_bp(float* img, const float* prj, const float* dc, const float* sr, const ctp_geometry& g, unsigned flags,
            void* workspace, size_t workspace_bytes, cudaStream_t s) {
    Scratch scr;
    int rc = scr.acquire(workspace, workspace_bytes, tomo_bp_workspace(g), s);
    if (rc) return rc;
    float* wprj = reinterpret_cast<float*>(scr.base());
    const size_t blocks_u = (g.nu + 127) / 128;
    tomo_preweight_kernel<<<(unsigned)(blocks_u * g.nv * g.nview * g.nbatch), 128, 0, s>>>(
        wprj, prj, dc, sr, (int)g.nview, make_det(g), g.dz, (unsigned)blocks_u);
    if ((rc = check_launch("tomo_preweight_kernel"))) return rc;
    (void)flags;
    if (!shared_rows(g)) {
        tomo_bp_voxel_kernel<<<dim3((unsigned)((g.nx + 31) / 32), (unsigned)((g.ny + 7) / 8),
                                    (unsigned)(g.nz * g.nbatch)),
                               256, 0, s>>>(img, wprj, dc, sr, (int)g.nview, make_grid(g), make_det(g));
        return check_launch("tomo_bp_voxel_kernel");
    }
    const int t = tomo_rows(g.nx, g.ny, g.nz * g.nbatch, 32);
    dim3 grid((unsigned)((g.nx + kTomoThreads - 1) / kTomoThreads), (unsigned)((g.ny + t - 1) / t),
              (unsigned)(g.nz * g.nbatch));
    auto k = t == 32 ? tomo_bp_kernel<32> : t == 16 ? tomo_bp_kernel<16> : tomo_bp_kernel<8>;
    k<<<grid, kTomoThreads, 0, s>>>(img, wprj, dc, sr, (int)g.nview, make_grid(g), make_det(g));
    return check_launch("tomo_bp_kernel");
}

}  // namespace ctp
