// siddon_columns.cu -- Siddon cone-beam projector pair for upright views,
// sm_100a: views whose detector v axis is the z axis and whose u axis has no z
// component (circular and helical scans of a flat panel).
//
// The operator is that of siddon.cu (siddonCone.cu:12-74, siddon.cu:104-332 of
// the reference): prj(u, v) = sum over voxels of the length of the ray inside
// the voxel times its value, and its transpose.  In an upright view the rays of
// one detector column u lie above one line in the x-y plane and differ only in
// their z: along the line, alpha in [0, 1] from the source to the panel, ray v
// is at z = zs + alpha (k0 + v kv), in voxels.  So the x-y walk (which pixel
// columns the line crosses, between which alphas) is computed once per detector
// column instead of once per ray, and within a pixel column the rays' voxels
// follow from z alone.  Neither kernel has a serial chain of crossings, and the
// back projection is a gather without atomics.
//
//  * view_setup_kernel decides per view (on the device: the geometry arrays
//    are device memory) and lists the views that are not upright; siddon.cu's
//    ray-driven kernels take those.
//  * columns_fp_kernel: half a warp per detector column, lanes over the rows.
//  * columns_bp_kernel: one thread per pixel column, gathering from running
//    sums of the detector columns (columns_prefix_kernel).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "siddon_columns.cuh"

namespace ctp {

namespace {

// floor (and ceil, below) by one directed rounding: x + 1.5*2^23 holds the integer in
// the low mantissa bits (for |x| < 2^22; further out the bits still grow with
// x, so clamps of the integer stay right, and NaN clamps to the high end).
constexpr float kMagic = 12582912.0f;
constexpr int kMagicBits = 0x4B400000;

__device__ __forceinline__ int floor_bits(float x) { return __float_as_int(__fadd_rd(x, kMagic)); }

// Whether a detector column's line runs along a grid plane of one axis (within
// 1e-5 voxels of it from the source, s, to the panel, s + d0 + iu du).  To which
// side such rays belong is decided ray by ray, where each enters the grid
// (siddon.cu init_ray: steps below 1e-6 count as none), as for the middle column
// of an odd detector over an even grid at 0, 90, 180 and 270 degrees.
__device__ __forceinline__ bool along_plane(double s, double d0, double du, int nu) {
    const double at = rint(-d0 / du);
    if (!(at >= 0.0 && at < nu)) return false;
    const double d = fabs(d0 + at * du);
    return d < 1e-5 && fabs(s - rint(s)) < 1e-5 + d;
}

// The same for a detector row at the source's height, z by z: the kernels below
// take z in FP32, and a ray that hardly rises near a plane would lie on the side
// that the rounding says.  (Exactly level on exactly a plane, as in the middle row
// of a circular scan, all agree; the lowest plane is at 0, where FP32 tells every
// side.)
__device__ __forceinline__ bool level_at_plane(double zs, double k0, double kv, int nv, int nz) {
    const double at = rint(-k0 / kv);
    if (!(at >= 0.0 && at < nv)) return false;
    const double plane = rint(zs), d = fabs(k0 + at * kv), off = fabs(zs - plane);
    if (!(plane >= 0.0 && plane <= nz) || (off == 0.0 && d < 1e-12)) return false;
    const double rounding = plane > 0.0 ? 2.4e-7 * (nz + 1.0) : 0.0;  // 2^-22 of the largest z
    return d < 1e-3 && off < rounding + d;
}

// One block.  Upright: v along z, u across z, and every corner of the grid at
// alpha in (1e-3, 1]: the source outside the grid with the grid in front of
// it and before the panel, so that no ray ends inside the grid; and no line or
// row along a grid plane.  rows_up: rows that go down are counted from the other
// end of the panel.
__global__ void __launch_bounds__(256) view_setup_kernel(UprightView* __restrict__ out, int* __restrict__ rest,
                                                         const float* __restrict__ dc, const float* __restrict__ du_,
                                                         const float* __restrict__ dv_, const float* __restrict__ sr,
                                                         int nview, Grid g, Det d, int rows_up) {
    __shared__ int n_rest;
    if (threadIdx.x == 0) n_rest = 0;
    __syncthreads();
    for (int view = threadIdx.x; view < nview; view += blockDim.x) {
        const double idx = 1.0 / (double)g.dx, idy = 1.0 / (double)g.dy, idz = 1.0 / (double)g.dz;
        const double u0 = (-(double)d.off_u - (d.nu - 1) / 2.0) * d.du, v0 = (-(double)d.off_v - (d.nv - 1) / 2.0) * d.dv;
        UprightView w;
        w.sx = ((double)sr[view * 3] - g.cx) * idx + 0.5 * g.nx;
        w.sy = ((double)sr[view * 3 + 1] - g.cy) * idy + 0.5 * g.ny;
        w.zs = ((double)sr[view * 3 + 2] - g.cz) * idz + 0.5 * g.nz;
        const double Ux = du_[view * 3], Uy = du_[view * 3 + 1], Uz = du_[view * 3 + 2];
        const double Vx = dv_[view * 3], Vy = dv_[view * 3 + 1], Vz = dv_[view * 3 + 2];
        w.ux = Ux * d.du * idx;
        w.uy = Uy * d.du * idy;
        w.dx0 = ((double)dc[view * 3] + Ux * u0 - sr[view * 3]) * idx;
        w.dy0 = ((double)dc[view * 3 + 1] + Uy * u0 - sr[view * 3 + 1]) * idy;
        w.k0 = ((double)dc[view * 3 + 2] + Vz * v0 - sr[view * 3 + 2]) * idz;
        w.kv = Vz * d.dv * idz;
        w.det = w.ux * w.dy0 - w.uy * w.dx0;
        bool up = Vx == 0 && Vy == 0 && Uz == 0 && w.kv != 0 && isfinite(w.kv) && isfinite(w.k0) && isfinite(w.zs) &&
                  w.det != 0 && isfinite(w.det);
        const double px[2] = {0.0 - w.sx, g.nx - w.sx}, py[2] = {0.0 - w.sy, g.ny - w.sy};
        for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2; ++b) {
                const double alpha = (w.ux * py[b] - w.uy * px[a]) / w.det;
                up = up && alpha > 1e-3 && alpha <= 1.0;
            }
        up = up && !along_plane(w.sx, w.dx0, w.ux, d.nu) && !along_plane(w.sy, w.dy0, w.uy, d.nu) &&
             !level_at_plane(w.zs, w.k0, w.kv, d.nv, g.nz);
        w.upright = up ? 1 : 0;
        w.turned = rows_up && w.kv < 0 ? 1 : 0;
        if (w.turned) {
            w.k0 += (d.nv - 1) * w.kv;
            w.kv = -w.kv;
        }
        out[view] = w;
        if (!up) rest[1 + atomicAdd(&n_rest, 1)] = view;
    }
    __syncthreads();
    if (threadIdx.x == 0) rest[0] = n_rest;
}

// Length of the ray to cell (iu, iv), mm.
__device__ __forceinline__ double xy_length2(const UprightView& w, int iu, const Grid& g) {
    const double x = (w.dx0 + iu * w.ux) * g.dx, y = (w.dy0 + iu * w.uy) * g.dy;
    return x * x + y * y;
}

// ---------------------------------------------------------------------------
// Forward projection.

// Zero cells below and above each column of the z-first copy.
constexpr int kPadZ = 4;

// [b][z][y][x] -> [b][y][x][kPadZ + z] with kPadZ zero cells below and above
// each column (pitch nz + 2 kPadZ), through 32 x 32 tiles of one y; the first
// block of a batch item also writes the zero column past the end.
template <typename T>
__global__ void __launch_bounds__(256) to_columns_kernel(T* __restrict__ out, const T* __restrict__ in, int nx, int ny,
                                                         int nz, size_t out_item) {
    __shared__ T t[32][33];
    const int x0 = blockIdx.x * 32, y = blockIdx.y;
    const int nzt = (nz + 31) / 32;
    const int z0 = (blockIdx.z % nzt) * 32, b = blockIdx.z / nzt;
    const int pitch = nz + 2 * kPadZ;
    const T* src = in + (size_t)b * nx * ny * nz;
    T* dst = out + (size_t)b * out_item;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int z = z0 + k, x = x0 + threadIdx.x;
        if (z < nz && x < nx) t[k][threadIdx.x] = src[((size_t)z * ny + y) * nx + x];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int x = x0 + k, z = z0 + threadIdx.x;
        if (x >= nx) continue;
        T* col = dst + ((size_t)y * nx + x) * pitch;
        if (z < nz) col[z + kPadZ] = t[threadIdx.x][k];
        if (z0 == 0 && threadIdx.x < kPadZ) col[threadIdx.x] = (T)0.f;
        if (z0 + 32 >= nz && threadIdx.x < kPadZ) col[nz + kPadZ + threadIdx.x] = (T)0.f;
    }
    if (x0 == 0 && y == 0 && z0 == 0)
        for (int k = threadIdx.y * 32 + threadIdx.x; k < pitch; k += 256)
            dst[(size_t)nx * ny * pitch + k] = (T)0.f;
}

constexpr int kFpSlabs = 32;   // slabs of the main axis per list chunk
constexpr int kFpCols = 2;     // detector columns per warp (16 lanes each)
constexpr int kFpUnroll = 4;   // list entries in flight

// x-y line of one detector column: main axis m (x or y), other axis o.
struct ColumnLine {
    double sm, so;  // source
    double dm, dO;  // direction
    double im, io;  // reciprocals
    int xm;         // main axis is x
    int i0, i1;     // slabs, in the ray's order, where the line may be within the grid
};

// The element of a column (at base, already moved back by the bits of cell 0)
// that the bits of a rounded z name: one wide multiply-add.
template <typename Tin>
__device__ __forceinline__ float column_at(unsigned long long base, int bits) {
    unsigned long long a;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(bits), "n"((int)sizeof(Tin)), "l"(base));
    return ldf(reinterpret_cast<const Tin*>(a));
}

// A chunk of pixel columns for N rows of a lane (row i at z = fma(alpha, k[i],
// zs[i])): the segments that stay in one voxel; those that cross z planes are
// noted in split (bits of the list's entries).  CLAMP: rows may leave the
// padded columns.
template <int N, bool CLAMP, typename Tin>
__device__ __forceinline__ void columns_fp_chunk(const float4* L, int len, float as, const float (&k)[N],
                                                 const float (&zs)[N], float (&acc)[N], unsigned (&split)[2][N],
                                                 const Tin* __restrict__ vol, int pitch) {
    int m[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        m[r] = floor_bits(fmaf(as, k[r], zs[r]));
        split[0][r] = split[1][r] = 0;
    }
    const unsigned long long base0 =
        reinterpret_cast<unsigned long long>(vol) - (unsigned long long)(kMagicBits - kPadZ) * sizeof(Tin);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        unsigned bit = 1;
        const int q1 = min(len, (h + 1) * 32);
#pragma unroll kFpUnroll
        for (int q = h * 32; q < q1; ++q) {
            const float4 e = L[q];
            const unsigned long long col = base0 + (unsigned long long)(unsigned)__float_as_int(e.z) * sizeof(Tin);
#pragma unroll
            for (int r = 0; r < N; ++r) {
                const int m1 = floor_bits(fmaf(e.x, k[r], zs[r]));
                const int at = CLAMP ? max(min(m1, kMagicBits - kPadZ + pitch - 1), kMagicBits - kPadZ) : m1;
                const float f = column_at<Tin>(col, at);
                if (m1 == m[r]) acc[r] = fmaf(e.y, f, acc[r]);
                else split[h][r] |= bit;
                m[r] = m1;
            }
            bit <<= 1;
        }
    }
}

// Rows first .. first + N - 1 of a lane over one chunk: rows outside the volume
// for the whole chunk are parked in a zero cell, nothing is done when the whole
// warp's are, and the clamps are left out when the others stay within the
// padded columns (z is monotonic along the ray).
template <int N, int R, typename Tin>
__device__ __forceinline__ void columns_fp_rows(int first, const float4* L, int len, float as, float ae, float zs,
                                                const float (&k)[R], float (&acc)[R], unsigned (&split)[2][R],
                                                const Tin* __restrict__ vol, int nz) {
    float kk[N], zz[N], sum[N];
    unsigned sp[2][N];
    bool need = false, clamp = false;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        kk[r] = k[first + r];
        zz[r] = zs;
        sum[r] = 0.f;
        const float za = fmaf(as, kk[r], zs), zb = fmaf(ae, kk[r], zs);
        const float lo = fminf(za, zb), hi = fmaxf(za, zb);
        if (!(hi >= 0.f && lo < (float)nz)) {
            kk[r] = 0.f;
            zz[r] = -0.5f;
        } else {
            need = true;
            clamp |= !(lo >= (float)(1 - kPadZ) && hi < (float)(nz + kPadZ - 1));
        }
        split[0][first + r] = split[1][first + r] = 0;
    }
    if (!__any_sync(0xffffffffu, need)) return;
    if (__any_sync(0xffffffffu, clamp))
        columns_fp_chunk<N, true>(L, len, as, kk, zz, sum, sp, vol, nz + 2 * kPadZ);
    else
        columns_fp_chunk<N, false>(L, len, as, kk, zz, sum, sp, vol, nz + 2 * kPadZ);
#pragma unroll
    for (int r = 0; r < N; ++r) {
        acc[first + r] += sum[r];
        split[0][first + r] = sp[0][r];
        split[1][first + r] = sp[1][r];
    }
}

// The segments of one chunk that cross z planes (about 1% of them, but some
// lane's in most steps of the loop above, so they are split here, each lane
// taking its own): a part for each cell, cells outside the volume being zero.
template <int R, typename Tin>
__device__ __forceinline__ void columns_fp_split(const float4* L, float as, float zs, const float (&k)[R],
                                                 float (&acc)[R], unsigned (&split)[2][R],
                                                 const Tin* __restrict__ vol, int pitch) {
    auto cell = [&](float z) { return max(min(floor_bits(z) - (kMagicBits - kPadZ), pitch - 1), 0); };
    for (;;) {
        unsigned bits = 0;
        int at = 0;
        float kr = 0.f;
#pragma unroll
        for (int i = 0; i < 2 * R; ++i)
            if (bits == 0 && split[i / R][i % R] != 0) {
                bits = split[i / R][i % R];
                at = i;
                kr = k[i % R];
            }
        if (bits == 0) break;
        const int q = __ffs(bits) - 1 + (at >= R ? 32 : 0);
        const float4 e = L[q];
        const float z0 = fmaf(q > 0 ? L[q - 1].x : as, kr, zs), z1 = fmaf(e.x, kr, zs);
        const Tin* col = vol + __float_as_int(e.z);
        int i = cell(z0);
        const int ib = cell(z1), step = ib > i ? 1 : -1;
        const float inv = __fdividef(1.f, z1 - z0);
        float t = 0.f, sum = 0.f;
        for (; i != ib; i += step) {
            // the plane between cells i and i + step (cell i spans z in [i, i + 1] - kPadZ)
            const float t1 = fminf(fmaxf(((float)((step > 0 ? i + 1 : i) - kPadZ) - z0) * inv, t), 1.f);
            if (t1 > t) sum = fmaf(t1 - t, ldf(col + i), sum);  // (no 0 * infinity)
            t = t1;
        }
        if (t < 1.f) sum = fmaf(1.f - t, ldf(col + ib), sum);
        sum *= e.y;
#pragma unroll
        for (int j = 0; j < 2 * R; ++j)
            if (at == j) {
                split[j / R][j % R] = bits & (bits - 1);
                acc[j % R] += sum;
            }
    }
}

// One warp takes two neighbouring detector columns of a view, 16 lanes each;
// lane l of a half has the rows l, l + 16, ... (R of them).  The x-y line of a
// column is walked slab by slab of its main axis: in a slab it meets at most
// one plane of the other axis, so each lane finds the one or two pixel columns
// of one slab on its own, in FP64, and the warp compacts 32 slabs' entries
// (alpha at the exit, the alpha spanned, the column's offset) into shared
// memory.  Then every lane runs down the list for its rows, two at a time: z
// at the exit by one FP32 multiply-add, the voxel by a directed rounding, one
// load and one multiply-add, all independent from entry to entry
// (columns_fp_chunk).  The rows of a warp read neighbouring z of one column:
// the volume is copied z first (to_columns_kernel).
//
// Bound by issue (two thirds of the slots) and by the voxel loads' latency: a
// segment costs about ten instructions, most of them on the integer and
// multiply-add pipes.  64 x 512 x 512 voxels onto 360 views of 736 x 64 cells:
// 9.57 ms ray by ray (siddon_fp_kernel), 5.23 ms here.  Branching to split a
// segment inside the list's loop keeps one load in flight: 24.8 ms.
template <int R, typename Tin, typename Tout>
__global__ void __launch_bounds__(256, 5) columns_fp_kernel(Tout* __restrict__ prj, const Tin* __restrict__ vol,
                                                            const UprightView* __restrict__ views, int nview, Grid g,
                                                            Det d, size_t item, int rows, int accumulate) {
    __shared__ float4 s_list[8][kFpCols][2 * kFpSlabs];
    __shared__ ColumnLine s_line[8][kFpCols];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int view = blockIdx.z % nview, b = blockIdx.z / nview;
    if (!views[view].upright) return;
    const int u0 = (blockIdx.x * 8 + warp) * kFpCols;
    if (u0 >= d.nu) return;
    const int half = lane >> 4, hl = lane & 15;
    const int v0 = blockIdx.y * rows;  // this block's rows
    const int pitch = g.nz + 2 * kPadZ;
    const int zero_col = g.nx * g.ny * pitch;
    vol += (size_t)b * item;

    // rows of this lane
    float zs, k[R], acc[R];
    {
        const UprightView& w = views[view];
        zs = (float)w.zs;
        const double k0 = w.k0, kv = w.kv;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            k[r] = (float)(k0 + (double)(v0 + hl + 16 * r) * kv);
            acc[r] = 0.f;
        }
        if (lane < kFpCols) {
            const int iu = min(u0 + lane, d.nu - 1);
            const double dx = w.dx0 + iu * w.ux, dy = w.dy0 + iu * w.uy;
            ColumnLine c;
            c.xm = fabs(dx) >= fabs(dy);
            c.dm = c.xm ? dx : dy;
            c.dO = c.xm ? dy : dx;
            c.sm = c.xm ? w.sx : w.sy;
            c.so = c.xm ? w.sy : w.sx;
            c.im = 1.0 / c.dm;
            c.io = 1.0 / c.dO;
            const int n = c.xm ? g.nx : g.ny, no = c.xm ? g.ny : g.nx;
            double a0 = -1e30, a1 = 1e30;
            if (c.dO != 0) {
                const double p = (0.0 - c.so) * c.io, q = (no - c.so) * c.io;
                a0 = fmin(p, q);
                a1 = fmax(p, q);
            } else if (c.so < 0 || c.so >= no) {
                a1 = -1e30;
            }
            const double e0 = c.sm + a0 * c.dm, e1 = c.sm + a1 * c.dm;
            const double o0 = c.dm > 0 ? e0 : n - e0, o1 = c.dm > 0 ? e1 : n - e1;
            c.i0 = (int)fmin(fmax(floor(o0) - 1.0, 0.0), (double)n);
            c.i1 = (int)fmin(fmax(ceil(o1) + 1.0, 0.0), (double)n);
            s_line[warp][lane] = c;
        }
    }
    __syncwarp();
    int chunks = 0;
#pragma unroll
    for (int c = 0; c < kFpCols; ++c)
        chunks = max(chunks, (s_line[warp][c].i1 - s_line[warp][c].i0 + kFpSlabs - 1) / kFpSlabs);

    for (int ch = 0; ch < chunks; ++ch) {
        int cnt[kFpCols];
        float astart[kFpCols];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kFpCols; ++c) {
            const ColumnLine& ln = s_line[warp][c];
            const int n = ln.xm ? g.nx : g.ny, no = ln.xm ? g.ny : g.nx;
            const int o = ln.i0 + ch * kFpSlabs + lane;
            const bool in = o < ln.i1;
            const int slab = ln.dm > 0 ? o : n - 1 - o;
            const int pin = ln.dm > 0 ? slab : slab + 1, pout = ln.dm > 0 ? slab + 1 : slab;
            const double aa = (pin - ln.sm) * ln.im, ab = (pout - ln.sm) * ln.im;
            const double ya = ln.so + aa * ln.dO, yb = ln.so + ab * ln.dO;
            int ja = (int)floor(fmin(fmax(ya, -2.0), no + 1.0)), jb = (int)floor(fmin(fmax(yb, -2.0), no + 1.0));
            // from corner to corner (45 degrees) rounding may show the cells on both sides of the one crossed
            if (abs(jb - ja) > 1) ja = jb = (ja + jb) / 2;
            double ac = ab;
            if (ja != jb) ac = fmin(fmax((max(ja, jb) - ln.so) * ln.io, aa), ab);
            const bool f1 = in && ja >= 0 && ja < no, f2 = in && ja != jb && jb >= 0 && jb < no;
            const unsigned b1 = __ballot_sync(0xffffffffu, f1), b2 = __ballot_sync(0xffffffffu, f2);
            const unsigned below = (1u << lane) - 1u;
            const int at = __popc(b1 & below) + __popc(b2 & below);
            const int c1 = (ln.xm ? ja * g.nx + slab : slab * g.nx + ja) * pitch;
            const int c2 = (ln.xm ? jb * g.nx + slab : slab * g.nx + jb) * pitch;
            if (f1) s_list[warp][c][at] = make_float4((float)ac, (float)(ac - aa), __int_as_float(c1), 0.f);
            if (f2) s_list[warp][c][at + (f1 ? 1 : 0)] = make_float4((float)ab, (float)(ab - ac), __int_as_float(c2), 0.f);
            cnt[c] = __popc(b1) + __popc(b2);
            // alpha where the chunk's first entry starts
            const unsigned any = b1 | b2;
            const int first = any ? __ffs(any) - 1 : 0;
            astart[c] = (float)__shfl_sync(0xffffffffu, f1 ? aa : ac, first);
        }
        const int len = max(cnt[0], cnt[1]);
        // the shorter list is filled up with empty segments in the zero column,
        // at its own last alpha
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kFpCols; ++c) {
            const float at = cnt[c] > 0 ? s_list[warp][c][cnt[c] - 1].x : astart[c];
            for (int q = cnt[c] + lane; q < len; q += 32)
                s_list[warp][c][q] = make_float4(at, 0.f, __int_as_float(zero_col), 0.f);
        }
        __syncwarp();
        const float4* L = s_list[warp][half];
        if (len == 0) continue;
        const float as = half ? astart[1] : astart[0], ae = L[len - 1].x;
        unsigned split[2][R];
        columns_fp_rows<(R >= 2 ? 2 : 1), R>(0, L, len, as, ae, zs, k, acc, split, vol, g.nz);
        if constexpr (R == 3) columns_fp_rows<1, R>(2, L, len, as, ae, zs, k, acc, split, vol, g.nz);
        if constexpr (R == 4) columns_fp_rows<2, R>(2, L, len, as, ae, zs, k, acc, split, vol, g.nz);
        columns_fp_split<R>(L, as, zs, k, acc, split, vol, pitch);
    }
    const int iu = u0 + half;
    if (iu >= d.nu) return;
    const UprightView& w = views[view];
    const double l2 = xy_length2(w, iu, g);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int iv = v0 + hl + 16 * r;
        if (hl + 16 * r >= rows || iv >= d.nv) continue;
        const double dz = (w.k0 + iv * w.kv) * g.dz;
        Tout* o = prj + (((size_t)b * nview + view) * d.nv + iv) * d.nu + iu;
        stf(o, (accumulate ? rdf(o) : 0.f) + acc[r] * (float)sqrt(l2 + dz * dz));
    }
}

// ---------------------------------------------------------------------------
// Back projection.

// Running sums of the detector columns restart every kSumStep rows and run over
// kSumRows of them, so that any kBpRows + 1 of them in a row lie within one run
// and no sum holds more than kSumRows cells, however tall the detector.
constexpr int kSumStep = 32;
constexpr int kSumRows = 96;
__host__ __device__ __forceinline__ int sum_runs(int nv) {
    return nv <= kSumRows ? 1 : (nv - kSumRows + kSumStep - 1) / kSumStep + 1;
}
// Rows of sums of one view: the runs one after the other, kSumRows + 1 each.
__host__ __device__ __forceinline__ int sum_rows(int nv) {
    return nv <= kSumRows ? nv + 1 : sum_runs(nv) * (kSumRows + 1);
}

// Running sums over the rows of every detector column of the upright views,
// each cell times its ray's length: P[b][view][run][k][iu] = sum over the cells
// from the run's middle to k (negative before it: only differences are used, and
// these numbers are half as large), in FP64, stored FP32 (row pitch a multiple of
// 4 cells); and per column the reciprocal steps of its x-y line.  stats[b][view][run][block]: the
// sum of the cells' magnitudes (each cell once) and the largest sum's, infinite
// when a cell is not finite; zeros for views that are not upright.
template <typename Tin>
__global__ void __launch_bounds__(128) columns_prefix_kernel(float* __restrict__ P, double2* __restrict__ inv,
                                                             float2* __restrict__ stats, const Tin* __restrict__ prj,
                                                             const UprightView* __restrict__ views, int nview, int view0,
                                                             int nviews, Grid g, Det d, int pitch) {
    __shared__ float2 s_stat[4];
    const int iu = blockIdx.x * 128 + threadIdx.x;
    const int runs = sum_runs(d.nv), vi = blockIdx.y, run_i = blockIdx.z % runs, b = blockIdx.z / runs;
    const int view = view0 + vi;
    float mag = 0.f, top = 0.f;
    if (iu < d.nu && views[view].upright) {
        const UprightView& w = views[view];
        if (blockIdx.z == 0) {
            // steps below 1e-6 voxels over the whole ray count as none (siddon.cu
            // kEps): marked by an infinite reciprocal
            const double dx = w.dx0 + iu * w.ux, dy = w.dy0 + iu * w.uy;
            inv[(size_t)vi * d.nu + iu] = make_double2(fabs(dx) < 1e-6 ? INFINITY : 1.0 / dx,
                                                       fabs(dy) < 1e-6 ? INFINITY : 1.0 / dy);
        }
        const float l2 = (float)xy_length2(w, iu, g);
        const float k0 = (float)(w.k0 * g.dz), kv = (float)(w.kv * g.dz);
        const int va = run_i * kSumStep, rows = min(kSumRows, d.nv - va);
        const int own = run_i + 1 < runs ? kSumStep : rows;  // rows that the next run does not start in
        const Tin* src = prj + (((size_t)b * nview + view) * d.nv) * d.nu + iu;
        float* out = P + (((size_t)b * nviews + vi) * sum_rows(d.nv) + run_i * (kSumRows + 1)) * pitch + iu;
        auto cell = [&](int v) {
            const float z = fmaf((float)(va + v), kv, k0);
            const int row = w.turned ? d.nv - 1 - (va + v) : va + v;
            const float p = ldf(src + (size_t)row * d.nu) * sqrtf(fmaf(z, z, l2));
            if (v < own) mag += fabsf(p);
            return (double)p;
        };
        auto put = [&](int k, double sum) {
            const float f = (float)sum;
            top = fmaxf(top, isfinite(f) ? fabsf(f) : INFINITY);
            out[(size_t)k * pitch] = f;
        };
        const int mid = rows / 2;
        double run = 0.0;
        put(mid, 0.0);
#pragma unroll 8
        for (int v = mid; v < rows; ++v) {
            run += cell(v);
            put(v + 1, run);
        }
        run = 0.0;
#pragma unroll 8
        for (int v = mid - 1; v >= 0; --v) {
            run -= cell(v);
            put(v, run);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mag += __shfl_xor_sync(0xffffffffu, mag, o);
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if ((threadIdx.x & 31) == 0) s_stat[threadIdx.x >> 5] = make_float2(mag, top);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 4; ++k) {
            mag += s_stat[k].x;
            top = fmaxf(top, s_stat[k].y);
        }
        stats[(((size_t)b * nviews + vi) * runs + run_i) * gridDim.x + blockIdx.x] = make_float2(mag, top);
    }
}

// Views that the running sums do not serve go to the ray-driven list instead: a
// sum that is not finite would spread over the column, and one far above the
// other cells would cost them their bits.  A voxel's sum is a difference of two
// FP32 numbers of the largest sum's size, so it may be off by 2^-24 of that in
// one view; kOutlier times the cells of half a run at their mean magnitude (over
// the views at hand) bounds this to 2^-24 x 32 x 48 = 1e-4 of a mean cell a view,
// 2e-7 of a voxel that 360 views meet with a cell or two each.  Sums reach
// one over the share of the columns that the object covers: 3% stay.
// One block; sums in a fixed order.
constexpr float kOutlier = 32.f;
__global__ void __launch_bounds__(256) retire_views_kernel(UprightView* __restrict__ views, int* __restrict__ rest,
                                                           const float2* __restrict__ stats, int view0, int nviews,
                                                           int nbatch, int per_view, Det d) {
    __shared__ float s_mag[256];
    __shared__ int s_up[256];
    float mag = 0.f;
    int up = 0;
    for (int vi = threadIdx.x; vi < nviews; vi += blockDim.x) {
        if (!views[view0 + vi].upright) continue;
        ++up;
        for (int b = 0; b < nbatch; ++b)
            for (int k = 0; k < per_view; ++k) {
                const float2 t = stats[((size_t)b * nviews + vi) * per_view + k];
                if (isfinite(t.y)) mag += t.x;
            }
    }
    s_mag[threadIdx.x] = mag;
    s_up[threadIdx.x] = up;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            s_mag[threadIdx.x] += s_mag[threadIdx.x + o];
            s_up[threadIdx.x] += s_up[threadIdx.x + o];
        }
        __syncthreads();
    }
    const float mean = s_mag[0] / ((float)max(s_up[0], 1) * (float)nbatch * (float)d.nu * (float)d.nv);
    const float most = kOutlier * 0.5f * (float)min(d.nv, kSumRows) * mean;
    for (int vi = threadIdx.x; vi < nviews; vi += blockDim.x) {
        if (!views[view0 + vi].upright) continue;
        bool keep = true;
        for (int b = 0; b < nbatch; ++b)
            for (int k = 0; k < per_view; ++k) keep = keep && stats[((size_t)b * nviews + vi) * per_view + k].y <= most;
        if (!keep) {
            views[view0 + vi].upright = 0;
            rest[1 + atomicAdd(rest, 1)] = view0 + vi;
        }
    }
}

constexpr int kBpTile = 16;    // pixel columns per side of a block's tile
constexpr int kBpZ = 32;       // z accumulators per thread
constexpr int kBpGroup = 8;    // z cells per group (skipped when no ray of the view reaches it)
constexpr int kBpWin = 64;     // detector columns of a staged window (a row spans all banks twice)
constexpr int kBpRows = 64;    // rows of a staged window: kBpRows + 1 running sums per column
constexpr int kBpStep = 2;     // views staged and taken between two barriers
constexpr int kBpViews = 20;   // views whose constants are computed together (at most a warp's lanes)
constexpr int kBpTerm = 60;    // views added up in registers before the sums join the volume (whole kBpViews)
// dynamic shared memory of a block, in floats: two buffers of staged windows,
// and the split rows' sums, one per plane and thread
constexpr int kBpWindow = (kBpRows + 1) * kBpWin;
constexpr int kBpStageFloats = 2 * kBpStep * kBpWindow;
constexpr int kBpSplitFloats = (kBpZ + 1) * 256;

// Constants of one view for one tile and z range.  The pixel centre (kx, ky)
// of the tile sees the detector column u = N / D (from the window's first
// cell) at alpha = ar D, N and D linear in kx, ky (both from cross products of
// the x-y geometry).
struct BpView {
    float n0, n1, n2, w0f, w1, w2;  // N = n0 + n1 kx + n2 ky, D = w0f + w1 kx + w2 ky
    float ar;                       // alpha of the tile's centre (alphas are kept relative to it)
    float zz0;                      // the z range's first plane minus the source's z
    float vc;                       // row coordinate of the source's z plane, from the staged rows' base
    float ikv;                      // 1 / kv
    float kbf, kvf;                 // kb and kv in FP32
    double bx, by;                  // tile origin minus the source, x and y
    double zd, kb, kv;              // zz0 in FP64; z rise over alpha 0 .. 1 of the staged rows: kb + k kv
    int c1;                         // cells of the window
    int first;                      // first cell of the window
    int row, nrow;                  // first running sum used, and how many
    int g0, g1;                     // groups of z cells that rays reach, [g0, g1)
    int vi;                         // view within the launch's views
};

// The x-y line of a detector column over one tile: alpha (relative to ar) of its
// first x and y planes and per pixel, in FP32; and in FP64 the difference between
// the lower x and the lower y plane of the tile's first pixel, and its steps.
struct BpLine {
    float x0, dx, y0, dy;
    double e, ex, ey;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ float lds_f32(unsigned addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// a * b + c rounded up and clamped to [0, 1] (NaN to 0): above an integer stays
// above it, for the ceiling that follows.
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float y;
    asm("fma.rp.sat.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

// The constants of view w for the tile at (tx0, ty0) and nz planes from z0;
// false when none of its rays comes near them.
__device__ __forceinline__ bool bp_view(const UprightView& w, int tx0, int ty0, int z0, int nz, const Grid& g,
                                        const Det& d, BpView& V) {
    // cross products at pixel corners of the tile: D = U x (p - s), N = (p - s) x d0
    const double ox = tx0 - w.sx, oy = ty0 - w.sy;
    const double wx = -w.uy, wy = w.ux, nx = w.dy0, ny = -w.dx0;  // gradients of D and N
    const double D0 = w.ux * oy - w.uy * ox, N0 = ox * w.dy0 - oy * w.dx0;
    const double tw = min(kBpTile, g.nx - tx0), th = min(kBpTile, g.ny - ty0);  // the tile's part of the grid
    double amin = 1e30, amax = -1e30, umin = 1e30, umax = -1e30;
    for (int q = 0; q < 4; ++q) {
        const double x = (q & 1) * tw, y = (q >> 1) * th;
        const double D = D0 + wx * x + wy * y, N = N0 + nx * x + ny * y;
        const double a = D / w.det, u = N / D;
        amin = fmin(amin, a);
        amax = fmax(amax, a);
        umin = fmin(umin, u);
        umax = fmax(umax, u);
    }
    umin = fmax(umin, -1e8);
    umax = fmin(umax, 1e8);
    const int ufirst = (int)floor(umin) - 1, ulast = (int)ceil(umax) + 1;
    V.first = max(ufirst, 0) & ~3;
    V.c1 = min(ulast + 1, d.nu) - V.first;
    const double Dc = D0 + wx * 0.5 * tw + wy * 0.5 * th;
    V.ar = (float)(Dc / w.det);
    const double iD = 1.0 / Dc;
    // at pixel centres, u relative to the window's first cell
    const double Dp = D0 + 0.5 * (wx + wy), Np = N0 + 0.5 * (nx + ny);
    V.w0f = (float)(Dp * iD);
    V.w1 = (float)(wx * iD);
    V.w2 = (float)(wy * iD);
    V.n0 = (float)((Np - V.first * Dp) * iD);
    V.n1 = (float)((nx - V.first * wx) * iD);
    V.n2 = (float)((ny - V.first * wy) * iD);
    V.bx = ox;
    V.by = oy;
    V.zz0 = (float)(z0 - w.zs);
    V.ikv = (float)(1.0 / w.kv);
    // z reached by the rows 0 and nv - 1 over the tile's alphas
    const double ka = w.k0, kb = w.k0 + (d.nv - 1) * w.kv;
    const double klo = fmin(ka, kb), khi = fmax(ka, kb);
    const double zlo = w.zs + klo * (klo < 0 ? amax : amin), zhi = w.zs + khi * (khi > 0 ? amax : amin);
    const double q0 = floor(zlo - 1e-3) - z0, q1 = floor(zhi + 1e-3) - z0;
    V.g0 = max(0, (int)floor(fmax(q0, 0.0) / kBpGroup));
    V.g1 = q1 < 0 ? 0 : min((nz + kBpGroup - 1) / kBpGroup, (int)floor(fmin(q1, 1e6) / kBpGroup) + 1);
    // rows between the range's first and last plane
    double rlo = 1e30, rhi = -1e30;
    for (int q = 0; q < 4; ++q) {
        const double a = (q & 1) ? amax : amin;
        const double zz = ((q >> 1) ? V.g1 * kBpGroup : V.g0 * kBpGroup) + z0 - w.zs;
        const double r = (zz / a - w.k0) / w.kv;
        rlo = fmin(rlo, r);
        rhi = fmax(rhi, r);
    }
    V.row = (int)fmin(fmax(floor(rlo) - 1, 0.0), (double)d.nv);
    V.nrow = (int)fmin(fmax(ceil(rhi) + 1, 0.0), (double)d.nv) - V.row + 1;
    V.vc = (float)(-w.k0 / w.kv - V.row);
    V.zd = z0 - w.zs;
    V.kb = w.k0 + V.row * w.kv;
    V.kv = w.kv;
    V.kbf = (float)V.kb;
    V.kvf = (float)w.kv;
    return V.g0 < V.g1 && V.c1 > 0 && V.nrow > 0;
}

// Whether a view's window and rows fit the staged ones (nrow <= nv + 1 <= rows +
// 1 where the launch stages fewer rows than kBpRows).
__device__ __forceinline__ bool bp_fits(const BpView& V) { return V.c1 <= kBpWin && V.nrow <= kBpRows + 1; }

// Views that do not fit on some tile and z range (a coarse grid under a fine
// detector) go to the ray-driven list.
__global__ void __launch_bounds__(128) bp_fit_kernel(UprightView* __restrict__ views, int* __restrict__ rest, int nview,
                                                     int zper, int zchunks, Grid g, Det d) {
    const int tile = blockIdx.x * 128 + threadIdx.x, view = blockIdx.y;
    const int tiles_x = (g.nx + kBpTile - 1) / kBpTile, tiles = tiles_x * ((g.ny + kBpTile - 1) / kBpTile);
    if (tile >= tiles || !views[view].upright) return;
    const UprightView w = views[view];
    const int tx0 = (tile % tiles_x) * kBpTile, ty0 = (tile / tiles_x) * kBpTile;
    for (int zc = 0; zc < zchunks; ++zc) {
        BpView V;
        if (bp_view(w, tx0, ty0, zc * zper, min(zper, g.nz - zc * zper), g, d, V) && !bp_fits(V)) {
            if (atomicExch(&views[view].upright, 0)) rest[1 + atomicAdd(rest, 1)] = view;
            return;
        }
    }
}

// One thread per pixel column (x, y), kBpZ voxels of it in registers; a block
// owns a 16 x 16 tile of columns and runs over the views, two between barriers.
// Per view the block stages the window of running sums that the tile projects
// onto (16-byte cp.async, two buffers: the next views' copies run under these
// views' arithmetic).  Per detector column whose line crosses the pixel,
// between alphas aA and aB:
//   the rays of the column below the plane z at alpha a are the rows below
//   v(z, a) = (z - zs) / (a kv) - k0 / kv (kv > 0: view_setup_kernel), so the sum of the rays below z is
//   the running sum at ceil(v), the same at both ends unless a row passes
//   through the plane inside the pixel; such rows count with the part of the
//   segment below (noted in a bit mask, added after the planes' loop).  The
//   voxel's sum is the difference between its two planes, times aB - aA.
// So a voxel costs one table read per crossing line, whatever the number of
// rows that meet it, and nothing is scattered.  Alphas are relative to the
// tile's centre, from per-line coefficients rounded from FP64.  A chord is a
// difference of two of them, so it is taken from the FP64 distance between the
// pixel's x and y planes instead (two multiply-adds per pixel and line), and the
// sums of kBpTerm views at a time join the volume.  64 x 192 x 192 voxels, 180
// views: 4.64e-7 from 64 bits (ray by ray 4.64e-7; with chords of FP32 alphas,
// 1e-6 of a voxel each, 4.9e-7, and with one sum over the views besides 5.15e-7),
// for 8% of the time.
//
// Bound by issue: per plane and crossing line two saturating multiply-adds, two
// directed roundings, a compare and a read.  The same volume and views: 14.9 ms
// ray by ray (siddon_bp_kernel's atomics), 6.40 ms here.  Measured and not taken,
// same volume, when the kernel took 5.96 ms (chords of FP32 alphas, one sum over
// the views): columns as the rows of the staged window (bank conflicts) 6.74 ms;
// one view between barriers 6.10; three blocks per SM at 80 registers 6.56; two
// threads per pixel, every other line each, 9.2.
template <bool ATOMIC>
__global__ void __launch_bounds__(256, 2) columns_bp_kernel(float* __restrict__ img, const float* __restrict__ P,
                                                            const double2* __restrict__ inv,
                                                            const UprightView* __restrict__ views, int view0,
                                                            int nviews, int vper, Grid g, Det d, int pitch, int rows,
                                                            int zper, int zchunks) {
    extern __shared__ float4 s_raw[];
    float* s_P = reinterpret_cast<float*>(s_raw);     // [2][kBpStep][kBpRows + 1][kBpWin]
    float* s_split = s_P + kBpStageFloats;            // [kBpZ + 1][256] sums of the split rows, per plane and thread
    __shared__ BpLine s_line[2][kBpStep][kBpWin];
    __shared__ float2 s_rowz[2][kBpStep][kBpRows + 1];  // staged rows' z at alpha ar from the first plane, see row_z
    __shared__ BpView s_view[kBpViews];
    __shared__ int s_n;
    const int tid = threadIdx.x;
    const int tiles_x = (g.nx + kBpTile - 1) / kBpTile;
    const int tx0 = (blockIdx.x % tiles_x) * kBpTile, ty0 = (blockIdx.x / tiles_x) * kBpTile;
    const int zc = blockIdx.y % zchunks, part = blockIdx.y / zchunks;
    const int b = blockIdx.z;
    const int z0 = zc * zper, nz = min(zper, g.nz - z0);
    const int tx = tid & (kBpTile - 1), ty = tid / kBpTile;
    const float kx = (float)tx, ky = (float)ty;
    const double dkx = tx, dky = ty;
    const float* Pb = P + (size_t)b * nviews * sum_rows(d.nv) * pitch;

    float acc[kBpZ];
#pragma unroll
    for (int q = 0; q < kBpZ; ++q) acc[q] = 0.f;
    for (int q = 0; q <= kBpZ; ++q) s_split[q * 256 + tid] = 0.f;

    // coefficients of a line: alphas of the tile's first planes (relative to
    // ar) and per pixel.  A line that keeps its x (or y) is within the planes
    // of its own pixel for every alpha, and of no other.
    auto line = [&](const BpView& V, int c) {
        const double2 q = inv[(size_t)V.vi * d.nu + V.first + c];
        double x0 = V.bx * q.x - (double)V.ar, dx = q.x, y0 = V.by * q.y - (double)V.ar, dy = q.y;
        if (isinf(q.x) || isinf(q.y)) {
            const UprightView& w = views[view0 + V.vi];
            const int iu = V.first + c;
            const double a = V.ar;
            if (isinf(q.x)) {
                dx = 1024.0;
                x0 = -1024.0 * ((int)floor(w.sx + a * (w.dx0 + iu * w.ux)) - tx0) - 512.0;
            }
            if (isinf(q.y)) {
                dy = 1024.0;
                y0 = -1024.0 * ((int)floor(w.sy + a * (w.dy0 + iu * w.uy)) - ty0) - 512.0;
            }
        }
        BpLine L;
        L.x0 = (float)x0;
        L.dx = (float)dx;
        L.y0 = (float)y0;
        L.dy = (float)dy;
        L.e = (x0 + fmin(dx, 0.0)) - (y0 + fmin(dy, 0.0));
        L.ex = dx;
        L.ey = dy;
        return L;
    };

    // z of running-sum row k at the tile centre's alpha, from the z range's first
    // plane: whole planes and the rest, which stays exact where it matters
    auto row_z = [&](const BpView& V, int k) {
        const double z = fma((double)V.ar, fma((double)k, V.kv, V.kb), -V.zd);
        const double whole = fmin(fmax(rint(z), -1e6), 1e6);
        return make_float2(__int_as_float((int)whole), (float)(z - whole));
    };

    // windows, lines and rows of the views i .. of a step
    auto stage = [&](int i, int n, int buf) {
        const int lane = tid & 31, half = lane & 15;
#pragma unroll
        for (int j = 0; j < kBpStep; ++j) {
            if (i + j >= n) break;
            const BpView& V = s_view[i + j];
            float* dst = s_P + (buf * kBpStep + j) * kBpWindow + 4 * half;
            // the run of sums that the rows lie in
            const int run = min(V.row / kSumStep, sum_runs(d.nv) - 1), va = run * kSumStep;
            const float* src = Pb + ((size_t)V.vi * sum_rows(d.nv) + run * (kSumRows + 1)) * pitch + V.first + 4 * half;
            const int row = V.row - va, last = min(kSumRows, d.nv - va), c1 = V.c1;
            if (4 * half < c1)
                for (int r = 2 * (tid >> 5) + (lane >> 4); r <= rows; r += 16)
                    cp_async16(dst + r * kBpWin, src + (size_t)min(row + r, last) * pitch);
            const int c = tid - j * 64;  // (warps 0, 1 and 2, 3; rows: 4, 5 and 6, 7)
            if (c >= 0 && c < c1) s_line[buf][j][c] = line(V, c);
            const int k = tid - 128 - j * 64;
            if (k >= 0 && k < 64) s_rowz[buf][j][k] = row_z(V, k);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // Detector column c of the view V staged in buf, j against this thread's pixel.
    // A running sum is read at the column's base plus the bits of ceil(v) times
    // the row's bytes; ceil is one directed rounding, and its clamps to [0, rows]
    // come with the saturating multiply-add before it (v scaled by a power of
    // two, which rounds alike).
    const float frows = (float)rows, irows = 1.f / frows;
    auto column = [&](const BpView& V, int buf, int j, int c) {
        const BpLine& L = s_line[buf][j][c];
        const float* col = s_P + (buf * kBpStep + j) * kBpWindow + c;
        // from the lower x plane to the lower y plane, and the chord: the pixel's
        // extent along the axis that it spans, less what the other plane cuts off
        const float e = (float)fma(dkx, L.ex, fma(-dky, L.ey, L.e));
        const float wx = fabsf(L.dx), wy = fabsf(L.dy);
        const float chord = fminf(fminf(wx, wy), fminf(wx + e, wy - e));
        if (!(chord > 0.f)) return;
        const float lo = e < 0.f ? fmaf(ky, L.dy, L.y0) + fminf(L.dy, 0.f) : fmaf(kx, L.dx, L.x0) + fminf(L.dx, 0.f);
        const float aA = V.ar + lo, aB = V.ar + (lo + chord);
        const float gA = __fdividef(V.ikv, aA), gB = __fdividef(V.ikv, aB);
        const int g0 = V.g0, g1 = V.g1;
        const float zz0 = V.zz0, vc = V.vc, kbf = V.kbf, kvf = V.kvf;
        unsigned split = 0;  // planes 0 .. 31 that a row passes through inside the pixel
        bool split_top = false;
        const float gA1 = gA * irows, gB1 = gB * irows, vc1 = vc * irows;
        const unsigned at = (unsigned)__cvta_generic_to_shared(col) - (unsigned)kMagicBits * (4u * kBpWin);
        auto plane = [&](int q) {
            const float zz = zz0 + (float)q;
            const unsigned iA = __float_as_uint(__fmaf_ru(fma_sat(zz, gA1, vc1), frows, kMagic));
            const unsigned iB = __float_as_uint(__fmaf_ru(fma_sat(zz, gB1, vc1), frows, kMagic));
            if (iA != iB) {
                if (q < 32) split |= 1u << q;
                else split_top = true;
            }
            return lds_f32(at + iA * (4u * kBpWin));
        };
        float below = 0.f;
#pragma unroll
        for (int grp = 0; grp < kBpZ / kBpGroup; ++grp) {
            if (grp < g0 || grp >= g1) continue;
            float s[kBpGroup + 1];
            s[0] = grp == g0 ? plane(grp * kBpGroup) : below;
#pragma unroll
            for (int q = 1; q <= kBpGroup; ++q) s[q] = plane(grp * kBpGroup + q);
#pragma unroll
            for (int q = 0; q < kBpGroup; ++q)
                acc[grp * kBpGroup + q] = fmaf(s[q + 1] - s[q], chord, acc[grp * kBpGroup + q]);
            below = s[kBpGroup];
        }
        // rows through a plane: the part of their segment below it, relative to
        // the sum taken above, which counts them as their end A says
        while (split || split_top) {
            const int q = split ? __ffs(split) - 1 : kBpZ;
            if (split) split &= split - 1;
            else split_top = false;
            const float zz = zz0 + (float)q;
            const int kA = __float_as_int(__fmaf_ru(fma_sat(zz, gA1, vc1), frows, kMagic)) - kMagicBits;
            const int kB = __float_as_int(__fmaf_ru(fma_sat(zz, gB1, vc1), frows, kMagic)) - kMagicBits;
            // row k is at z = zs + alpha kappa: its part on A's side of the plane is
            // (z - zs - aA kappa) / ((aB - aA) kappa); the numerator cancels, so it is
            // taken from the row's z at the tile centre (row_z)
            float part = 0.f;
            const int e = max(kA, kB);
            for (int k = min(kA, kB); k < e; ++k) {  // nearly always one row
                const float2 rz = s_rowz[buf][j][k];
                const float kappa = fmaf((float)k, kvf, kbf);
                const float f = __saturatef(__fdividef(fmaf(-lo, kappa, (float)(q - __float_as_int(rz.x)) - rz.y),
                                                       chord * kappa));
                part = fmaf(col[(k + 1) * kBpWin] - col[k * kBpWin], kA > kB ? f - 1.f : 1.f - f, part);
            }
            s_split[q * 256 + tid] += part * chord;
        }
    };

    // detector columns [ca, cb] whose lines may cross this thread's pixel
    auto candidates = [&](const BpView& V, int& ca, int& cb) {
        const float D = fmaf(V.w1, kx, fmaf(V.w2, ky, V.w0f)), N = fmaf(V.n1, kx, fmaf(V.n2, ky, V.n0));
        const float uc = __fdividef(N, D);
        // half the pixel's extent on the detector: a corner's u - uc is the
        // first-order term over the D of the corner (with a margin for rounding)
        const float hw = __fdividef(0.5005f * (fabsf(fmaf(-uc, V.w1, V.n1)) + fabsf(fmaf(-uc, V.w2, V.n2))),
                                    D - 0.5f * (fabsf(V.w1) + fabsf(V.w2))) + 4e-3f;
        ca = max((int)ceilf(uc - hw), 0);
        cb = min((int)floorf(uc + hw), V.c1 - 1);
    };

    auto compute = [&](int i, int n, int buf) {
#pragma unroll 1
        for (int j = 0; j < kBpStep; ++j) {
            if (i + j >= n) break;
            const BpView& V = s_view[i + j];
            int ca, cb;
            candidates(V, ca, cb);
            for (int c = ca; c <= cb; ++c) column(V, buf, j, c);
        }
    };

    // the sums so far join the volume
    auto store = [&]() {
        int ix = tx0 + tx;
        asm volatile("" : "+r"(ix));  // (its addresses are formed here, not kept through the views)
        const int iy = ty0 + ty;
        const bool in = ix < g.nx && iy < g.ny;
        float* o = img + (((size_t)b * g.nz + z0) * g.ny + iy) * g.nx + ix;
        float below = s_split[tid];
#pragma unroll
        for (int q = 0; q < kBpZ; ++q) {
            const float above = s_split[(q + 1) * 256 + tid], sum = acc[q] + (above - below);
            if (in && q < nz) {
                if (ATOMIC)
                    atomicAdd(o, sum);
                else
                    *o += sum;
            }
            o += (size_t)g.nx * g.ny;
            s_split[q * 256 + tid] = 0.f;
            acc[q] = 0.f;
            below = above;
        }
        s_split[kBpZ * 256 + tid] = 0.f;
    };

    const int vb = part * vper, ve = min(nviews, vb + vper);
    for (int v0 = vb; v0 < ve; v0 += kBpViews) {
        if (v0 > vb && (v0 - vb) % kBpTerm == 0) store();
        __syncthreads();
        if (tid < 32) {
            const int vi = v0 + tid;
            BpView V;
            bool use = tid < kBpViews && vi < ve && views[view0 + vi].upright;
            if (use) use = bp_view(views[view0 + vi], tx0, ty0, z0, nz, g, d, V);
            V.c1 = min(V.c1, kBpWin);  // (bp_fit_kernel)
            V.vi = vi;
            const unsigned mask = __ballot_sync(0xffffffffu, use);
            if (use) s_view[__popc(mask & ((1u << tid) - 1u))] = V;
            if (tid == 0) s_n = __popc(mask);
        }
        __syncthreads();
        const int n = s_n;
        if (n > 0) stage(0, n, 0);
        for (int i = 0, buf = 0; i < n; i += kBpStep, buf ^= 1) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (i + kBpStep < n) stage(i + kBpStep, n, buf ^ 1);
            compute(i, n, buf);
        }
    }
    store();
}

// Bytes of running sums held at a time: the views are taken in groups.
constexpr size_t kPrefixBytes = (size_t)256 << 20;

size_t setup_bytes(const ctp_geometry& g) {
    return align_up(g.nview * sizeof(UprightView)) + align_up((g.nview + 1) * sizeof(int));
}

size_t fp_item_elems(const ctp_geometry& g) { return ((size_t)g.nx * g.ny + 1) * (g.nz + 2 * kPadZ); }

int fp_rows(const ctp_geometry& g, int& passes) {
    passes = (int)((g.nv + 63) / 64);
    return (int)((g.nv + passes - 1) / passes);
}

template <typename Tin, typename Tout>
int launch_columns_fp(void* prj, const void* img, const ctp_geometry& g, unsigned flags, const ColumnsPlan& plan,
                      char* copy, cudaStream_t s) {
    Tin* vol = reinterpret_cast<Tin*>(copy);
    const size_t item = fp_item_elems(g);
    const int nzt = (int)((g.nz + 31) / 32);
    to_columns_kernel<Tin><<<dim3((unsigned)((g.nx + 31) / 32), (unsigned)g.ny, (unsigned)(nzt * g.nbatch)),
                             dim3(32, 8), 0, s>>>(vol, (const Tin*)img, (int)g.nx, (int)g.ny, (int)g.nz, item);
    int rc = check_launch("to_columns_kernel");
    if (rc) return rc;
    int passes = 0;
    const int rows = fp_rows(g, passes);
    const dim3 grid((unsigned)((g.nu + 8 * kFpCols - 1) / (8 * kFpCols)), (unsigned)passes,
                    (unsigned)(g.nview * g.nbatch));
    auto go = [&](auto kern) {
        kern<<<grid, 256, 0, s>>>((Tout*)prj, vol, plan.views, (int)g.nview, make_grid(g), make_det(g), item, rows,
                                  (flags & CTP_FLAG_ZERO_OUT) ? 0 : 1);
    };
    switch ((rows + 15) / 16) {
        case 1: go(columns_fp_kernel<1, Tin, Tout>); break;
        case 2: go(columns_fp_kernel<2, Tin, Tout>); break;
        case 3: go(columns_fp_kernel<3, Tin, Tout>); break;
        default: go(columns_fp_kernel<4, Tin, Tout>); break;
    }
    return check_launch("columns_fp_kernel");
}

int setup_views(ColumnsPlan& plan, char* base, const float* dc, const float* du_, const float* dv_, const float* sr,
                const ctp_geometry& g, bool rows_up, cudaStream_t s) {
    plan.views = reinterpret_cast<UprightView*>(base);
    plan.rest = reinterpret_cast<int*>(base + align_up(g.nview * sizeof(UprightView)));
    view_setup_kernel<<<1, 256, 0, s>>>(plan.views, plan.rest, dc, du_, dv_, sr, (int)g.nview, make_grid(g),
                                        make_det(g), rows_up ? 1 : 0);
    return check_launch("view_setup_kernel");
}

}  // namespace

// By size: the lanes that have a row (three quarters at least, of 32 rows or
// more) and nearly two waves of blocks, below which the list's chain of loads is
// exposed.  By rays and by columns: 42 x 172 x 176 voxels, 71 views of 274 x 47
// cells (98%, 1278 blocks) 235 and 180 us; 33 x 187 x 201, 97 of 251 x 37 (77%)
// 277 and 226; 24 x 388 x 379, 107 of 432 x 17 (53%) 422 and 449; 13 x 173 x 192,
// 137 of 283 x 9 134 and 136.
bool columns_fp_applies(const ctp_geometry& g, unsigned flags) {
    if (g.nv < 8) return false;
    int passes = 0;
    const int rows = fp_rows(g, passes);
    const size_t lanes = (size_t)passes * ((rows + 15) / 16) * 16;
    const size_t blocks = (g.nu + 8 * kFpCols - 1) / (8 * kFpCols) * passes * g.nview * g.nbatch;
    if (!(flags & CTP_FLAG_SIDDON_COLUMNS) && (g.nv < 32 || 4 * g.nv < 3 * lanes || blocks < 1200)) return false;
    return fp_item_elems(g) < (1ull << 31) && g.nview * g.nbatch <= 65535 &&
           ((g.nz + 31) / 32) * g.nbatch <= 65535 && g.ny <= 65535;
}

size_t columns_fp_bytes(const ctp_geometry& g, unsigned flags) {
    return setup_bytes(g) + align_up(g.nbatch * fp_item_elems(g) * elem_size_in(flags));
}

int columns_fp(ColumnsPlan& plan, char* scratch, void* prj, const void* img, const float* dc, const float* du_,
               const float* dv_, const float* sr, const ctp_geometry& g, unsigned flags, cudaStream_t s) {
    int rc = setup_views(plan, scratch, dc, du_, dv_, sr, g, false, s);
    if (rc) return rc;
    char* copy = scratch + setup_bytes(g);
    if (flags & CTP_FLAG_IN_BF16)
        return (flags & CTP_FLAG_OUT_BF16)
                   ? launch_columns_fp<__nv_bfloat16, __nv_bfloat16>(prj, img, g, flags, plan, copy, s)
                   : launch_columns_fp<__nv_bfloat16, float>(prj, img, g, flags, plan, copy, s);
    if (flags & CTP_FLAG_IN_FP16)
        return (flags & CTP_FLAG_OUT_FP16) ? launch_columns_fp<__half, __half>(prj, img, g, flags, plan, copy, s)
                                           : launch_columns_fp<__half, float>(prj, img, g, flags, plan, copy, s);
    return launch_columns_fp<float, float>(prj, img, g, flags, plan, copy, s);
}

namespace {

size_t bp_pitch(const ctp_geometry& g) { return (g.nu + 3) & ~(size_t)3; }

size_t bp_view_bytes(const ctp_geometry& g) { return g.nbatch * sum_rows((int)g.nv) * bp_pitch(g) * sizeof(float); }

// Statistics of a view (columns_prefix_kernel), per batch item.
size_t bp_view_stats(const ctp_geometry& g) { return sum_runs((int)g.nv) * ((g.nu + 127) / 128); }

size_t bp_views(const ctp_geometry& g) {
    return std::max<size_t>(1, std::min<size_t>(g.nview, kPrefixBytes / bp_view_bytes(g)));
}

}  // namespace

// By size, from the two kernels' times (ms): a ray costs its crossings (0.58e9
// cells of detector row times pixels per ms: 14.9 ms at 64 x 512 x 512 voxels
// under 360 views of 736 x 64 cells, 0.34 at 33 x 187 x 201 under 97 of 251 x
// 37), a crossing line 40 instructions a z range and 10 a plane whatever the
// rows.  The factor and the 0.06 ms (nine launches) are where both take the same
// time: 13 x 260 x 317 voxels, 284 views of 346 x 11 cells 585 us by rays, 659 by
// columns; 42 x 106 x 110, 238 of 119 x 35 273 and 323; the other side 21 x 394 x
// 384, 143 of 596 x 22 1113 and 870; 27 x 242 x 262, 148 of 294 x 25 (forward and
// back) 951 and 754.
bool columns_bp_applies(const ctp_geometry& g, unsigned flags) {
    const double lines = (double)g.nview * g.nbatch * g.nu * std::max(g.nx, g.ny);
    const double ray = lines * g.nv / 0.58e9;
    const double column = lines * 1.27 * (40.0 * ((g.nz + kBpZ - 1) / kBpZ) + 10.0 * g.nz) / 2.14e10;
    if (!(flags & CTP_FLAG_SIDDON_COLUMNS) && ray < 1.75 * column + 0.06) return false;
    return g.nz >= 4 && g.nv >= 2 && g.nv < (1u << 28) && g.nbatch * sum_runs((int)g.nv) <= 65535 &&
           g.nview <= 65535 && bp_view_bytes(g) <= kPrefixBytes && g.nu < (1u << 28);
}

size_t columns_bp_bytes(const ctp_geometry& g) {
    const size_t nv = bp_views(g);
    return setup_bytes(g) + align_up(nv * bp_view_bytes(g)) + align_up(nv * g.nu * sizeof(double2)) +
           align_up(nv * g.nbatch * bp_view_stats(g) * sizeof(float2));
}

int columns_bp(ColumnsPlan& plan, char* scratch, float* img, const void* prj, const float* dc, const float* du_,
               const float* dv_, const float* sr, const ctp_geometry& g, unsigned flags, cudaStream_t s) {
    int rc = setup_views(plan, scratch, dc, du_, dv_, sr, g, true, s);
    if (rc) return rc;
    const size_t nv = bp_views(g);
    char* p = scratch + setup_bytes(g);
    float* P = reinterpret_cast<float*>(p);
    p += align_up(nv * bp_view_bytes(g));
    double2* inv = reinterpret_cast<double2*>(p);
    p += align_up(nv * g.nu * sizeof(double2));
    float2* stats = reinterpret_cast<float2*>(p);
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int zchunks = (int)((g.nz + kBpZ - 1) / kBpZ);
    const int zper = (int)(((g.nz + zchunks - 1) / zchunks + kBpGroup - 1) / kBpGroup * kBpGroup);
    const size_t tiles = ((g.nx + kBpTile - 1) / kBpTile) * ((g.ny + kBpTile - 1) / kBpTile);
    const size_t smem = sizeof(float) * (kBpStageFloats + kBpSplitFloats);
    const Grid gr = make_grid(g);
    const Det dt = make_det(g);
    bp_fit_kernel<<<dim3((unsigned)((tiles + 127) / 128), (unsigned)g.nview), 128, 0, s>>>(
        plan.views, plan.rest, (int)g.nview, zper, zchunks, gr, dt);
    if ((rc = check_launch("bp_fit_kernel"))) return rc;
    for (size_t v0 = 0; v0 < g.nview; v0 += nv) {
        const int n = (int)std::min(nv, g.nview - v0);
        const dim3 pg((unsigned)((g.nu + 127) / 128), (unsigned)n, (unsigned)(g.nbatch * sum_runs((int)g.nv)));
        auto prefix = [&](auto* in) {
            using Tin = std::remove_pointer_t<decltype(in)>;
            columns_prefix_kernel<Tin><<<pg, 128, 0, s>>>(P, inv, stats, (const Tin*)prj, plan.views, (int)g.nview,
                                                          (int)v0, n, gr, dt, (int)bp_pitch(g));
        };
        if (flags & CTP_FLAG_IN_BF16) prefix((__nv_bfloat16*)nullptr);
        else if (flags & CTP_FLAG_IN_FP16) prefix((__half*)nullptr);
        else prefix((float*)nullptr);
        if ((rc = check_launch("columns_prefix_kernel"))) return rc;
        retire_views_kernel<<<1, 256, 0, s>>>(plan.views, plan.rest, stats, (int)v0, n, (int)g.nbatch,
                                               (int)bp_view_stats(g), dt);
        if ((rc = check_launch("retire_views_kernel"))) return rc;
        // launches of few waves (two blocks per SM) split the views into the
        // parts, added with atomics, that take the least time: the waves and one
        // block's time more (blocks at the grid's corners meet fewer lines, so the
        // last wave is ragged), times a part's views and about four more (its start
        // and the atomics).  54 x 119 x 135 voxels, 299 views of 145 x 47 cells: 662 ->
        // 564 us against whole waves
        const size_t blocks = tiles * zchunks * g.nbatch;
        int parts = 1;
        if (blocks < 12 * (size_t)sms) {
            auto rounds = [&](int p) { return ((double)blocks * p / (2.0 * sms) + 1.0) * ((n + p - 1) / p + 4); };
            for (int p = 2; p <= std::min(16, n / 8); ++p)
                if (rounds(p) < 0.97 * rounds(parts)) parts = p;
        }
        const dim3 grid((unsigned)tiles, (unsigned)(zchunks * parts), (unsigned)g.nbatch);
        int rows = 8;  // rows staged: a power of two (see column), nv or more up to kBpRows
        while (rows < kBpRows && rows < (int)g.nv) rows *= 2;
        auto k = parts > 1 ? columns_bp_kernel<true> : columns_bp_kernel<false>;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k<<<grid, 256, smem, s>>>(img, P, inv, plan.views, (int)v0, n, (n + parts - 1) / parts, gr, dt, (int)bp_pitch(g),
                                  rows, zper, zchunks);
        if ((rc = check_launch("columns_bp_kernel"))) return rc;
    }
    return CTP_OK;
}

}  // namespace ctp
