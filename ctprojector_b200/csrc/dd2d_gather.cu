// dd2d_gather.cu -- distance-driven back projection as a tiled gather, fan
// (equiangular) and parallel beams, sm_100a.
//
// Operators (reference: DDBPFanKernel distanceDriven2DBoxInt.cu:319-396,
// DDBPParallelKernel :409-497, pre-weights distanceDriven2DUtils.cu:8-65):
//   mean    the normalised back projection: per view the mean of the
//           (length-weighted) detector row over the pixel's footprint
//   fbp     the same without the length weight; fan beams with the FBP
//           distance weight
//   adjoint the exact transpose of the forward projector
//   pixel   the pixel-driven back projection (bpFanKernel3D fbp.cu:265-337 with
//           the FBP distance weight, bpParallelKernel3D fbpParallel.cu:200-250):
//           the detector row interpolated linearly at the pixel's centre
// The mean is a difference of F, the running integral of a detector row, at
// the detector coordinates j of the pixel's two edges: (F(j1) - F(j0)) /
// (j1 - j0).  The transpose is the integral from j0 to j1 too: the forward
// projector spreads cell k over the interval between its edge rays on the
// pixel's line, so the pixel's share of the cell is the overlap of [j0, j1]
// with [k, k + 1].  It is added up cell by cell, not as a difference of F: a
// gradient may hold cells of any size, or that are not finite, and they count
// for the pixels that they meet alone.  For parallel beams j is linear along
// the line.  For fan beams the edge rays sit at angles k du while the forward
// projector's cells are linear in position; with f the fraction of the cell in
// angle and T the tangent of the ray's angle to the line's normal, sin and cos
// addition theorems give the fraction in position
//   f + f (1 - f) (du T + du^2 (2 f - 1) / 3) + O(du^3).
//
// A sweep is one view with one kind of edge: the pixels' x-edges (views traced
// along y) or y-edges; views of the blend band make two.  A CTA owns a 32 x 32
// tile of S slices and takes its x-edge sweeps first, then its y-edge sweeps (it
// lists them in shared memory), so that a thread holds one set of accumulators:
// 4 neighbouring pixels along x, then 4 along y (added up in shared memory),
// with 5 edges evaluated for 4 pixels.  Per 64 sweeps one thread per sweep forms
// the tile's constants in FP64; per 16 the warps stage the window of cells the
// tile projects onto as window-local midpoint tables, and the threads add the
// sweeps by table lookups.  Batches and chunks run on from the x-edge sweeps to
// the y-edge ones (a part of 32 views has some of each: 2 x 168 x 140, 255 views,
// filtered back projection 56 -> 52 us).  No atomics; every sum in a fixed order.
//
// Measured (B200): parallel mean, 16 x 512^2, 720 views 1.72 -> 1.42 ms against
// two sets of accumulators and one 8-byte read per slice and lookup (bound now
// by shared-memory wavefronts, 76%, at 68% issue); fan mean, 4 x 512^2, 984 views
// 1.39 -> 0.94 ms, with the edges' angles relative to the tile's centre by a
// short series instead of an atanf each (57% issue: the window's tables leave two
// CTAs per SM, where the registers allow three); adjoint, fan 2 x 512^2, 984 views
// 12.6 -> 0.97 ms and parallel 3 x 317 x 413, 501 views 3.4 -> 0.21 ms against the
// kernel that intersects every cell with every pixel (as differences of F: 0.85
// and 0.17 ms); pixel-driven fan, 4 x 512^2, 984 views 3.6 -> 0.80 ms.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <climits>

#include "dd2d_gather.cuh"

namespace ctp {

namespace {

constexpr int kT = 32;        // tile edge
constexpr int kChunk = 16;    // sweeps per staged chunk
constexpr int kBatch = 64;    // sweeps whose constants are formed together
constexpr int kMaxWin = 255;  // staged cells per sweep (tables hold win + 1 entries)
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: x + kMagic rounds x to an integer in the low mantissa bits
constexpr unsigned kMagicBits = 0x4B400000u;

constexpr int kList = 1024;   // views listed at a time

// Weights of the x-edge and y-edge sweeps of a view (0: no such sweep).
// Parallel beams: the factor of a difference of F, over the signed step for the
// mean; fan beams: the blend weight (the length factors are per cell,
// cell_weights_kernel).  An angle that is not finite gives NaN.
__device__ __forceinline__ void sweep_weights(float th, int geom, int mode, const Grid& g, const Det& d, double& c,
                                              double& s, float& w0, float& w1) {
    sincos((double)th, &s, &c);
    const double ac = fabs(c), as = fabs(s);
    const bool ym = fabsf(__cosf(th)) > fabsf(__sinf(th));  // the reference's axis switch, :362
    const double r = (ac - as + kDDMarginD) / (2 * kDDMarginD);
    const double wx = r < 0 ? 0.0 : (r > 1 ? 1.0 : r);
    if (mode == kGatherAdjoint) {
        const float wf = (float)wx;
        w0 = wf;
        w1 = 1.f - wf;
        if (geom == 1) {
            if (w0 > 0.f) w0 *= (float)((double)g.dy / ac) * (c * d.du > 0 ? -1.f : 1.f);  // sign of the step along x
            if (w1 > 0.f) w1 *= (float)((double)g.dx / as) * (s * d.du > 0 ? -1.f : 1.f);
        }
    } else if (mode == kGatherPixel) {
        w0 = 1.f;
        w1 = 0.f;
    } else if (geom == 1) {
        const double jx = -c * g.dx / (double)d.du, jy = -s * g.dy / (double)d.du;
        const double pw = mode == kGatherFbp ? 1.0 : (ym ? g.dy / ac : g.dx / as);  // Utils.cu:39-65
        w0 = wx > 0 ? (float)(pw * wx / jx) : 0.f;
        w1 = wx < 1 ? (float)(pw * (1 - wx) / jy) : 0.f;
    } else {
        w0 = ym ? 1.f : 0.f;
        w1 = ym ? 0.f : 1.f;
    }
    if (!isfinite(th)) {
        w0 = NAN;
        w1 = mode == kGatherAdjoint || (geom == 1 && mode != kGatherPixel) ? NAN : 0.f;
    }
}

// Fan beams: the ray-length factor of every cell times the sweep's weight:
// out[view][nu] for the mean (each view has one sweep), out[edge][view][nu] for
// the adjoint.
__global__ void cell_weights_kernel(float* __restrict__ out, const float* __restrict__ deg, int nview, int mode, Grid g,
                                    Det d) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, view = blockIdx.y;
    if (k >= d.nu) return;
    double c, s;
    float w0, w1;
    sweep_weights(deg[view], 0, mode, g, d, c, s, w0, w1);
    const double a = (-((double)k - 0.5 * (d.nu - 1)) - (double)d.off_u) * (double)d.du;
    const double th = (double)deg[view] - a;
    const size_t i = (size_t)view * d.nu + k;
    if (mode == kGatherAdjoint) {
        if (w0 != 0.f) out[i] = w0 * (float)((double)g.dy / fabs(cos(th)));
        if (w1 != 0.f) out[(size_t)nview * d.nu + i] = w1 * (float)((double)g.dx / fabs(sin(th)));
    } else {
        out[i] = w0 != 0.f ? w0 * (float)((double)g.dy / fabs(cos(th))) : (float)((double)g.dx / fabs(sin(th)));
    }
}

// Two FP32 numbers in one register pair, one instruction for both.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ void lds_entry(unsigned addr, f32x2& m, f32x2& v) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(m), "=l"(v) : "r"(addr));
}
__device__ __forceinline__ void lds_entry(unsigned addr, float& m, float& v) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m), "=f"(v) : "r"(addr));
}
__device__ __forceinline__ void lds_value(unsigned addr, f32x2& v) {
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr));
}
__device__ __forceinline__ void lds_value(unsigned addr, float& v) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
}

// Midpoint tables of two detector rows, staged by one warp: entries k = 0 ..
// win of (running sum of the window cells before k + value / 2, value) for the
// cells from w0 (cells off the detector, and the entry past the window, are
// zero).  Lane l scans the PER consecutive entries from l PER: all 2 PER loads
// are issued before the sums, the warp scans the lane sums.  lw (may be null):
// weights of the cells.
template <typename Tp>
struct RowItem {
    const Tp* row;    // null: `off` for every cell
    const float* lw;  // weights of the row's cells, or null
    int w0;
    float off;        // value of cells off the detector
    float scale;      // of the values (adjoint)
};

// kGatherPixel: entries (value of cell k, step to cell k + 1; the last cell steps
// by zero) for linear interpolation instead.  kGatherAdjoint: the values alone,
// lane l those of k = l, l + 32, ...
template <int PER, bool PAIR, int MODE, typename Tp>
__device__ __forceinline__ void stage_rows_per(const RowItem<Tp> (&it)[2], float* t0, float* t1, int win, int nu,
                                               int lane) {
    constexpr int kNext = MODE == kGatherAdjoint ? 32 : 1;
    const int k0 = MODE == kGatherAdjoint ? lane : lane * PER;
    float v[2][PER], run[2], incl[2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int k = k0 + q * kNext, cell = it[m].w0 + k;
            const bool in = it[m].row && k < win && cell >= 0 && cell < nu;
            v[m][q] = in ? ldf(it[m].row + cell) : it[m].off;
            if (it[m].lw && in) v[m][q] *= __ldg(it[m].lw + cell);
            if (MODE == kGatherAdjoint) v[m][q] *= it[m].scale;
        }
    if constexpr (MODE == kGatherAdjoint) {
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int k = k0 + q * kNext;
            if (k > win) continue;
            if constexpr (PAIR) {
                reinterpret_cast<float2*>(t0)[k] = make_float2(v[0][q], v[1][q]);
            } else {
                t0[k] = v[0][q];
                if (t1) t1[k] = v[1][q];
            }
        }
    } else if constexpr (MODE == kGatherPixel) {
        const float next[2] = {__shfl_down_sync(0xffffffffu, v[0][0], 1), __shfl_down_sync(0xffffffffu, v[1][0], 1)};
        auto step_of = [&](int m, int q, float& after) {
            const int cell = it[m].w0 + k0 + q;
            after = q + 1 < PER ? v[m][q + 1] : next[m];
            return cell >= 0 && cell + 1 < nu ? after - v[m][q] : 0.f;
        };
        auto put = [&](int q, float s0, float s1) {
            const int k = k0 + q;
            if (k > win) return;
            if constexpr (PAIR) {
                reinterpret_cast<float4*>(t0)[k] = make_float4(v[0][q], v[1][q], s0, s1);
            } else {
                reinterpret_cast<float2*>(t0)[k] = make_float2(v[0][q], s0);
                if (t1) reinterpret_cast<float2*>(t1)[k] = make_float2(v[1][q], s1);
            }
        };
        float finite = 0.f, after;  // NaN when a step is not finite
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const float s0 = step_of(0, q, after), s1 = step_of(1, q, after);
            finite = fmaf(s0, 0.f, fmaf(s1, 0.f, finite));
            put(q, s0, s1);
        }
        if (finite != 0.f) {
            // from an infinite cell to one that does not contradict it: no step
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                float s[2];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    s[m] = step_of(m, q, after);
                    if (isinf(v[m][q]) && (isfinite(after) || after == v[m][q])) s[m] = 0.f;
                }
                put(q, s[0], s[1]);
            }
        }
    } else {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            run[m] = 0.f;
#pragma unroll
            for (int q = 0; q < PER; ++q) run[m] += v[m][q];
            incl[m] = run[m];
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float t = __shfl_up_sync(0xffffffffu, incl[m], o);
                if (lane >= o) incl[m] += t;
            }
        float b0 = incl[0] - run[0], b1 = incl[1] - run[1];
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int k = k0 + q;
            if (k <= win) {
                const float m0 = fmaf(0.5f, v[0][q], b0), m1 = fmaf(0.5f, v[1][q], b1);
                if constexpr (PAIR) {
                    reinterpret_cast<float4*>(t0)[k] = make_float4(m0, m1, v[0][q], v[1][q]);
                } else {
                    reinterpret_cast<float2*>(t0)[k] = make_float2(m0, v[0][q]);
                    if (t1) reinterpret_cast<float2*>(t1)[k] = make_float2(m1, v[1][q]);
                }
            }
            b0 += v[0][q];
            b1 += v[1][q];
        }
    }
}

template <bool PAIR, int MODE, typename Tp>
__device__ __forceinline__ void stage_rows(const RowItem<Tp> (&it)[2], float* t0, float* t1, int win, int nu, int lane) {
    switch ((win + 1 + 31) / 32) {
        case 1: stage_rows_per<1, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 2: stage_rows_per<2, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 3: stage_rows_per<3, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 4: stage_rows_per<4, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 5: stage_rows_per<5, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 6: stage_rows_per<6, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        case 7: stage_rows_per<7, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
        default: stage_rows_per<8, PAIR, MODE>(it, t0, t1, win, nu, lane); break;
    }
}

// Accumulators and lookups of S slices: pairs of slices share an entry (16
// bytes, one load) and packed arithmetic; one slice runs scalar.
template <int S>
struct Lanes {
    static constexpr int NP = S / 2;       // pairs
    static constexpr int kEntry = 16;      // bytes of a table entry (the adjoint's: half of it)
    f32x2 a[NP][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k) a[p][k] = 0ull;
    }
    struct Point {
        f32x2 f[NP];
    };
    // F of every slice at the entry at addr (plane: bytes between the pairs' tables) and offset fr from its midpoint
    __device__ __forceinline__ static Point at(unsigned addr, unsigned plane, float fr) {
        Point p;
        const f32x2 fr2 = pack2(fr, fr);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            f32x2 m, v;
            lds_entry(addr + q * plane, m, v);
            p.f[q] = fma2(v, fr2, m);
        }
        return p;
    }
    __device__ __forceinline__ void add(int k, const Point& lo, const Point& hi, float w) {
        const f32x2 w2 = pack2(w, w), neg = pack2(-1.f, -1.f);
#pragma unroll
        for (int q = 0; q < NP; ++q) a[q][k] = fma2(fma2(lo.f[q], neg, hi.f[q]), w2, a[q][k]);
    }
    __device__ __forceinline__ void add(int k, const Point& p, float w) {
        const f32x2 w2 = pack2(w, w);
#pragma unroll
        for (int q = 0; q < NP; ++q) a[q][k] = fma2(p.f[q], w2, a[q][k]);
    }
    // every slice's value of the cell at addr
    __device__ __forceinline__ static Point value(unsigned addr, unsigned plane) {
        Point p;
#pragma unroll
        for (int q = 0; q < NP; ++q) lds_value(addr + q * plane, p.f[q]);
        return p;
    }
    __device__ __forceinline__ static Point zero_point() {
        Point p;
#pragma unroll
        for (int q = 0; q < NP; ++q) p.f[q] = 0ull;
        return p;
    }
    __device__ __forceinline__ static void scale_add(Point& t, const Point& v, float w) {
        const f32x2 w2 = pack2(w, w);
#pragma unroll
        for (int q = 0; q < NP; ++q) t.f[q] = fma2(v.f[q], w2, t.f[q]);
    }
    __device__ __forceinline__ void add(int k, const Point& t) {
        const f32x2 one = pack2(1.f, 1.f);
#pragma unroll
        for (int q = 0; q < NP; ++q) a[q][k] = fma2(t.f[q], one, a[q][k]);
    }
    __device__ __forceinline__ float get(int s, int k) const {
        float x, y;
        unpack2(a[s / 2][k], x, y);
        return s & 1 ? y : x;
    }
    __device__ __forceinline__ void set(int p, int k, float x, float y) { a[p][k] = pack2(x, y); }
};

template <>
struct Lanes<1> {
    static constexpr int NP = 1;
    static constexpr int kEntry = 8;
    float a[4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = 0.f;
    }
    struct Point {
        float f;
    };
    __device__ __forceinline__ static Point at(unsigned addr, unsigned, float fr) {
        float m, v;
        lds_entry(addr, m, v);
        return Point{fmaf(v, fr, m)};
    }
    __device__ __forceinline__ void add(int k, const Point& lo, const Point& hi, float w) {
        a[k] = fmaf(hi.f - lo.f, w, a[k]);
    }
    __device__ __forceinline__ void add(int k, const Point& p, float w) { a[k] = fmaf(p.f, w, a[k]); }
    __device__ __forceinline__ static Point value(unsigned addr, unsigned) {
        Point p;
        lds_value(addr, p.f);
        return p;
    }
    __device__ __forceinline__ static Point zero_point() { return Point{0.f}; }
    __device__ __forceinline__ static void scale_add(Point& t, const Point& v, float w) { t.f = fmaf(v.f, w, t.f); }
    __device__ __forceinline__ void add(int k, const Point& t) { a[k] += t.f; }
    __device__ __forceinline__ float get(int, int k) const { return a[k]; }
    __device__ __forceinline__ void set(int, int k, float x, float) { a[k] = x; }
};

// Constants of a sweep for one tile, and those of its pixel runs.
// Parallel: j of the pixel centre (kx, ky) is jb + kx jx + ky jy, from the
// window's first cell's midpoint; w weighs a difference.
// Fan: the pixel point (x, y), in pixels from the tile's centre, is seen at
// the angle of the centre plus atan(z), z = (cx x + cy y) / (1 + bx x + by y);
// j = jb + atan(z) / du.  gx, gy: the centre minus the source in pixels.
struct TileSweep {
    float jb, jx, jy, w;      // parallel; fan: jb, cx, cy, dso^2 / (distance of the centre)^2
    float bx, by, gx, gy;     // fan
};

struct GatherArgs {
    void* img;           // output, or the parts' partial volumes
    const void* prj;
    const float* deg;
    const float* lw;     // fan: weights of the cells (cell_weights_kernel), or null
    int mode, nview, vper, nslices, win, wide, parts, accumulate, out_lp, one_to_one;
    size_t part_elems;
    float dso;
    Grid g;
    Det d;
};

__device__ __forceinline__ void store_out(void* img, size_t i, float v, int lp, int accumulate) {
    if (lp == 0) {
        float* o = static_cast<float*>(img) + i;
        *o = accumulate ? *o + v : v;
    } else if (lp == 1) {
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(img) + i;
        stf(o, accumulate ? rdf(o) + v : v);
    } else {
        __half* o = static_cast<__half*>(img) + i;
        stf(o, accumulate ? rdf(o) + v : v);
    }
}

// Bytes of a table entry: two numbers per slice, for the adjoint one.
template <int MODE, int S>
constexpr int entry_bytes() { return MODE == kGatherAdjoint ? Lanes<S>::kEntry / 2 : Lanes<S>::kEntry; }

// Bytes of a CTA's dynamic shared memory: the tables of a chunk and the tile's sums.
template <int MODE, int S>
size_t gather_smem(int win) {
    const size_t tab = (size_t)Lanes<S>::NP * entry_bytes<MODE, S>() * kChunk * (win + 1);
    const size_t acc = (size_t)S * kT * (kT + 1) * sizeof(float);
    return tab + acc;
}

template <bool FAN, int MODE, int S, typename Tp>
__global__ void __launch_bounds__(256, (S == 4 ? 3 : 4)) gather_bp_kernel(const GatherArgs A) {
    extern __shared__ float4 s_raw[];
    __shared__ __align__(16) TileSweep s_tile[kBatch];
    __shared__ int s_w0[kBatch];
    __shared__ unsigned short s_list[2][kList];  // views of the x-edge and y-edge sweeps
    __shared__ int s_cnt[2][8];
    using L = Lanes<S>;
    const Grid& g = A.g;
    const Det& d = A.d;
    const int stride = A.win + 1;
    constexpr int kEntry = entry_bytes<MODE, S>();
    const unsigned plane = kChunk * stride * kEntry;  // bytes of one pair's tables
    float* tab = reinterpret_cast<float*>(s_raw);
    float* s_sum = tab + L::NP * plane / 4;  // [S][kT][kT + 1]
    const int tiles_x = (g.nx + kT - 1) / kT;
    const int tx0 = (blockIdx.x % tiles_x) * kT, ty0 = (blockIdx.x / tiles_x) * kT;
    const int s0 = blockIdx.y * S, ns = min(S, A.nslices - s0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // x layout: 4 pixels along x from (xl_col, xl_row), eight rows to a quarter
    // warp: its 16-byte reads lie within 8 cells (the views of x-edge sweeps
    // move by less than a cell per row), so on distinct banks or one word.  y
    // layout: 4 along y, lane = column, likewise.
    const int xl_row = (warp >> 1) * 8 + (lane & 7), xl_col = ((warp & 1) * 4 + (lane >> 3)) * 4;
    const int yl_col = lane, yl_row = warp * 4;
    // the tile's part of the grid, and up to 4 pixels past it for the runs at the grid's edge
    const int tw = min(kT, g.nx - tx0 + 4), th = min(kT, g.ny - ty0 + 4);

    // detector row of each slice (truncation, distanceDriven2DBoxInt.cu:383); none off the detector
    const Tp* rows[S];
    bool any_row = false;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int slice = s0 + min(s, ns - 1), iz = slice % g.nz, b = slice / g.nz;
        const float zc = ((float)iz - g.nz / 2.f) * g.dz + g.cz + g.dz / 2;
        int iv = A.one_to_one ? iz : (int)(zc / d.dv + d.off_v + d.nv / 2.f - 0.5f);
        bool ok = s < ns && iv >= 0 && iv < d.nv;
        if (MODE == kGatherPixel) {  // one detector row, not interpolated (fbp.cu:308, fbpParallel.cu:228)
            const float pv = (((float)iz + 0.5f - g.nz / 2.f) * g.dz + g.cz) / d.dv + d.off_v;
            iv = 0;
            ok = s < ns && pv >= 0.f && pv < 1.f;
        }
        rows[s] = ok ? static_cast<const Tp*>(A.prj) + ((size_t)b * A.nview * d.nv + iv) * d.nu : nullptr;
        any_row |= ok;
    }
    const size_t vstride = (size_t)d.nv * d.nu;

    L acc;
    acc.zero();
    for (int i = threadIdx.x; i < S * kT * (kT + 1); i += 256) s_sum[i] = 0.f;  // (barriers below)
    const int vb = blockIdx.z * A.vper, ve = min(A.nview, vb + A.vper);
    const unsigned tab_addr = (unsigned)__cvta_generic_to_shared(tab) - kEntry * kMagicBits;  // (wraps)
    const float idu = 1.f / d.du;

    for (int vs = vb; vs < ve; vs += kList) {
        int nlist[2] = {0, 0};
        for (int t0 = vs; t0 < min(ve, vs + kList); t0 += 256) {
            const int v = t0 + threadIdx.x;
            double c, s;
            float w0 = 0.f, w1 = 0.f;
            if (v < ve) sweep_weights(A.deg[v], FAN ? 0 : 1, A.mode, g, d, c, s, w0, w1);
            const unsigned m0 = __ballot_sync(0xffffffffu, w0 != 0.f), m1 = __ballot_sync(0xffffffffu, w1 != 0.f);
            if (lane == 0) {
                s_cnt[0][warp] = __popc(m0);
                s_cnt[1][warp] = __popc(m1);
            }
            __syncthreads();
            const unsigned below = (1u << lane) - 1u;
            int p0 = nlist[0] + __popc(m0 & below), p1 = nlist[1] + __popc(m1 & below);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (q < warp) {
                    p0 += s_cnt[0][q];
                    p1 += s_cnt[1][q];
                }
                nlist[0] += s_cnt[0][q];
                nlist[1] += s_cnt[1][q];
            }
            if (w0 != 0.f) s_list[0][p0] = (unsigned short)(v - vs);
            if (w1 != 0.f) s_list[1][p1] = (unsigned short)(v - vs);
            __syncthreads();
        }
        // the x-edge sweeps, then the y-edge ones; a batch or chunk may hold both
        const int nx_sweeps = nlist[0], sweeps = any_row ? nlist[0] + nlist[1] : 0;
        auto view_of = [&](int q) { return vs + (q < nx_sweeps ? s_list[0][q] : s_list[1][q - nx_sweeps]); };
        // the sweeps of one kind join the tile's sums (the layouts differ)
        auto join = [&](int o) {
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (o == 0) s_sum[(s * kT + xl_row) * (kT + 1) + xl_col + k] += acc.get(s, k);
                    else s_sum[(s * kT + yl_row + k) * (kT + 1) + yl_col] += acc.get(s, k);
                }
            acc.zero();
        };
        for (int q0 = 0; q0 < sweeps; q0 += kChunk) {
            const int n = min(kChunk, sweeps - q0), qt = q0 & (kBatch - 1);  // (kBatch: a power of two)
            if (qt == 0 && threadIdx.x < min(kBatch, sweeps - q0)) {
                const int q = q0 + threadIdx.x, o = q >= nx_sweeps;
                double c, s;
                float w0_, w1_;
                sweep_weights(A.deg[view_of(q)], FAN ? 0 : 1, A.mode, g, d, c, s, w0_, w1_);
                const double du = d.du;
                TileSweep T;
                double jmin, jmax, jref;
                if (FAN) {
                    // centre of the tile, relative to the source (dso sin, -dso cos)
                    const double ax = (tx0 + 0.5 * tw - 0.5 * g.nx) * g.dx + g.cx - (double)A.dso * s;
                    const double ay = (ty0 + 0.5 * th - 0.5 * g.ny) * g.dy + g.cy + (double)A.dso * c;
                    const double a2 = ax * ax + ay * ay, ia2 = 1.0 / a2;
                    // fan angle atan(rx / ry) of the centre
                    const double a = atan2(ax * c + ay * s, -ax * s + ay * c);
                    jref = -(a / du + (double)d.off_u) + 0.5 * d.nu;
                    const double cx = -ay * g.dx * ia2, cy = ax * g.dy * ia2, bx = ax * g.dx * ia2, by = ay * g.dy * ia2;
                    double zmax = 0.0;
                    for (int e = 0; e < 4; ++e) {
                        const double x = (e & 1) ? 0.5 * tw : -0.5 * tw, y = (e & 2) ? 0.5 * th : -0.5 * th;
                        zmax = fmax(zmax, fabs((cx * x + cy * y) / (1.0 + bx * x + by * y)));
                    }
                    jmin = jref - atan(zmax) / fabs(du);
                    jmax = jref + atan(zmax) / fabs(du);
                    T.jx = (float)cx;
                    T.jy = (float)cy;
                    T.w = (float)((double)A.dso * A.dso * ia2);
                    T.bx = (float)bx;
                    T.by = (float)by;
                    T.gx = (float)(ax / g.dx);
                    T.gy = (float)(ay / g.dy);
                } else {
                    const double jx = -c * g.dx / du, jy = -s * g.dy / du;
                    const double xc0 = (tx0 + 0.5 - 0.5 * g.nx) * g.dx + g.cx;
                    const double yc0 = (ty0 + 0.5 - 0.5 * g.ny) * g.dy + g.cy;
                    jref = -((xc0 * c + yc0 * s) / du + d.off_u) + 0.5 * d.nu;
                    const double hm = 0.5 * fabs(o == 0 ? jx : jy);
                    jmin = jref + fmin(0.0, (kT - 1) * jx) + fmin(0.0, (kT - 1) * jy) - hm;
                    jmax = jref + fmax(0.0, (kT - 1) * jx) + fmax(0.0, (kT - 1) * jy) + hm;
                    T.jx = (float)jx;
                    T.jy = (float)jy;
                    T.w = o == 0 ? w0_ : w1_;
                    T.bx = T.by = T.gx = T.gy = 0.f;
                }
                // two spare cells on each side: every lookup lands inside the table
                int w0 = 0;
                const bool ok = jmin > -1e9 && jmax < 1e9 && (int)ceil(jmax) + 4 - (int)floor(jmin) <= A.win;
                if (ok) w0 = (int)floor(jmin) - 2;
                T.jb = (float)(jref - w0 - 0.5);
                if (!ok) {  // an angle that is not a number: so is the result (the lookups stay inside)
                    const float step = 1.f / 4096;
                    T.jb = 1.f;
                    T.jx = T.jy = FAN ? step * d.du : step;
                    T.bx = T.by = 0.f;
                    T.gx = copysignf(1e6f, d.du);
                    T.gy = -T.gx;
                    T.w = NAN;
                }
                s_tile[threadIdx.x] = T;
                s_w0[threadIdx.x] = ok ? w0 : INT_MIN;
            }
            __syncthreads();
            // stage the tables: pairs of slices of a sweep, or (S = 1) pairs of sweeps
            auto item = [&](RowItem<Tp>& it, const Tp* row, int vi) {
                const int w0 = s_w0[qt + vi], view = view_of(q0 + vi);
                const bool ok = w0 != INT_MIN;
                it.row = row && ok ? row + (size_t)view * vstride : nullptr;
                const size_t kind = MODE == kGatherAdjoint && q0 + vi >= nx_sweeps ? A.nview : 0;
                it.lw = A.lw ? A.lw + (kind + view) * d.nu : nullptr;
                it.w0 = ok ? w0 : 0;
                it.off = ok ? 0.f : NAN;
                it.scale = MODE == kGatherAdjoint && !FAN ? fabsf(s_tile[qt + vi].w) : 1.f;
            };
            if constexpr (S >= 2) {
                for (int i = warp; i < n * L::NP; i += 8) {
                    const int vi = i / L::NP, p = i - vi * L::NP;
                    RowItem<Tp> it[2];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const Tp* r = rows[m];
#pragma unroll
                        for (int q = 1; q < L::NP; ++q)
                            if (p == q) r = rows[2 * q + m];
                        item(it[m], r, vi);
                    }
                    stage_rows<true, MODE>(it, tab + (p * plane + vi * stride * kEntry) / 4, nullptr, A.win, d.nu,
                                           lane);
                }
            } else {
                for (int i = warp * 2; i < n; i += 16) {
                    RowItem<Tp> it[2];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        item(it[m], rows[0], min(i + m, n - 1));
                    }
                    float* t = tab + (size_t)i * stride * (kEntry / 4);
                    stage_rows<false, MODE>(it, t, i + 1 < n ? t + stride * (kEntry / 4) : nullptr, A.win, d.nu, lane);
                }
            }
            __syncthreads();
            const int nx_here = min(max(nx_sweeps - q0, 0), n);
            for (int o = 0; o < (MODE == kGatherPixel ? 1 : 2); ++o) {
                const int first = o == 0 ? 0 : nx_here, end = o == 0 ? nx_here : n;
                if (o == 1 && first < end && q0 + first == nx_sweeps && nx_sweeps > 0) join(0);
                // the run's first pixel (runs past the grid, whose sums are dropped, take one inside)
                const float px = (float)min(o == 0 ? xl_col : yl_col, g.nx - tx0 - 1);
                const float py = (float)min(o == 0 ? xl_row : yl_row, g.ny - ty0 - 1);
                for (int vi = first; vi < end; ++vi) {
                    const float4 T = *reinterpret_cast<const float4*>(&s_tile[qt + vi]);  // jb, jx, jy, w
                    const unsigned base = tab_addr + vi * stride * kEntry;
                    typename L::Point prev;
                    // adjoint: the run's next edge, at x along the direction in which j moves
                    // (dir: j itself or -j), in fractions f of a cell from its middle.  The
                    // pixel before it takes its share of the last edge's cell, of this one's,
                    // and the cells in between; no share, no term (0 x infinity).
                    int cell_prev = 0;
                    unsigned at_prev = 0;
                    float x_prev = -INFINITY, f_prev = 0.f;
                    auto edge = [&](int k, float x, float dir, auto fraction) {
                        x = fmaxf(x, x_prev);  // (NaN: x_prev)
                        const float tt = x + kMagic;
                        const int cell = __float_as_int(tt), step = dir < 0.f ? -kEntry : kEntry;
                        const unsigned at = base + kEntry * kMagicBits + (unsigned)(step * (cell - (int)kMagicBits));
                        const float f = fraction(x - (tt - kMagic));
                        const typename L::Point v = L::value(at, plane);
                        if (k > 0) {
                            const int n = cell - cell_prev;
                            const float both = 0.5f * (f - f_prev);  // one cell: half from each of its readings
                            const float a = n > 0 ? 0.5f - f_prev : both, b = n > 0 ? 0.5f + f : both;
                            typename L::Point t = L::zero_point();
                            if (!(a <= 0.f)) L::scale_add(t, prev, a);
                            if (!(b <= 0.f)) L::scale_add(t, v, b);
                            if (n > 1) L::scale_add(t, L::value(at_prev + step, plane), 1.f);
                            if (n > 2)
                                for (int i = 2; i < n; ++i) L::scale_add(t, L::value(at_prev + i * step, plane), 1.f);
                            acc.add(k - 1, t);
                        }
                        prev = v;
                        at_prev = at;
                        cell_prev = cell;
                        x_prev = x;
                        f_prev = f;
                    };
                    if constexpr (MODE == kGatherPixel) {
                        // 4 pixel centres; xs from the window's first cell's centre
                        float x, dx, cr = 0.f, dd = 1.f, dcr = 0.f, ddt = 0.f;
                        if constexpr (FAN) {
                            const float4 B = *reinterpret_cast<const float4*>(&s_tile[qt + vi].bx);
                            const float x0 = px - 0.5f * (float)tw + 0.5f, y0 = py - 0.5f * (float)th + 0.5f;
                            cr = fmaf(T.y, x0, T.z * y0);
                            dd = fmaf(B.x, x0, fmaf(B.y, y0, 1.f));
                            dcr = T.y;
                            ddt = B.x;
                        } else {
                            x = fmaf(px, T.y, fmaf(py, T.z, T.x));
                            dx = T.y;
                        }
    #pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            float xs, w = T.w;
                            if constexpr (FAN) {
                                const float z = __fdividef(cr, dd), z2 = z * z;
                                const float at = A.wide ? atanf(z)
                                                        : fmaf(z * z2, fmaf(z2, fmaf(z2, -1.f / 7.f, 0.2f), -1.f / 3.f), z);
                                xs = fmaf(at, idu, T.x);
                                w = __fdividef(T.w, fmaf(cr, cr, dd * dd));
                                cr += dcr;
                                dd += ddt;
                            } else {
                                xs = fmaf((float)k, dx, x);
                            }
                            const float tt = __fadd_rd(xs, kMagic);  // floor
                            acc.add(k, L::at(base + kEntry * __float_as_uint(tt), plane, xs - (tt - kMagic)), w);
                        }
                    } else if constexpr (!FAN) {
                        // the run's first edge, half a pixel before its first centre
                        float e0 = fmaf(px - (o == 0 ? 0.5f : 0.f), T.y, fmaf(py - (o == 0 ? 0.f : 0.5f), T.z, T.x));
                        float step = o == 0 ? T.y : T.z;
                        const float dir = copysignf(1.f, step);
                        if constexpr (MODE == kGatherAdjoint) {
                            e0 *= dir;
                            step *= dir;
                        }
    #pragma unroll
                        for (int k = 0; k < 5; ++k) {
                            const float xs = fmaf((float)k, step, e0);
                            if constexpr (MODE == kGatherAdjoint) {
                                edge(k, xs, dir, [](float f) { return f; });
                            } else {
                                const float tt = xs + kMagic;
                                const typename L::Point p =
                                    L::at(base + kEntry * __float_as_uint(tt), plane, xs - (tt - kMagic));
                                if (k > 0) acc.add(k - 1, prev, p, T.w);
                                prev = p;
                            }
                        }
                    } else {
                        const float4 B = *reinterpret_cast<const float4*>(&s_tile[qt + vi].bx);  // bx, by, gx, gy
                        // the run's first edge point, in pixels from the tile's centre
                        const float x0 = px - 0.5f * (float)tw + (o == 0 ? 0.f : 0.5f);
                        const float y0 = py - 0.5f * (float)th + (o == 0 ? 0.5f : 0.f);
                        const float cr0 = fmaf(T.y, x0, T.z * y0), dt0 = fmaf(B.x, x0, fmaf(B.y, y0, 1.f));
                        const float dcr = o == 0 ? T.y : T.z, ddt = o == 0 ? B.x : B.y;
                        // du T at the run's first point and its step (y fixed along an x run)
                        float t0 = 0.f, dt = 0.f;
                        if (MODE == kGatherAdjoint) {
                            const float r = g.dx / g.dy;
                            if (o == 0) {
                                dt = __fdividef(d.du * r, B.w + y0);
                                t0 = (B.z + x0) * dt;
                            } else {
                                dt = -__fdividef(d.du, r * (B.z + x0));
                                t0 = (B.w + y0) * dt;
                            }
                        }
                        const float c3 = d.du * d.du * (2.f / 3.f);
                        // the adjoint takes j, du T and 1 / du along the direction of j
                        const float dir = copysignf(1.f, idu * (o == 0 ? -(B.w + y0) : B.z + x0));
                        const float jc = MODE == kGatherAdjoint ? dir * T.x : T.x;
                        const float jdu = MODE == kGatherAdjoint ? dir * idu : idu;
                        t0 *= dir;
                        dt *= dir;
                        float jprev = 0.f;
                        float crp = 0.f, dtp = 0.f;
    #pragma unroll
                        for (int k = 0; k < 5; ++k) {
                            const float cr = fmaf((float)k, dcr, cr0), dd = fmaf((float)k, ddt, dt0);
                            const float z = __fdividef(cr, dd), z2 = z * z;
                            // atan(z) by its series (|z| <= 0.12: the next term is below 6e-10), unless a tile spans more
                            const float at = A.wide ? atanf(z)
                                                    : fmaf(z * z2, fmaf(z2, fmaf(z2, -1.f / 7.f, 0.2f), -1.f / 3.f), z);
                            const float xs = fmaf(at, jdu, jc);
                            if constexpr (MODE == kGatherAdjoint) {
                                const float duT = fmaf((float)k, dt, t0);
                                edge(k, xs, dir, [&](float f) { return fmaf(fmaf(-f, f, 0.25f), fmaf(c3, f, duT), f); });
                                continue;
                            }
                            const float tt = xs + kMagic;
                            const typename L::Point p =
                                L::at(base + kEntry * __float_as_uint(tt), plane, xs - (tt - kMagic));
                            if (k > 0) {
                                float w = __fdividef(1.f, xs - jprev);
                                if (MODE == kGatherFbp) {
                                    // dso^2 over the squared distance of the pixel's centre
                                    const float cc = 0.5f * (cr + crp), dc = 0.5f * (dd + dtp);
                                    w *= __fdividef(T.w, fmaf(cc, cc, dc * dc));
                                }
                                acc.add(k - 1, prev, p, w);
                            }
                            prev = p;
                            jprev = xs;
                            crp = cr;
                            dtp = dd;
                        }
                    }
                }
            }
            __syncthreads();
        }
        join(MODE != kGatherPixel && nlist[1] > 0 ? 1 : 0);
        __syncthreads();
    }
    const int ix = tx0 + yl_col;
    if (ix >= g.nx) return;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (s >= ns) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int iy = ty0 + yl_row + k;
            if (iy >= g.ny) continue;
            const size_t i = ((size_t)(s0 + s) * g.ny + iy) * g.nx + ix;
            const float v = s_sum[(s * kT + yl_row + k) * (kT + 1) + yl_col];
            if (A.parts > 1) static_cast<float*>(A.img)[blockIdx.z * A.part_elems + i] = v;
            else store_out(A.img, i, v, A.out_lp, A.accumulate);
        }
    }
}

// Sum of the parts of a split back projection into the output, in order.
__global__ void __launch_bounds__(256) gather_sum_kernel(void* __restrict__ img, const float* __restrict__ parts,
                                                         int nparts, size_t elems, int lp, int accumulate) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < elems; i += (size_t)gridDim.x * blockDim.x) {
        float a = 0.f;
#pragma unroll 8
        for (int q = 0; q < nparts; ++q) a += parts[(size_t)q * elems + i];
        store_out(img, i, a, lp, accumulate);
    }
}

// Staged cells per sweep: the largest extent of a tile on the detector, or 0
// if it does not fit.  zmax: fan, the largest tangent of the angle between a
// point of a tile and its centre.
int gather_window(const ctp_geometry& g, int geom, double* zmax) {
    const double du = fabs((double)g.du);
    double cells;
    if (geom == 0) {
        // the grid and the 4 pixels past it that a tile may reach
        const double ex = (0.5 * g.nx + 4) * g.dx, ey = (0.5 * g.ny + 4) * g.dy;
        const double rmax = sqrt((fabs(g.cx) + ex) * (fabs(g.cx) + ex) + (fabs(g.cy) + ey) * (fabs(g.cy) + ey));
        const double diag = kT * sqrt((double)g.dx * g.dx + (double)g.dy * g.dy);
        const double near = (double)g.dso - rmax;
        if (!(near > diag)) return 0;
        // a corner is at most diag / 2 from the centre, which is at least near from the source
        const double x = 0.5 * diag / near;
        *zmax = x / sqrt(1 - x * x);
        cells = 2 * asin(x) / du;
    } else {
        *zmax = 0;
        cells = ((kT - 1) * ((double)g.dx + g.dy) + fmax((double)g.dx, (double)g.dy)) / du;
    }
    if (!(cells < kMaxWin)) return 0;
    const int win = (int)ceil(cells) + 8;
    return win <= kMaxWin ? win : 0;
}

// CTAs resident on an SM by the kernels' registers; windows of more than 103 cells
// (fan, S = 4) leave one less by shared memory.
int ctas_per_sm(int S) { return S == 4 ? 3 : 4; }

int sm_count() {
    int sms = 148, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Most parts that the views may be split into (the workspace holds as many
// partial volumes), from the tiles times groups of two slices (fan) or four
// (parallel; calls this small take such groups, see slices_per_cta): enough for
// four CTAs per SM, and chunks of 16 views at least, when there are fewer than
// two; for launches of up to three waves of two per SM the count that fills them
// best; none for larger ones, whose tail is spread over the SMs.  Fan mean, 4 x
// 139 x 166, 112 views: 36 us with 4 parts of 32 views, 28 with 7 of 16.
int gather_most_parts(const ctp_geometry& g, int geom) {
    const size_t n = g.nbatch * g.nz, per = geom == 0 ? (n >= 2 ? 2 : 1) : n >= 3 ? 4 : n;
    const size_t units = ((g.nx + kT - 1) / kT) * ((g.ny + kT - 1) / kT) * ((n + per - 1) / per);
    const int sms = sm_count();
    int parts = 1, least = 2 * kChunk;
    if (units > 0 && units < 2 * (size_t)sms) {
        parts = (int)std::min<size_t>(16, (4 * (size_t)sms + units - 1) / units);
        least = kChunk;
    } else if (units > 0 && units < 6 * (size_t)sms) {
        auto fill = [&](int p) {
            const double waves = (double)units * p / (2.0 * sms);
            return waves / std::ceil(waves);
        };
        if (fill(1) < 0.95)
            for (int p = 2; p <= 8; ++p)
                if (fill(p) > fill(parts) + 0.02) parts = p;
    }
    return std::max(1, std::min(parts, (int)((g.nview + least - 1) / least)));
}

// Slices per CTA (the last CTA of a stack may hold fewer): four share a view's
// constants, positions and weights, but where that leaves SMs without a CTA even
// with the most parts, groups of two or one slice.  Fan mean, 4 x 139 x 166, 112
// views: 30 tiles x 4 parts 46 us with four slices, 2 groups as many CTAs 38.
int slices_per_cta(const ctp_geometry& g, int geom) {
    const size_t n = g.nbatch * g.nz, tiles = ((g.nx + kT - 1) / kT) * ((g.ny + kT - 1) / kT);
    const size_t most = (size_t)gather_most_parts(g, geom), sms = (size_t)sm_count();
    int S = n >= 3 ? 4 : n == 2 ? 2 : 1;
    while (S > 1 && tiles * ((n + S - 1) / S) * most < sms) S /= 2;
    return S;
}

// The parts taken: of those, the count that fills the SMs best.  vper: views per part.
int gather_parts(const ctp_geometry& g, int geom, int& vper) {
    const int most = gather_most_parts(g, geom), S = slices_per_cta(g, geom);
    const size_t ctas = ((g.nx + kT - 1) / kT) * ((g.ny + kT - 1) / kT) * ((g.nbatch * g.nz + S - 1) / S);
    const double slots = (double)ctas_per_sm(S) * sm_count();
    int parts = 1;
    auto fill = [&](int p) {
        const double waves = (double)ctas * p / slots;
        return waves / std::ceil(waves);
    };
    for (int p = 2; p <= most; ++p)
        if (fill(p) > fill(parts) + 0.02) parts = p;
    vper = (int)(((g.nview + parts - 1) / parts + kChunk - 1) / kChunk * kChunk);
    return (int)((g.nview + vper - 1) / vper);
}

// Fan mean: the cells' weights of a view, in the room that the workspace query
// keeps for a weighted copy of the sinogram (the general kernel's).
size_t weight_bytes(const ctp_geometry& g, int geom, GatherMode mode) {
    if (geom != 0 || mode == kGatherFbp || mode == kGatherPixel) return 0;
    if (mode == kGatherAdjoint) return align_up(2 * g.nview * g.nu * sizeof(float));
    return align_up(g.nbatch * g.nview * g.nv * g.nu * sizeof(float));
}

template <bool FAN, int MODE, typename Tp>
int launch_gather(const GatherArgs& A, dim3 grid, int S, cudaStream_t s) {
    auto go = [&](auto kern, size_t smem) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<grid, 256, smem, s>>>(A);
        return check_launch("gather_bp_kernel");
    };
    if (S == 4) return go(gather_bp_kernel<FAN, MODE, 4, Tp>, gather_smem<MODE, 4>(A.win));
    if (S == 2) return go(gather_bp_kernel<FAN, MODE, 2, Tp>, gather_smem<MODE, 2>(A.win));
    return go(gather_bp_kernel<FAN, MODE, 1, Tp>, gather_smem<MODE, 1>(A.win));
}

template <bool FAN, int MODE>
int launch_gather_type(const GatherArgs& A, dim3 grid, int S, unsigned flags, cudaStream_t s) {
    if (flags & CTP_FLAG_IN_BF16) return launch_gather<FAN, MODE, __nv_bfloat16>(A, grid, S, s);
    if (flags & CTP_FLAG_IN_FP16) return launch_gather<FAN, MODE, __half>(A, grid, S, s);
    return launch_gather<FAN, MODE, float>(A, grid, S, s);
}

}  // namespace

bool gather_applies(const ctp_geometry& g, int geom, GatherMode mode, bool slices_match_rows) {
    if (mode == kGatherPixel && g.nv != 1) return false;
    if (g.nview == 0 || g.nu == 0 || g.nx == 0 || g.ny == 0 || g.nz == 0) return false;
    if (mode == kGatherAdjoint) {
        if (!slices_match_rows) return false;
        // the fan's position within a cell is expanded in the angular cell size
        if (geom == 0 && !(fabs((double)g.du) <= 0.01)) return false;
    }
    double zmax;
    return gather_window(g, geom, &zmax) > 0 && g.nview <= 65535;
}

size_t gather_bytes(const ctp_geometry& g, int geom, GatherMode mode) {
    size_t need = weight_bytes(g, geom, mode);
    const int parts = gather_most_parts(g, geom);
    if (parts > 1) need += align_up((size_t)parts * g.nbatch * g.nz * g.ny * g.nx * sizeof(float));
    return need;
}

int gather_bp(void* img, const void* prj, const float* deg, const ctp_geometry& g, int geom, GatherMode mode,
              unsigned flags, char* ws, cudaStream_t s) {
    GatherArgs A;
    A.prj = prj;
    A.g = make_grid(g);
    A.d = make_det(g);
    A.dso = g.dso;
    A.nview = (int)g.nview;
    A.nslices = (int)(g.nbatch * g.nz);
    double zmax;
    A.win = gather_window(g, geom, &zmax);
    A.wide = zmax > 0.12;
    A.parts = gather_parts(g, geom, A.vper);
    A.mode = (int)mode;
    A.deg = deg;
    A.part_elems = g.nbatch * g.nz * g.ny * g.nx;
    A.accumulate = (flags & CTP_FLAG_ZERO_OUT) ? 0 : 1;
    A.out_lp = (flags & CTP_FLAG_OUT_BF16) ? 1 : (flags & CTP_FLAG_OUT_FP16) ? 2 : 0;
    A.one_to_one = mode == kGatherAdjoint ? 1 : 0;
    float* lw = reinterpret_cast<float*>(ws);
    float* partial = reinterpret_cast<float*>(ws + weight_bytes(g, geom, mode));
    int rc = CTP_OK;
    A.lw = nullptr;
    if (weight_bytes(g, geom, mode)) {
        cell_weights_kernel<<<dim3((unsigned)((g.nu + 127) / 128), (unsigned)g.nview), 128, 0, s>>>(
            lw, deg, (int)g.nview, (int)mode, A.g, A.d);
        if ((rc = check_launch("cell_weights_kernel"))) return rc;
        A.lw = lw;
    }
    A.img = A.parts > 1 ? (void*)partial : img;
    const int S = slices_per_cta(g, geom);
    const dim3 grid((unsigned)(((g.nx + kT - 1) / kT) * ((g.ny + kT - 1) / kT)),
                    (unsigned)((g.nbatch * g.nz + S - 1) / S), (unsigned)A.parts);
    if (mode == kGatherPixel)
        rc = geom == 1 ? launch_gather<false, kGatherPixel, float>(A, grid, S, s)
                       : launch_gather<true, kGatherPixel, float>(A, grid, S, s);
    else if (geom == 1)
        rc = mode == kGatherAdjoint ? launch_gather_type<false, kGatherAdjoint>(A, grid, S, flags, s)
                                    : launch_gather_type<false, kGatherMean>(A, grid, S, flags, s);
    else if (mode == kGatherMean) rc = launch_gather_type<true, kGatherMean>(A, grid, S, flags, s);
    else if (mode == kGatherFbp) rc = launch_gather_type<true, kGatherFbp>(A, grid, S, flags, s);
    else rc = launch_gather_type<true, kGatherAdjoint>(A, grid, S, flags, s);
    if (rc || A.parts == 1) return rc;
    gather_sum_kernel<<<(unsigned)std::min<size_t>((A.part_elems + 255) / 256, 148 * 8), 256, 0, s>>>(
        img, partial, A.parts, A.part_elems, A.out_lp, A.accumulate);
    return check_launch("gather_sum_kernel");
}

}  // namespace ctp
