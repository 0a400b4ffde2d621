// siddon_columns.cuh -- column-wise Siddon cone projectors of upright views
// (siddon_columns.cu), called by siddon.cu.
#pragma once

#include "ctp_common.cuh"

namespace ctp {

// One view in voxel coordinates (x, y, z / voxel size from the grid's low
// corner): the source, and the direction to cell (iu, iv), alpha = 1 at the
// panel: (dx0 + iu ux, dy0 + iu uy, k0 + iv kv).
struct UprightView {
    double sx, sy, zs;
    double dx0, dy0, ux, uy;
    double k0, kv;
    double det;   // (ux, uy) x (dx0, dy0)
    int upright;  // 0: the ray-driven kernels take this view
    int turned;   // k0 and kv count the rows from the panel's other end (columns_bp)
};

// Device memory of one call: the views, and rest[0] = the number of views that
// are left to the ray-driven kernels, rest[1..] those views.
struct ColumnsPlan {
    UprightView* views = nullptr;
    int* rest = nullptr;
};

// Whether the sizes suit the column kernels, and the scratch they take.
bool columns_fp_applies(const ctp_geometry& g, unsigned flags);
size_t columns_fp_bytes(const ctp_geometry& g, unsigned flags);
bool columns_bp_applies(const ctp_geometry& g, unsigned flags);
size_t columns_bp_bytes(const ctp_geometry& g);

// The upright views of a call; the caller runs the ray-driven kernel on
// plan.rest afterwards.  columns_bp adds to img.
int columns_fp(ColumnsPlan& plan, char* scratch, void* prj, const void* img, const float* dc, const float* du_,
               const float* dv_, const float* sr, const ctp_geometry& g, unsigned flags, cudaStream_t s);
int columns_bp(ColumnsPlan& plan, char* scratch, float* img, const void* prj, const float* dc, const float* du_,
               const float* dv_, const float* sr, const ctp_geometry& g, unsigned flags, cudaStream_t s);

}  // namespace ctp
