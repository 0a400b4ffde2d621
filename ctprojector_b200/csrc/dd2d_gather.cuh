// dd2d_gather.cuh -- tiled gather back projection of the distance-driven
// fan-beam and parallel-beam operators (dd2d_gather.cu), called by dd2d.cu.
#pragma once

#include "ctp_common.cuh"

namespace ctp {

enum GatherMode { kGatherMean = 0, kGatherFbp = 1, kGatherAdjoint = 2, kGatherPixel = 3 };

// Whether the geometry suits the tiled kernels (the detector window of a tile
// fits shared memory; the adjoint: slices projected one to one onto detector
// rows; pixel-driven: one detector row), and the scratch of one call.
bool gather_applies(const ctp_geometry& g, int geom, GatherMode mode, bool slices_match_rows);
size_t gather_bytes(const ctp_geometry& g, int geom, GatherMode mode);

int gather_bp(void* img, const void* prj, const float* deg, const ctp_geometry& g, int geom, GatherMode mode,
              unsigned flags, char* ws, cudaStream_t s);

}  // namespace ctp
