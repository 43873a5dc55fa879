// Tile counts of the voxel-per-lane kernels when the voxel grid is found on the device (plain C++,
// shared by the planner and its CPU test).
#pragma once

#include <cstdint>

namespace mach_b200 {

// Smallest contiguous and outer extents that a probed grid is tiled by.
constexpr int64_t kProbeMinFast = 16;
constexpr int64_t kProbeMinOuter = 128;

// Tiles of wf x (voxels / wf) voxels that a launch needs for any extent that the probe may report.
// For a contiguous extent f >= 16 and an outer extent o >= 128 with f o = n_vox, the tiles are
// ceil(o / q) ceil(f / wf) with q = voxels / wf, at most (o / q + 1) (f / wf + 1), which is at most
// (1 + q / 128) (1 + wf / 16) n_vox / voxels; without a grid ceil(n_vox / voxels) are needed, fewer.
inline int64_t probed_tiles(int64_t n_vox, int voxels, int wf) {
    const double q = static_cast<double>(voxels) / wf;
    const double bound = (1.0 + q / kProbeMinOuter) * (1.0 + static_cast<double>(wf) / kProbeMinFast) *
                         static_cast<double>(n_vox) / voxels;
    return static_cast<int64_t>(bound) + 2;
}

}  // namespace mach_b200
