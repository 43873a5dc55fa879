// Gather kernels for bf16 channel-data storage (one translation unit per storage type
// so the library compiles in parallel).
#include "das_launch.cuh"

namespace mach_b200 {
template cudaError_t launch_das<kBF16>(const DasArgs&, int, const LaunchPlan&, cudaStream_t);
template cudaError_t launch_das_staged<kBF16>(const DasArgs&, const StagedArgs&, const CUtensorMap&, int,
                                             const LaunchPlan&, cudaStream_t);
template cudaError_t launch_lane_voxel_persistent<kBF16>(int, int, bool, const PersistentLaunch&, cudaStream_t);
template cudaError_t launch_staged_persistent<kBF16>(int, int, const PersistentLaunch&, cudaStream_t);
template cudaError_t launch_das_ensemble<kBF16>(const DasArgs&, const StagedArgs&, const EnsembleArgs&,
                                               const CUtensorMap&, int, size_t, cudaStream_t);
template cudaError_t launch_das_frame_lane<kBF16>(const DasArgs&, const FrameLaneArgs&, int, const LaunchPlan&,
                                                cudaStream_t);
template cudaError_t launch_frame_lane_persistent<kBF16>(int, int, bool, const PersistentLaunch&, cudaStream_t);
template cudaError_t launch_frame_group_persistent<kBF16>(int, int, bool, const PersistentLaunch&,
                                                               cudaStream_t);
}  // namespace mach_b200
