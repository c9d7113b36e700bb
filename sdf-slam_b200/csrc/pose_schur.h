// Schur complements on the FP64 tensor cores (pose_schur.cu): of the grid fronts
// into their pose root, and of a level's children into their parents.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace sdfgpu {

/// What KPoseSchur reads and writes besides the view.
struct PoseSchurArgs {
  const PoseTask* tasks;
  int64_t count;
  const int32_t* fronts;   // Symbolic::pose_fronts
  const uint64_t* mask;    // Symbolic::pose_mask
  const int32_t* start;    // Symbolic::pose_start
  const double* dvec;
  double* parts;           // workspace tiles of the split tiles
  int32_t* counters;       // arrivals per split tile (zero between launches)
};

/// Doubles of the workspace of `slots` part tiles.
inline size_t PoseSchurDoubles(int64_t slots) {
  return static_cast<size_t>(slots) * kPoseTile * kPoseTile;
}

/// Subtracts the products L D L^T of every front's pose rows from the pose
/// roots; fp32: the view may hold FP32 fronts (a mixed solve). Returns the
/// number of kernels launched.
int LaunchPoseSchur(const DeviceView& V, const PoseSchurArgs& args, bool fp32, cudaStream_t stream);

/// Adds the children's Schur complements into the fronts of `count` > 0 tile
/// tasks (one level, FP64 fronts).
void LaunchChildSchur(const DeviceView& V, const ChildTask* tasks, int64_t count, const ChildEntry* entries,
                      const double* dvec, cudaStream_t stream);

}  // namespace sdfgpu
