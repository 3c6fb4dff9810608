// The quad form's kernels of kLo to kHi rows per lane, in FP32x2 or (kDouble) one read a half in FP64, each
// range instantiated in its quad_*.cu so that they compile side by side.
#pragma once
#include "kernels.cuh"

namespace fgkl {

template <bool kDouble, int kLo, int kHi>
struct QuadRange {
  static size_t scratch(int rows, int max_slots, int max_nodes, int max_segs);
  static int occupancy(int rows, int warps, int* threads);
  static cudaError_t launch(int rows, int blocks, const LaunchArgs& a, cudaStream_t s, int warps);
};

}  // namespace fgkl
