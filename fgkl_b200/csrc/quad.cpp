// Choice among the quad form's ranges.
#include "quad.cuh"

namespace fgkl {

namespace {
template <class F>
auto quad_range(int rows, F&& f) {
  if (rows <= 8) return f(QuadRange<2, 8>{});
  if (rows <= 10) return f(QuadRange<10, 10>{});
  return f(QuadRange<12, kQuadMaxRows>{});
}
}  // namespace

size_t quad_scratch_bytes(int rows, int max_slots, int max_nodes, int max_segs) {
  return quad_range(rows, [&](auto q) { return q.scratch(rows, max_slots, max_nodes, max_segs); });
}

void quad_occupancy(int rows, int* blocks, int* threads) {
  *blocks = quad_range(rows, [&](auto q) { return q.occupancy(rows, threads); });
}

cudaError_t quad_launch(int rows, int blocks, const LaunchArgs& args, cudaStream_t stream) {
  return quad_range(rows, [&](auto q) { return q.launch(rows, blocks, args, stream); });
}

}  // namespace fgkl
