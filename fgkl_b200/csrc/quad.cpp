// Choice among the quad form's ranges.
#include "quad.cuh"

namespace fgkl {

namespace {
template <class F>
auto quad_range(Kind k, int rows, F&& f) {
  if (k == Kind::kPairF64) return f(QuadRange<true, 2, kQuadMaxRows>{});
  if (rows <= 8) return f(QuadRange<false, 2, 8>{});
  if (rows <= 10) return f(QuadRange<false, 10, 10>{});
  return f(QuadRange<false, 12, kQuadMaxRows>{});
}
}  // namespace

size_t quad_scratch_bytes(Kind k, int rows, int max_slots, int max_nodes, int max_segs) {
  return quad_range(k, rows, [&](auto q) { return q.scratch(rows, max_slots, max_nodes, max_segs); });
}

void quad_occupancy(Kind k, int rows, int* blocks, int* threads, int warps) {
  *blocks = quad_range(k, rows, [&](auto q) { return q.occupancy(rows, warps, threads); });
}

cudaError_t quad_launch(Kind k, int rows, int blocks, const LaunchArgs& args, cudaStream_t stream, int warps) {
  return quad_range(k, rows, [&](auto q) { return q.launch(rows, blocks, args, stream, warps); });
}

}  // namespace fgkl
