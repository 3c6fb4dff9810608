// Definitions of a range of the quad form (quad.cuh): kLo, kLo + 2, .. kHi rows per lane.
#pragma once
#include "plain_kernel.cuh"
#include "quad.cuh"

namespace fgkl {

namespace {
constexpr int kQuadWarps = block_warps<kQuadLanes>();

// Calls f with the compile-time value of `rows`, one of R, R + 2, .. kHi.
template <int R, int kHi, class F>
void rows_at(int rows, F&& f) {
  if (rows == R)
    f(std::integral_constant<int, R>{});
  else if constexpr (R + 2 <= kHi)
    rows_at<R + 2, kHi>(rows, f);
}

template <bool kDouble>
using QuadPolicy = std::conditional_t<kDouble, OneF64Table, PackedF32>;

template <bool kDouble, int R>
constexpr size_t quad_smem(int warps) {
  return warps * Layout<QuadPolicy<kDouble>, R>::kSmemPerWarp;
}

// Warps of a block when `warps` are asked for.
constexpr int quad_warps(int warps) { return warps < kQuadWarps ? warps : kQuadWarps; }
}  // namespace

template <bool kDouble, int kLo, int kHi>
size_t QuadRange<kDouble, kLo, kHi>::scratch(int rows, int max_slots, int max_nodes, int max_segs) {
  size_t bytes = 0;
  rows_at<kLo, kHi>(rows, [&](auto r) { bytes = scratch_size<QuadPolicy<kDouble>, decltype(r)::value>(max_slots, max_nodes, max_segs); });
  return bytes;
}

template <bool kDouble, int kLo, int kHi>
int QuadRange<kDouble, kLo, kHi>::occupancy(int rows, int warps, int* threads) {
  int blocks = 0;
  warps = quad_warps(warps);
  *threads = warps * 32;
  rows_at<kLo, kHi>(rows, [&](auto r) {
    constexpr int R = decltype(r)::value;
    static std::atomic<int> cache[kQuadWarps][kMaxDevices];
    blocks = resident_blocks(pairhmm_kernel<QuadPolicy<kDouble>, R, kQuadLanes>, quad_smem<kDouble, R>(warps), warps * 32, cache[warps - 1],
                             quad_smem<kDouble, R>(kQuadWarps));
  });
  return blocks;
}

template <bool kDouble, int kLo, int kHi>
cudaError_t QuadRange<kDouble, kLo, kHi>::launch(int rows, int blocks, const LaunchArgs& a, cudaStream_t s, int warps) {
  warps = quad_warps(warps);
  rows_at<kLo, kHi>(rows, [&](auto r) {
    constexpr int R = decltype(r)::value;
    pairhmm_kernel<QuadPolicy<kDouble>, R, kQuadLanes><<<blocks, warps * 32, quad_smem<kDouble, R>(warps), s>>>(a);
  });
  return cudaGetLastError();
}

}  // namespace fgkl
