// The quad form in FP64 (one read on each half of the lanes).
#include "quad_kernel.cuh"

namespace fgkl {
template struct QuadRange<true, 2, 14>;
}  // namespace fgkl
