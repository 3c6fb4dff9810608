// The quad form at 10 rows per lane.
#include "quad_kernel.cuh"

namespace fgkl {
template struct QuadRange<false, 10, 10>;
}  // namespace fgkl
