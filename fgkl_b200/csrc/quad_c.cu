// The quad form at 12 to 14 rows per lane.
#include "quad_kernel.cuh"

namespace fgkl {
template struct QuadRange<false, 12, 14>;
}  // namespace fgkl
