// The quad form at 2 to 8 rows per lane.
#include "quad_kernel.cuh"

namespace fgkl {
template struct QuadRange<false, 2, 8>;
}  // namespace fgkl
