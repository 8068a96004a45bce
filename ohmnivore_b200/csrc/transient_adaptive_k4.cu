// Adaptive transient kernel, 4 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
AdaptFn adaptive_kernel_for<4>() { return adaptive_kernel<4>; }

}  // namespace ohm
