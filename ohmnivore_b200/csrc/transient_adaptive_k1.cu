// Adaptive transient kernel, 1 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
AdaptFn adaptive_kernel_for<1>() { return adaptive_kernel<1>; }

}  // namespace ohm
