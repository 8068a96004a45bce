// Fixed-step transient kernel, 1 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
TranFn transient_kernel_for<1>() { return transient_kernel<1>; }

}  // namespace ohm
