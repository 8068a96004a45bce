// Adaptive transient kernel, 1 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<AdaptFn> adaptive_kernel_for<1>() {
    return {adaptive_kernel<1, GridTeam>, adaptive_kernel<1, GlobalTeam>};
}

}  // namespace ohm
