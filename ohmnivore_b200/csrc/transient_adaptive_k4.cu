// Adaptive transient kernel, 4 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<AdaptFn> adaptive_kernel_for<4>() {
    return {adaptive_kernel<4, GridTeam>, adaptive_kernel<4, GlobalTeam>};
}

}  // namespace ohm
