// Adaptive transient kernel, 8 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<AdaptFn> adaptive_kernel_for<8>() {
    return {adaptive_kernel<8, GridTeam>, adaptive_kernel<8, GlobalTeam>};
}

}  // namespace ohm
