// Fixed-step transient kernel, 4 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<TranFn> transient_kernel_for<4>() {
    return {transient_kernel<4, GridTeam>, transient_kernel<4, GlobalTeam>};
}

}  // namespace ohm
