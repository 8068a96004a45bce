// Fixed-step transient kernel, 1 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<TranFn> transient_kernel_for<1>() {
    return {transient_kernel<1, GridTeam>, transient_kernel<1, GlobalTeam>};
}

}  // namespace ohm
