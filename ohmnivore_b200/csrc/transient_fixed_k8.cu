// Fixed-step transient kernel, 8 lane(s) per row.
#include "transient_kernel.cuh"

namespace ohm {

template <>
KernelPair<TranFn> transient_kernel_for<8>() {
    return {transient_kernel<8, GridTeam>, transient_kernel<8, GlobalTeam>};
}

}  // namespace ohm
