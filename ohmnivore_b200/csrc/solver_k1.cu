// Persistent solver, 1 lane(s) per row.
#include "internal.cuh"

template <>
KernelPair<KernelFn> persistent_kernel_for<1>() { return {ohm::persistent_solver<1>, ohm::persistent_solver_wide<1>}; }
