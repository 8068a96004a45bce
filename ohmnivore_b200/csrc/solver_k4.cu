// Persistent solver, 4 lane(s) per row.
#include "internal.cuh"

template <>
KernelPair<KernelFn> persistent_kernel_for<4>() { return {ohm::persistent_solver<4>, ohm::persistent_solver_wide<4>}; }
