// Persistent solver, 16 lane(s) per row.
#include "internal.cuh"

template <>
KernelPair<KernelFn> persistent_kernel_for<16>() { return {ohm::persistent_solver<16>, ohm::persistent_solver_wide<16>}; }
