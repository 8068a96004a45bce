// Persistent solver, 32 lane(s) per row.
#include "internal.cuh"

template <>
KernelPair<KernelFn> persistent_kernel_for<32>() { return {ohm::persistent_solver<32>, ohm::persistent_solver_wide<32>}; }
