// Persistent solver, 8 lane(s) per row.
#include "internal.cuh"

template <>
KernelPair<KernelFn> persistent_kernel_for<8>() { return {ohm::persistent_solver<8>, ohm::persistent_solver_wide<8>}; }
