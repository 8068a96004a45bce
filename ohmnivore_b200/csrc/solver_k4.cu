// Persistent solver, 4 lane(s) per row.
#include "internal.cuh"

template <>
KernelFn persistent_kernel_for<4>() { return ohm::persistent_solver<4>; }
