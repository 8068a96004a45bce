// Persistent solver, 8 lane(s) per row.
#include "internal.cuh"

template <>
KernelFn persistent_kernel_for<8>() { return ohm::persistent_solver<8>; }
