// fdtd_flat_f16.cu -- the flat step kernels of one storage type.
#include "fdtd_flat_kernels.cuh"

FLAT_INSTANCE(__half)
