// fdtd_flat_bf16.cu -- the flat step kernels of one storage type.
#include "fdtd_flat_kernels.cuh"

FLAT_INSTANCE(__nv_bfloat16)
