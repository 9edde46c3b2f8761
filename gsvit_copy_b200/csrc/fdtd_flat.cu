// fdtd_flat.cu -- launches of the flat step kernels (fdtd_flat_kernels.cuh).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/gsvit_b200.h"
#include "fdtd_flat.cuh"

template <class T>
cudaError_t flat_h_t(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, cudaStream_t st);
template <class T>
cudaError_t flat_e_t(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, bool ade, int npoles, bool beside_h, cudaStream_t st);

int flat_width(int storage, int zr)
{
    if (storage == FDTD_STORE_F64) return zr % 2 == 0 ? 2 : 1;
    return zr % 4 == 0 ? 4 : 1;
}

namespace {

cudaError_t flat_h(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, int storage, cudaStream_t st)
{
    if (!l.n) return cudaSuccess;
    if (storage == FDTD_STORE_F64) return flat_h_t<double>(p, plans, l, width, st);
    if (storage == FDTD_STORE_F16) return flat_h_t<__half>(p, plans, l, width, st);
    if (storage == FDTD_STORE_BF16) return flat_h_t<__nv_bfloat16>(p, plans, l, width, st);
    return flat_h_t<float>(p, plans, l, width, st);
}

cudaError_t flat_e(const DevPlan *p, const DevPlan *plans, const FlatList &l, int width, bool ade, int npoles, int storage,
                   bool beside_h, cudaStream_t st)
{
    if (!l.n) return cudaSuccess;
    if (storage == FDTD_STORE_F64) return flat_e_t<double>(p, plans, l, width, ade, npoles, beside_h, st);
    if (storage == FDTD_STORE_F16) return flat_e_t<__half>(p, plans, l, width, ade, npoles, beside_h, st);
    if (storage == FDTD_STORE_BF16) return flat_e_t<__nv_bfloat16>(p, plans, l, width, ade, npoles, beside_h, st);
    return flat_e_t<float>(p, plans, l, width, ade, npoles, beside_h, st);
}

}  // namespace

cudaError_t launch_flat_h(const DevPlan &p, const FlatList &l, int width, int storage, cudaStream_t st)
{
    return flat_h(&p, nullptr, l, width, storage, st);
}

cudaError_t launch_flat_e(const DevPlan &p, const FlatList &l, int width, bool ade, int npoles, int storage, bool beside_h,
                          cudaStream_t st)
{
    return flat_e(&p, nullptr, l, width, ade, npoles, storage, beside_h, st);
}

cudaError_t launch_flat_h_batch(const DevPlan *plans, const FlatList &l, int width, int storage, cudaStream_t st)
{
    return flat_h(nullptr, plans, l, width, storage, st);
}

cudaError_t launch_flat_e_batch(const DevPlan *plans, const FlatList &l, int width, bool ade, int npoles, int storage,
                                cudaStream_t st)
{
    return flat_e(nullptr, plans, l, width, ade, npoles, storage, false, st);
}
