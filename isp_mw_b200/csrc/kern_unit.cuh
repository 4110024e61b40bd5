// Shared part of the kernel translation units (kern_*.cu): the definitions
// behind the handles of bm3d_kernels.h and this unit's table upload.
#pragma once

#include "bm3d_batch.cuh"
#include "bm3d_kernels.h"

namespace bm3d {

template <typename T, bool W, int NPL, int KS> const void *stage_kernel_fn()
{
    return reinterpret_cast<const void *>(&stage_kernel<T, W, NPL, KS>);
}

template <typename T, bool W, int NPL, int BSC> const void *generic_kernel_fn()
{
    return reinterpret_cast<const void *>(&generic_stage_kernel<T, W, NPL, BSC>);
}

template <bool W, int NPL, int KS, int GEN> const void *batch_kernel_fn()
{
    return reinterpret_cast<const void *>(&batch_stage_kernel<float, W, NPL, KS, GEN>);
}

static cudaError_t upload_dct_tables_here(const DctTables &t) { return cudaMemcpyToSymbol(c_dct, &t, sizeof(t)); }

}  // namespace bm3d

#define BM3D_KERNEL_UNIT(name)                                                      \
    cudaError_t bm3d_upload_dct_tables_##name(const bm3d::DctTables &t)            \
    {                                                                               \
        return bm3d::upload_dct_tables_here(t);                                     \
    }
