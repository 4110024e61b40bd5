// Generic stage kernels (BlockSize <= 16, GroupSize <= 32), float: BlockSize 8,
// 11 and the others.
#include "kern_unit.cuh"

BM3D_KERNEL_UNIT(generic_f32)

namespace bm3d {
template const void *generic_kernel_fn<float, false, 1, 0>();
template const void *generic_kernel_fn<float, false, 3, 0>();
template const void *generic_kernel_fn<float, true, 1, 0>();
template const void *generic_kernel_fn<float, true, 3, 0>();
template const void *generic_kernel_fn<float, false, 1, 8>();
template const void *generic_kernel_fn<float, false, 3, 8>();
template const void *generic_kernel_fn<float, true, 1, 8>();
template const void *generic_kernel_fn<float, true, 3, 8>();
template const void *generic_kernel_fn<float, false, 1, 11>();
template const void *generic_kernel_fn<float, false, 3, 11>();
template const void *generic_kernel_fn<float, true, 1, 11>();
template const void *generic_kernel_fn<float, true, 3, 11>();
}  // namespace bm3d
