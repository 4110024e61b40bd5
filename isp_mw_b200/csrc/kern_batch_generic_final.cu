// Persistent batched stage kernels, final stage, generic bodies: BlockSize 8, 11 and
// the others, one plane or three planes sharing luma groups.
#include "kern_unit.cuh"

BM3D_KERNEL_UNIT(batch_generic_final)

namespace bm3d {
template const void *batch_kernel_fn<true, 1, 1, 0>();
template const void *batch_kernel_fn<true, 3, 1, 0>();
template const void *batch_kernel_fn<true, 1, 1, 8>();
template const void *batch_kernel_fn<true, 3, 1, 8>();
template const void *batch_kernel_fn<true, 1, 1, 11>();
template const void *batch_kernel_fn<true, 3, 1, 11>();
}  // namespace bm3d
