// Persistent batched stage kernels, final stage: register-resident bodies (KS =
// 4 and 1), one plane or three planes sharing luma groups.
#include "kern_unit.cuh"

BM3D_KERNEL_UNIT(batch_final)

namespace bm3d {
template const void *batch_kernel_fn<true, 1, 4, -1>();
template const void *batch_kernel_fn<true, 1, 1, -1>();
template const void *batch_kernel_fn<true, 3, 4, -1>();
template const void *batch_kernel_fn<true, 3, 1, -1>();
}  // namespace bm3d
