// Batched BM3D stages: many planes of different sizes and noise levels in one
// persistent launch per stage. Each CTA pulls (image, tile) work items from a
// device counter; an image's items are its tiles, numbered after the items of
// the images before it (tile_base is the exclusive prefix sum). The per-tile
// work is the same body as the single-plane kernels, so results are
// bit-identical to per-plane calls.
#pragma once

#include "bm3d_generic.cuh"

namespace bm3d {

// Dynamic shared memory starts with the CTA's current item (16 bytes) and a copy
// of its image's arguments: the tile body reads them all through, and a
// shared-memory copy takes one address register and no global loads.
constexpr int kBatchHeader = 16 + static_cast<int>((sizeof(StageArgs<float>) + 15) / 16 * 16);

// GEN: -1 for the register-resident body, else the generic body's BSC.
template <typename T, bool WIENER, int NPL, int KS, int GEN>
__global__ void __launch_bounds__((GEN >= 0 ? generic_max_warps(sizeof(T), GEN) : stage_max_warps<T>()) * kWarp, 1)
    batch_stage_kernel(const StageArgs<T> *__restrict__ args, const int *__restrict__ tile_base,
                       int nimg, int *counter)
{
    extern __shared__ __align__(16) unsigned char smem[];
    int *item = reinterpret_cast<int *>(smem);
    StageArgs<T> &a = *reinterpret_cast<StageArgs<T> *>(smem + 16);
    int held = -1;  // the image whose arguments are held
    const int total = tile_base[nimg];
    const unsigned avail = dynamic_smem_bytes() - kBatchHeader;
    for (;;) {
        if (threadIdx.x == 0) *item = atomicAdd(counter, 1);
        __syncthreads();
        const int it = *item;
        if (it >= total) break;
        int lo = 0, hi = nimg - 1;  // last image whose first item is <= it
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (tile_base[mid] <= it) lo = mid;
            else hi = mid - 1;
        }
        if (lo != held) {  // uniform over the CTA; no warp reads them between items
            static_assert(sizeof(StageArgs<T>) % 8 == 0, "copied by 8-byte words");
            const auto *from = reinterpret_cast<const unsigned long long *>(args + lo);
            auto *to = reinterpret_cast<unsigned long long *>(&a);
            for (int i = threadIdx.x; i < static_cast<int>(sizeof(StageArgs<T>) / 8); i += blockDim.x)
                to[i] = from[i];
            held = lo;
            __syncthreads();
        }
        unsigned char *body = smem + kBatchHeader;
        if constexpr (GEN >= 0 && NPL == 3) generic_tile_body_seq3<T, WIENER, GEN>(a, it - tile_base[lo], body, avail);
        else if constexpr (GEN >= 0) generic_tile_body<T, WIENER, NPL, GEN>(a, it - tile_base[lo], body, avail);
        else if constexpr (NPL == 3) stage_tile_body_seq3<T, WIENER, KS>(a, it - tile_base[lo], body, avail);
        else stage_tile_body<T, WIENER, NPL, KS>(a, it - tile_base[lo], body, avail);
        __syncthreads();  // every thread has read *item before it is replaced
    }
}

// Zero each plane's sums, fold its max finite |src| and count its non-finite
// pixels (grid.y = plane).
template <typename T> __global__ void prep_batch_kernel(const PlaneJob<T> *planes)
{
    prep_plane<T>(planes[blockIdx.y], blockIdx.x, gridDim.x);
}

// dst = num / den for every plane (grid.y = plane), a CTA per tile; planes
// smaller than the grid leave CTAs without one.
template <typename T>
__global__ void __launch_bounds__(256) normalize_batch_kernel(const PlaneJob<T> *planes)
{
    const PlaneJob<T> q = planes[blockIdx.y];
    if (static_cast<int>(blockIdx.x) < normalize_tiles<T>(q.width, q.height))
        normalize_job(q, static_cast<int>(blockIdx.x));
}

}  // namespace bm3d
