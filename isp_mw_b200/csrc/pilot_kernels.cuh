// Kernels of the learned pilot: an 8-layer 3 x 3 convolutional network with
// 48 hidden channels, ReLU, BF16 weights and activations and FP32
// accumulation, whose output (noisy + predicted residual) stands in for the
// BM3D basic estimate that feeds the final (Wiener) stage.
//
// Layer 1 (2 -> 48: the noisy plane and a noise-level plane) and layer 8
// (48 -> 1) are small and run on the FP32 pipes. Layers 2-7 (48 -> 48, 98 %
// of the arithmetic) and their backward passes run on the tensor cores
// (tcgen05, accumulators in tensor memory).
//
// Activations are BF16, NHWC with 48 channels (96 bytes per pixel), images
// stored back to back. A 48 -> 48 layer works on tiles of 16 x 8 output pixels
// (the MMA's M = 128). The tile's input, with a one-pixel halo, sits in shared
// memory as 18 columns of [channel / 8][row (10)][channel % 8] BF16 -- 960
// bytes per column. A core matrix (8 rows x 16 bytes) may start at any 16-byte
// boundary, so the 128 x 48 operand of tap (dy, dx) starts dx columns and dy
// rows into the tile (K-major, no swizzle: LBO = 160 bytes between 8-channel
// groups, SBO = 960 bytes between 8-pixel columns), and each tap is three
// MMAs of K = 16 with no data movement. Read as an MN-major operand the same
// tile gives the weight gradient's pixel-reduction MMAs: the three dx shifts
// of 48 channels are 18 channel groups 160 bytes apart (960 = 6 x 160),
// columns LBO = 960 apart.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "pilot_tc.cuh"

namespace pilot {

constexpr int kC = 48;                          // hidden channels
constexpr int kTX = 16, kTY = 8;                // output tile (128 pixels)
constexpr int kHaloRows = kTY + 2;              // 10 input rows per column
constexpr int kGroupBytes = kHaloRows * 16;     // 160: one 8-channel group of a halo column
constexpr int kHaloColBytes = 6 * kGroupBytes;  // 960: one halo column
constexpr int kCols = kTX + 2;                  // 18 input columns
constexpr int kTileBytes = kCols * kHaloColBytes;  // 17280: the input tile with its halo
constexpr int kTileChunks = kTileBytes / 16;    // 1080 16-byte chunks
constexpr int kTapBytes = kC * kC * 2;          // 4608: one tap, [co / 8][ci / 8][co % 8][ci % 8]
constexpr int kWeightBytes = 9 * kTapBytes;     // 41472
constexpr int kConvThreads = 128;               // four warps: one per 32 TMEM lanes
constexpr int kAccCols = 64;                    // TMEM columns per accumulator (48 used)
constexpr uint32_t kWaitLimit = 1u << 24;       // polls before a wait gives up
constexpr uint32_t kIdescFwd = instr_desc_bf16(128, kC, false, false);

// Parameters: W1 48x2x3x3 + b1, six 48x48x3x3 + biases, W8 1x48x3x3 + b8.
constexpr int kW1 = kC * 2 * 9, kWmid = kC * kC * 9, kW8 = kC * 9;
constexpr int kOffB1 = kW1;
constexpr int kOffMid = kOffB1 + kC;  // layer l (2..7): W at kOffMid + (l - 2) (kWmid + kC)
constexpr int kOffW8 = kOffMid + 6 * (kWmid + kC);
constexpr int kOffB8 = kOffW8 + kW8;
constexpr int kParams = kOffB8 + 1;
__host__ __device__ constexpr int off_w(int layer) { return kOffMid + (layer - 2) * (kWmid + kC); }
__host__ __device__ constexpr int off_b(int layer) { return off_w(layer) + kWmid; }

enum ConvMode { kBiasRelu = 0, kBias = 1, kMaskPrev = 2 };

struct ConvArgs {
    const __nv_bfloat16 *x;    // input activations [n][h][w][48]
    __nv_bfloat16 *y;          // output [n][h][w][48]
    const uint4 *wt;           // packed weights (kWeightBytes)
    const float *bias;         // [48]: kBiasRelu, kBias
    const __nv_bfloat16 *aux;  // kMaskPrev: y = acc where aux > 0, else 0
    int n, h, w;
    int tiles_x, tiles_y, tiles;
    int mode;
    unsigned *err;             // set when a wait gave up
};

__device__ __forceinline__ void tile_origin(int tile, int tiles_x, int tiles_y, int &img, int &y0,
                                            int &x0)
{
    const int per = tiles_x * tiles_y;
    img = tile / per;
    const int r = tile - img * per;
    const int ty = r / tiles_x;
    y0 = ty * kTY;
    x0 = (r - ty * tiles_x) * kTX;
}

// A tile's input with its one-pixel halo (zero outside the image): chunk
// (column, channel / 8, row) at byte 16 ((column * 6 + channel / 8) * 10 + row)
// (row 0 = y0 - 1). Thread i copies the i-th 16-byte chunk of the halo in
// global order (row, column, channel / 8), so a warp reads 512 contiguous bytes
// of one input row.
__device__ __forceinline__ void load_conv_tile(const __nv_bfloat16 *x, int h, int w, int img, int y0,
                                               int x0, unsigned char *buf)
{
    for (int i = threadIdx.x; i < kTileChunks; i += blockDim.x) {
        const int yy = i / (kCols * 6);
        const int r = i - yy * (kCols * 6);
        const int col = r / 6;
        const int ch = r - col * 6;
        const int gy = y0 + yy - 1, gx = x0 + col - 1;
        const bool ok = gy >= 0 && gy < h && gx >= 0 && gx < w;
        const __nv_bfloat16 *src =
            ok ? x + ((static_cast<long long>(img) * h + gy) * w + gx) * kC + ch * 8 : x;
        cp_async16(buf + ((col * 6 + ch) * kHaloRows + yy) * 16, src, ok);
    }
    cp_async_commit();
}

// 27 MMAs: 9 taps x 3 steps of 16 input channels, into accumulator d_tmem.
// The operand tile's tap (dy, dx) starts dy * DY + dx * DX bytes in. Issued
// by one thread, so the loop is fully unrolled and every descriptor is a base
// descriptor plus a compile-time constant: the start-address field holds
// address >> 4 in 14 bits and shared addresses stay below 256 KB, so the sum
// never carries out of it. (Rebuilding both descriptors per MMA made this
// thread's dependent scalar chain, not the tensor pipe, set the pace.)
template <int DY, int DX>
__device__ __forceinline__ void issue_tile_mmas(uint32_t a_base, uint32_t w_base, uint32_t d_tmem)
{
    const uint64_t ad0 = smem_desc(a_base, kGroupBytes, kHaloColBytes);
    const uint64_t bd0 = smem_desc(w_base, 128, 768);
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const uint64_t ad = ad0 + static_cast<uint64_t>(
                                          ((tap / 3) * DY + (tap % 3) * DX + s * 2 * kGroupBytes) >> 4);
            const uint64_t bd = bd0 + static_cast<uint64_t>((tap * kTapBytes + s * 256) >> 4);
            mma_bf16(d_tmem, ad, bd, kIdescFwd, tap > 0 || s > 0);
        }
    }
}

// The cp.async kernel's tiles: columns kHaloColBytes apart, rows 16 bytes.
__device__ __forceinline__ void issue_conv_mmas(uint32_t a_base, uint32_t w_base, uint32_t d_tmem)
{
    issue_tile_mmas<16, kHaloColBytes>(a_base, w_base, d_tmem);
}

// Epilogue of one tile. Each thread reads its pixel's (TMEM lane m = column
// * 8 + row) 48 accumulators, applies the bias (and ReLU) and rounds to BF16
// into `stage` at m * kOutPitch (a 112-byte pitch: the eight lanes of a
// 16-byte store phase land on distinct banks). Then the 128 threads write the
// tile's rows out, consecutive threads on consecutive 16-byte chunks of a row
// (16 pixels x 96 bytes contiguous), masking by the previous layer's output in
// kMaskPrev mode (masking after rounding equals rounding the masked value).
// Contains two __syncthreads: every thread of the CTA calls it.
constexpr int kOutPitch = 112;
static_assert(kTX * kTY * kOutPitch <= kTileBytes, "output staging fits an operand buffer");

__device__ __forceinline__ void conv_epilogue(const ConvArgs &a, int tile, uint32_t acc_taddr,
                                              unsigned char *stage)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float v[48];
    {
        float t0[16], t1[16], t2[16];
        const uint32_t ta = acc_taddr + (static_cast<uint32_t>(32 * warp) << 16);
        tmem_ld16(ta, t0);
        tmem_ld16(ta + 16, t1);
        tmem_ld16(ta + 32, t2);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            v[i] = t0[i];
            v[16 + i] = t1[i];
            v[32 + i] = t2[i];
        }
    }
    if (a.mode != kMaskPrev) {
#pragma unroll
        for (int c = 0; c < kC; ++c) {
            v[c] += __ldg(a.bias + c);
            if (a.mode == kBiasRelu) v[c] = fmaxf(v[c], 0.0f);
        }
    }
    const int m = 32 * warp + lane;
    uint4 *st = reinterpret_cast<uint4 *>(stage + m * kOutPitch);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        uint32_t p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(v[q * 8 + 2 * k], v[q * 8 + 2 * k + 1]);
            p[k] = *reinterpret_cast<const uint32_t *>(&b2);
        }
        st[q] = make_uint4(p[0], p[1], p[2], p[3]);
    }
    __syncthreads();
    int img, y0, x0;
    tile_origin(tile, a.tiles_x, a.tiles_y, img, y0, x0);
    for (int j = threadIdx.x; j < kTX * kTY * 6; j += blockDim.x) {
        const int r = j / (kTX * 6);
        const int rem = j - r * (kTX * 6);
        const int c = rem / 6;
        const int q = rem - c * 6;
        const int gy = y0 + r, gx = x0 + c;
        if (gy >= a.h || gx >= a.w) continue;
        uint4 u = *reinterpret_cast<const uint4 *>(stage + (c * kTY + r) * kOutPitch + q * 16);
        const long long px = (static_cast<long long>(img) * a.h + gy) * a.w + gx;
        if (a.mode == kMaskPrev) {
            const uint4 mk = __ldg(reinterpret_cast<const uint4 *>(a.aux + px * kC) + q);
            const unsigned mw[4] = {mk.x, mk.y, mk.z, mk.w};
            unsigned uw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // bf16 > 0: sign bit clear and nonzero
                if ((mw[k] & 0x8000u) || (mw[k] & 0xffffu) == 0) uw[k] &= 0xffff0000u;
                if ((mw[k] >> 31) || (mw[k] >> 16) == 0) uw[k] &= 0x0000ffffu;
            }
            u = make_uint4(uw[0], uw[1], uw[2], uw[3]);
        }
        reinterpret_cast<uint4 *>(a.y + px * kC)[q] = u;
    }
    __syncthreads();
}

// One 48 -> 48 3 x 3 convolution (padding 1) over every tile: persistent CTAs
// of 128 threads, two per SM (93 KB of shared memory and 128 TMEM columns
// each). Shared memory: weights | three operand tiles | 2 mbarriers | TMEM
// slot. Iteration t waits for tile t's operands, issues its 27 MMAs into
// accumulator t % 2, then, while they run, drains tile t - 1's accumulator
// through tile t - 1's (now free) operand buffer and refills that buffer with
// tile t + 2's input: each load has a whole iteration to land.
constexpr int kConvStages = 3;
constexpr int kConvSmem = kWeightBytes + kConvStages * kTileBytes + 64;
constexpr int kConvCtasPerSm = 2;

__global__ void __launch_bounds__(kConvThreads, kConvCtasPerSm) conv48_kernel(const ConvArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *wsm = smem;
    unsigned char *const abuf0 = smem + kWeightBytes;  // operand tile b at abuf0 + b * kTileBytes
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + kWeightBytes + kConvStages * kTileBytes);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 2);
    __shared__ int abort_flag;

    const int tid = threadIdx.x;
    if (blockIdx.x >= a.tiles) return;
    for (int i = tid; i < kWeightBytes / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(wsm)[i] = __ldg(a.wt + i);
    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        fence_mbar_init();
    }
    if ((tid >> 5) == 0) tmem_alloc(tslot, 2 * kAccCols);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    const uint32_t w_base = smem_u32(wsm);

    int img, y0, x0;
    for (int k = 0; k < 2; ++k) {  // tiles 0 and 1 of this CTA (empty groups past the end)
        const int tile = blockIdx.x + k * gridDim.x;
        if (tile < a.tiles) {
            tile_origin(tile, a.tiles_x, a.tiles_y, img, y0, x0);
            load_conv_tile(a.x, a.h, a.w, img, y0, x0, abuf0 + k * kTileBytes);
        } else {
            cp_async_commit();
        }
    }
    int it = 0, prev = -1;
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
        const int b = it % kConvStages;
        cp_async_wait<1>();
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            tc_fence_after();
            issue_conv_mmas(smem_u32(abuf0 + b * kTileBytes), w_base, tbase + (it & 1) * kAccCols);
            mma_commit(&mbar[it & 1]);
        }
        unsigned char *const freed = abuf0 + ((it + 2) % kConvStages) * kTileBytes;
        if (prev >= 0) {  // epilogue of the previous tile while these MMAs run
            const int pa = (it - 1) & 1;
            const bool ok = __syncthreads_and(mbar_wait(&mbar[pa], ((it - 1) >> 1) & 1, kWaitLimit));
            if (!ok) {
                if (tid == 0) {
                    abort_flag = 1;
                    if (a.err) atomicOr(a.err, 1u);
                }
            } else {
                tc_fence_after();
                conv_epilogue(a, prev, tbase + pa * kAccCols, freed);  // freed = tile it - 1's buffer
            }
        }
        tc_fence_before();
        const int next = tile + 2 * gridDim.x;
        if (next < a.tiles) {
            tile_origin(next, a.tiles_x, a.tiles_y, img, y0, x0);
            load_conv_tile(a.x, a.h, a.w, img, y0, x0, freed);
        } else {
            cp_async_commit();
        }
        prev = tile;
    }
    __syncthreads();
    if (!abort_flag && prev >= 0) {
        const int pa = (it - 1) & 1;
        const bool ok = __syncthreads_and(mbar_wait(&mbar[pa], ((it - 1) >> 1) & 1, kWaitLimit));
        if (!ok) {
            if (tid == 0 && a.err) atomicOr(a.err, 1u);
        } else {
            tc_fence_after();
            conv_epilogue(a, prev, tbase + pa * kAccCols, abuf0 + ((it - 1) % kConvStages) * kTileBytes);
        }
    }
    cp_async_wait_all();
    tc_fence_before();
    __syncthreads();
    if ((tid >> 5) == 0) {
        tc_fence_after();
        tmem_dealloc(tbase, 2 * kAccCols);
    }
}

// ---------------------------------------------------------------------------
// The same convolution as a warp-specialised TMA pipeline. Output tiles are 8
// pixels wide and 16 tall (MMA row m = row * 8 + column). A tile's input with
// its halo, 10 columns x 18 rows, arrives by ONE TMA load of a 5-D view of the
// NHWC activations -- (channel % 8, x, channel / 8, y, image) with byte
// strides (2, 96, 16, 96 w, 96 w h) -- whose box {8, 10, 6, 18, 1} lands as
// [row][channel / 8][column][channel % 8]: the K-major core-matrix layout with
// LBO = 160 bytes between channel groups and SBO = 960 bytes between pixel
// rows, so tap (dy, dx) starts dy * 960 + dx * 16 bytes in. The copy
// zero-fills the halo outside the image.
//
// Warps: 0 loads (lane 0), 1 issues the MMAs (lane 0), the others drain: kSets
// accumulators, each with four warps per 16 channels -- warp w reads TMEM lanes
// 32 (w % 4) .. + 31, pixel rows 4 (w % 4) .. + 3 -- which store their 4 x 8
// pixels with a TMA store of a 4-D view (channel, x, y, image) from a per-warp
// staging buffer (the store clips at the image edges). kTmaStages operand buffers
// and the accumulators are handed on by mbarriers (full / empty for each); no
// CTA-wide barrier runs inside the tile loop. What bounds it: operand fetch from
// shared memory, 101 cycles an MMA (see conv48_n144_kernel). (Four warps
// draining whole pixels of both accumulators, with the mask read after the MMAs,
// were slower than that: data gradient of 32 crops of 128 x 128 52 -> 43 us.)
constexpr int kT2X = 8, kT2Y = 16;
constexpr int kTmaStages = 4;
constexpr int kSets = 2;    // accumulators, each with its own set of draining warps
constexpr int kSplit = 3;   // 16-channel parts of an accumulator
constexpr int kSetWarps = 4 * kSplit;
constexpr int kTmaThreads = 64 + 32 * kSets * kSetWarps;  // producer, MMA issuer, the draining sets
constexpr int kStoreBytes = 32 * 16 * 2;  // one warp's 16 channels of 4 x 8 output pixels
constexpr int kTmaOffStage = kWeightBytes;
constexpr int kTmaOffStore = kTmaOffStage + kTmaStages * kTileBytes;
constexpr int kTmaOffBias = kTmaOffStore + kSets * kSetWarps * 2 * kStoreBytes;
constexpr int kTmaOffBar = kTmaOffBias + kC * 4;
constexpr int kTmaSmem = kTmaOffBar + 8 * (2 * kTmaStages + 2 * kSets) + 16;
static_assert(kTmaOffStage % 128 == 0 && kTmaOffStore % 128 == 0 && kTileBytes % 128 == 0,
              "TMA buffers 128-byte aligned");

__device__ __forceinline__ void tile_origin_8x16(int tile, int tiles_x, int tiles_y, int &img,
                                                 int &y0, int &x0)
{
    const int per = tiles_x * tiles_y;
    img = tile / per;
    const int r = tile - img * per;
    const int ty = r / tiles_x;
    y0 = ty * kT2Y;
    x0 = (r - ty * tiles_x) * kT2X;
}

// Two FP32 values to a BF16 pair (lo in the low half), optionally through ReLU.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi, bool relu)
{
    uint32_t d;
    if (relu)
        asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// All ones in each half of a BF16 pair that is positive: sign bit clear and nonzero.
__device__ __forceinline__ uint32_t bf16x2_positive(uint32_t x)
{
    const uint32_t t = ((x & 0x7fff7fffu) + 0x7fff7fffu) & ~x;  // bit 15: nonzero and not negative
    uint32_t m;  // the sign bits of bytes 1 and 3, spread
    asm("prmt.b32 %0, %1, 0, 0xbb99;" : "=r"(m) : "r"(t));
    return m;
}

__global__ void __launch_bounds__(kTmaThreads, 1)
    conv48_tma_kernel(const __grid_constant__ CUtensorMap tm_in,
                      const __grid_constant__ CUtensorMap tm_out, const ConvArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTmaOffBar);
    uint64_t *empty = full + kTmaStages;
    uint64_t *accf = empty + kTmaStages;
    uint64_t *acce = accf + kSets;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + kSets);
    float *bias_s = reinterpret_cast<float *>(smem + kTmaOffBias);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (blockIdx.x >= a.tiles) return;

    for (int i = tid; i < kWeightBytes / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(smem)[i] = __ldg(a.wt + i);
    if (tid < kC) bias_s[tid] = a.mode != kMaskPrev ? __ldg(a.bias + tid) : 0.0f;
    if (tid == 0) {
        for (int s = 0; s < kTmaStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < kSets; ++k) {
            mbar_init(&accf[k], 1);
            mbar_init(&acce[k], kSetWarps);  // one arrival per draining warp of set k
        }
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, 2 * kAccCols);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {  // producer
            int it = 0;
            for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
                const int s = it % kTmaStages;
                if (!mbar_wait(&empty[s], ((it / kTmaStages) & 1) ^ 1, kWaitLimit)) {
                    ok = false;
                    break;
                }
                int img, y0, x0;
                tile_origin_8x16(tile, a.tiles_x, a.tiles_y, img, y0, x0);
                mbar_arrive_expect_tx(&full[s], kTileBytes);
                tma_load_5d(smem + kTmaOffStage + s * kTileBytes, &tm_in, &full[s], 0, x0 - 1, 0,
                            y0 - 1, img);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issue
            const uint32_t w_base = smem_u32(smem);
            int it = 0;
            for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
                const int s = it % kTmaStages, k = it & 1;
                if (!mbar_wait(&full[s], (it / kTmaStages) & 1, kWaitLimit) ||
                    !mbar_wait(&acce[k], ((it >> 1) & 1) ^ 1, kWaitLimit)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                // 8 x 16 tiles: rows kHaloColBytes (960) apart, columns 16 bytes
                issue_tile_mmas<kHaloColBytes, 16>(smem_u32(smem + kTmaOffStage + s * kTileBytes),
                                                   w_base, tbase + k * kAccCols);
                mma_commit(&empty[s]);  // the operand buffer is free once these MMAs finish
                mma_commit(&accf[k]);
            }
        }
    } else {  // drain: set (warp - 2) / 12, TMEM lanes 32 (warp % 4) .. + 31, 16 channels
        const int q = warp & 3, set = (warp - 2) / kSetWarps;
        const int c0 = (warp - 2 - set * kSetWarps) / 4 * 16;  // the first channel
        unsigned char *const stage0 = smem + kTmaOffStore + (warp - 2) * 2 * kStoreBytes;
        const uint32_t ta = tbase + set * kAccCols + c0 + (static_cast<uint32_t>(32 * q) << 16);
        const bool relu = a.mode == kBiasRelu;
        int use = 0;  // times this set's accumulator was filled
        for (int tile = blockIdx.x + set * gridDim.x; tile < a.tiles;
             tile += kSets * gridDim.x, ++use) {
            int img, y0, x0;
            tile_origin_8x16(tile, a.tiles_x, a.tiles_y, img, y0, x0);
            // the mask's loads return while the tile's MMAs run
            uint4 mk[2] = {};
            if (a.mode == kMaskPrev) {
                const int gy = y0 + 4 * q + (lane >> 3), gx = x0 + (lane & 7);
                if (gy < a.h && gx < a.w) {
                    const uint4 *mp = reinterpret_cast<const uint4 *>(
                        a.aux + ((static_cast<long long>(img) * a.h + gy) * a.w + gx) * kC + c0);
                    mk[0] = __ldg(mp);
                    mk[1] = __ldg(mp + 1);
                }
            }
            if (!__all_sync(0xffffffffu, mbar_wait(&accf[set], use & 1, kWaitLimit))) {
                ok = false;
                break;
            }
            tc_fence_after();
            float v[16];
            tmem_ld16(ta, v);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[set]);  // the accumulator may be overwritten

            uint32_t pk[8];
            if (a.mode == kMaskPrev) {
                const unsigned mw[8] = {mk[0].x, mk[0].y, mk[0].z, mk[0].w,
                                        mk[1].x, mk[1].y, mk[1].z, mk[1].w};
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    pk[e] = pack_bf16(v[2 * e], v[2 * e + 1], false) & bf16x2_positive(mw[e]);
            } else {
                const float4 *b4 = reinterpret_cast<const float4 *>(bias_s + c0);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 b = b4[j];
                    pk[2 * j] = pack_bf16(v[4 * j] + b.x, v[4 * j + 1] + b.y, relu);
                    pk[2 * j + 1] = pack_bf16(v[4 * j + 2] + b.z, v[4 * j + 3] + b.w, relu);
                }
            }
            unsigned char *const stg = stage0 + (use & 1) * kStoreBytes;
            if (lane == 0) bulk_wait_read_1();  // this warp's store two tiles back has read it
            __syncwarp();
            uint4 *dst = reinterpret_cast<uint4 *>(stg + lane * 32);
            dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                // rows wholly below the image store nothing; the (then empty)
                // group is still committed, so wait_group.read 1 keeps pairing
                // each buffer with the store two tiles back
                if (y0 + 4 * q < a.h) tma_store_4d(&tm_out, stg, c0, x0, y0 + 4 * q, img);
                bulk_commit();
            }
        }
        if (lane == 0) bulk_wait_all();
    }
    if (!ok && a.err) atomicOr(a.err, 1u);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tbase, 2 * kAccCols);
    }
}

// ---------------------------------------------------------------------------
// Forward 48 -> 48 convolution with the three column taps in N. Here an MMA is
// M = 128 input pixels (16 rows x 8 columns, m = row * 8 + column) by
// N = 144 = (column tap dx, output channel) by K = 16 input channels:
//   D[(r, c)][dx][co] = sum over row taps dy and channels of
//                       X[r + dy][c][ci] W[co][ci][dy][dx]      (halo coords)
// 9 MMAs per tile (3 row taps x 3 channel steps), A = the input tile started
// dy rows in. The output pixel (r, j) is D[(r, j)][0] + D[(r, j + 1)][1] +
// D[(r, j + 2)][2]: TMEM lanes m, m + 1, m + 2 of the same warp, added with
// two shuffles per channel in the epilogue. Each tile yields 16 rows x 6
// columns (the input's 8 columns minus the two the taps reach past). The
// input tile, 8 columns x 18 rows, arrives by one TMA load as 128-byte swizzled
// rows of one pixel (48 channels and 16 zeros from outside the tensor): a tile row
// is one 1024-byte swizzle atom. Warp roles, mbarriers and stores as
// conv48_tma_kernel, except that there are kT3Sets accumulators (144 of 160
// TMEM columns each) and as many sets of four draining warps, each warp with all
// 48 channels: set k (warps 2 + 4k .. 5 + 4k) takes the tiles of accumulator k,
// so each tile's epilogue (nine TMEM loads, 96 shuffles per lane) has kT3Sets MMA
// tiles' time. Forward modes (bias, ReLU) only.
//
// What bounds it: operand fetch from shared memory, 55 bytes a cycle whatever
// the layout -- an MMA takes 0.56 M + 0.59 N cycles, 158 here where its
// arithmetic takes 72, and M = 128, N = 48 with nine taps takes 101 for a third of
// the products. On a 1080p plane a layer takes 110 us; with a third of the MMAs
// 82, without the stores 102, without the shuffles 106. Tiles of 16-byte chunks
// (the unswizzled core-matrix layout, six times the TMA's requests) took 115,
// 32-byte swizzled ones 110, twelve warps draining 16 channels each 125.
constexpr int kT3X = 6, kT3Y = 16;
constexpr int kIn3X = 8;
constexpr int kRow3Bytes = kIn3X * 128;               // 1024: one input row
constexpr int kTile3Bytes = (kT3Y + 2) * kRow3Bytes;  // 18432
constexpr int kN3 = 3 * kC;                          // 144
constexpr int kAcc3Cols = 160;                       // TMEM column stride of the accumulators (144 used)
constexpr int kStore3Bytes = 4 * kT3X * kC * 2;      // one warp's 4 x 6 output pixels: 2304
constexpr int kT3Stages = 4;
constexpr int kT3Sets = 3;  // accumulators, each with its own set of four draining warps
constexpr int kT3Threads = 64 + 128 * kT3Sets;  // producer, MMA issuer, the draining sets
constexpr int kTap3Elems = kN3 * 64;                  // one row tap's weights: [n][64], 48 used
constexpr int kPack3Elems = 3 * kTap3Elems;
constexpr int kT3OffStage = kPack3Elems * 2;
constexpr int kT3OffStore = kT3OffStage + kT3Stages * kTile3Bytes;
constexpr int kT3OffBias = kT3OffStore + 4 * kT3Sets * 2 * kStore3Bytes;
constexpr int kT3OffBar = kT3OffBias + kC * 4;
constexpr int kT3Smem = kT3OffBar + 8 * (2 * kT3Stages + 2 * kT3Sets) + 16 + 1024;  // to align to 1024
static_assert(kT3Sets * kAcc3Cols <= 512 && kAcc3Cols % 32 == 0, "accumulators fit TMEM");
constexpr uint32_t kIdesc3 = instr_desc_bf16(128, kN3, false, false);
static_assert(kTap3Elems * 2 % 1024 == 0 && kT3OffStage % 1024 == 0 && kTile3Bytes % 1024 == 0,
              "swizzled rows repeat every 1024 bytes");
static_assert(kT3OffStore % 128 == 0 && kStore3Bytes % 128 == 0, "TMA buffers 128-byte aligned");

__device__ __forceinline__ void tile_origin_6x16(int tile, int tiles_x, int tiles_y, int &img,
                                                 int &y0, int &x0)
{
    const int per = tiles_x * tiles_y;
    img = tile / per;
    const int r = tile - img * per;
    const int ty = r / tiles_x;
    y0 = ty * kT3Y;
    x0 = (r - ty * tiles_x) * kT3X;
}

__global__ void __launch_bounds__(kT3Threads, 1)
    conv48_n144_kernel(const __grid_constant__ CUtensorMap tm_in,
                       const __grid_constant__ CUtensorMap tm_out, const ConvArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *const smem = smem_raw + (1024 - (smem_u32(smem_raw) & 1023)) % 1024;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kT3OffBar);
    uint64_t *empty = full + kT3Stages;
    uint64_t *accf = empty + kT3Stages;
    uint64_t *acce = accf + kT3Sets;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + kT3Sets);
    float *bias_s = reinterpret_cast<float *>(smem + kT3OffBias);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (blockIdx.x >= a.tiles) return;

    for (int i = tid; i < kPack3Elems * 2 / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(smem)[i] = __ldg(a.wt + i);
    if (tid < kC) bias_s[tid] = __ldg(a.bias + tid);
    if (tid == 0) {
        for (int st = 0; st < kT3Stages; ++st) {
            mbar_init(&full[st], 1);
            mbar_init(&empty[st], 1);
        }
        for (int k = 0; k < kT3Sets; ++k) {
            mbar_init(&accf[k], 1);
            mbar_init(&acce[k], 4);  // one arrival per draining warp of set k
        }
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {  // producer
            int it = 0;
            for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
                const int st = it % kT3Stages;
                if (!mbar_wait(&empty[st], ((it / kT3Stages) & 1) ^ 1, kWaitLimit)) {
                    ok = false;
                    break;
                }
                int img, y0, x0;
                tile_origin_6x16(tile, a.tiles_x, a.tiles_y, img, y0, x0);
                mbar_arrive_expect_tx(&full[st], kTile3Bytes);
                tma_load_4d(smem + kT3OffStage + st * kTile3Bytes, &tm_in, &full[st], 0, x0 - 1,
                            y0 - 1, img);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issue: 9 MMAs, descriptors = bases + compile-time offsets
            int it = 0;
            for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
                const int st = it % kT3Stages, k = it % kT3Sets;
                if (!mbar_wait(&full[st], (it / kT3Stages) & 1, kWaitLimit) ||
                    !mbar_wait(&acce[k], ((it / kT3Sets) & 1) ^ 1, kWaitLimit)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t ad0 =
                    smem_desc_sw128(smem_u32(smem + kT3OffStage + st * kTile3Bytes), kRow3Bytes);
                const uint64_t bd0 = smem_desc_sw128(smem_u32(smem), 1024);
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
#pragma unroll
                    for (int s3 = 0; s3 < 3; ++s3) {
                        const uint64_t ad =
                            ad0 + static_cast<uint64_t>((dy * kRow3Bytes + s3 * 32) >> 4);
                        const uint64_t bd =
                            bd0 + static_cast<uint64_t>((dy * kTap3Elems * 2 + s3 * 32) >> 4);
                        mma_bf16(tbase + k * kAcc3Cols, ad, bd, kIdesc3, dy > 0 || s3 > 0);
                    }
                }
                mma_commit(&empty[st]);  // the operand buffer is free once these MMAs finish
                mma_commit(&accf[k]);
            }
        }
    } else {  // drain: set (warp - 2) / 4, TMEM lanes 32 (warp % 4) .. + 31
        const int q = warp & 3, set = (warp - 2) >> 2;
        const int rr = lane >> 3, c = lane & 7;  // pixel row 4q + rr, input column c
        unsigned char *const stage0 = smem + kT3OffStore + (warp - 2) * 2 * kStore3Bytes;
        const uint32_t lane_base = static_cast<uint32_t>(32 * q) << 16;
        const bool relu = a.mode == kBiasRelu;
        int it = set;  // this set's tiles: it = set, set + kT3Sets, ...
        for (int tile = blockIdx.x + set * gridDim.x; tile < a.tiles;
             tile += kT3Sets * gridDim.x, it += kT3Sets) {
            const int k = set;  // == it % kT3Sets
            if (!__all_sync(0xffffffffu, mbar_wait(&accf[k], (it / kT3Sets) & 1, kWaitLimit))) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t ta = tbase + k * kAcc3Cols + lane_base;
            uint32_t pk[24];
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {  // 16 output channels at a time
                float d0[16], d1[16], d2[16];
                tmem_ld16(ta + ch * 16, d0);
                tmem_ld16(ta + kC + ch * 16, d1);
                tmem_ld16(ta + 2 * kC + ch * 16, d2);
                tmem_wait_ld();
                const float4 *b4 = reinterpret_cast<const float4 *>(bias_s + ch * 16);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        v[e] = d0[i + e] + __shfl_down_sync(0xffffffffu, d1[i + e], 1) +
                               __shfl_down_sync(0xffffffffu, d2[i + e], 2);
                    const float4 b = b4[i / 4];
                    pk[ch * 8 + i / 2] = pack_bf16(v[0] + b.x, v[1] + b.y, relu);
                    pk[ch * 8 + i / 2 + 1] = pack_bf16(v[2] + b.z, v[3] + b.w, relu);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[k]);  // the accumulator may be overwritten

            int img, y0, x0;
            tile_origin_6x16(tile, a.tiles_x, a.tiles_y, img, y0, x0);
            unsigned char *const stg = stage0 + ((it / kT3Sets) & 1) * kStore3Bytes;
            if (lane == 0) bulk_wait_read_1();  // this warp's store two tiles back has read it
            __syncwarp();
            if (c < kT3X) {
                uint4 *dst = reinterpret_cast<uint4 *>(stg + (rr * kT3X + c) * kC * 2);
#pragma unroll
                for (int j = 0; j < 6; ++j)
                    dst[j] = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                // rows wholly below the image store nothing; the (then empty)
                // group is still committed, as in conv48_tma_kernel
                if (y0 + 4 * q < a.h) tma_store_4d(&tm_out, stg, 0, x0, y0 + 4 * q, img);
                bulk_commit();
            }
        }
        if (lane == 0) bulk_wait_all();
    }
    if (!ok && a.err) atomicOr(a.err, 1u);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tbase, 512);
    }
}

// ---------------------------------------------------------------------------
// Weight gradient of a 48 -> 48 layer on the tensor cores:
//   dW[co][ci][ky][kx] = sum over pixels p of G[p][co] * X[p + (ky - 1, kx - 1)][ci]
// One MMA per K-step of 16 pixels (two tile columns) and input-row shift dy:
// A = G (MN-major, M = 64 rows of which co 0..47 are real; the rest read the
// bytes that follow and are discarded), B = the halo tile of X starting dy rows
// down, read as N = 144 = (dx, ci) (MN-major: 18 channel groups 160 bytes apart
// across the three dx shifts), D[dy] = 64 x 144 FP32 in TMEM. Each CTA
// accumulates over its tiles and writes a partial dW (and the bias gradient from
// G) that reduce_partials_kernel sums.
//
// What bounds it: operand fetch from shared memory, 121 cycles an MMA (see
// conv48_n144_kernel; 158 with M = 128, as it was: 61 us where this takes 47). Under that stay: tiles read in the order of global memory,
// 16-byte chunks of whole rows of pixels, G's channel groups 144 bytes apart so
// that a row's chunks land on distinct banks; kWgStages - 1 tiles on their way;
// chunk addresses worked out once; the bias summed by six warps. One tile ahead,
// with G gathered 16 bytes at a time down its columns, addresses divided out per
// chunk, 48 threads summing the bias and dW written element by element 1728
// bytes apart, a layer of 32 crops of 128 x 128 took 124 us; now 47.
constexpr int kWgGroupBytes = kTY * 16 + 16;        // 144: one 8-channel group of a G column
constexpr int kWgColBytes = 6 * kWgGroupBytes;      // 864
constexpr int kGTileBytes = kTX * kWgColBytes;      // 13824
constexpr int kWgBuf = kGTileBytes + kTileBytes;
constexpr int kWgStages = 4;
constexpr int kWgThreads = 512;
constexpr int kWgBiasThreads = 2 * kTX * 6;         // the last six warps: (rows, column, group)
constexpr int kWgGChunks = (kTX * kTY * 6 + kWgThreads - 1) / kWgThreads;
constexpr int kWgXChunks = (kTileChunks + kWgThreads - 1) / kWgThreads;
constexpr int kWgOffRed = kWgStages * kWgBuf;       // bias sums, [rows, column][channel]
constexpr int kWgOffBar = kWgOffRed + 2 * kTX * kC * 4;
constexpr int kWgSmem = kWgOffBar + 8 * kWgStages + 16;
constexpr uint32_t kIdescWg = instr_desc_bf16(64, 3 * kC, true, true);
constexpr int kWgPartial = kWmid + kC;  // per CTA: dW as [dy][dx][ci][co], then db
static_assert(15 * kWgColBytes + 8 * kWgGroupBytes <= kWgBuf, "the discarded rows' reads stay in the buffer");
static_assert(kWgThreads >= kWgBiasThreads + 32, "the issuing warp sums no bias");

struct WgradArgs {
    const __nv_bfloat16 *x;  // layer input [n][h][w][48]
    const __nv_bfloat16 *g;  // gradient at the layer's pre-activation output [n][h][w][48]
    float *partial;          // [gridDim.x][kWgPartial]
    int n, h, w;
    int tiles_x, tiles_y, tiles;
    unsigned *err;
};

// The chunks a thread copies of every tile: where each lies in the buffer, its
// row and column, and its elements from the tile's first pixel. Worked out once
// (redone per chunk, the divisions were most of the kernel's instructions).
template <int N> struct WgradChunks {
    int at[N], rc[N], off[N];
    // rows x cols x 6 chunks; `halo` pixels before the tile in both directions
    __device__ __forceinline__ void init(int rows, int cols, int halo, int col_bytes, int group_bytes, int w)
    {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int i = threadIdx.x + k * kWgThreads;
            const int yy = i / (cols * 6), r = i - yy * (cols * 6);
            const int col = r / 6, ch = r - col * 6;
            at[k] = yy < rows ? col * col_bytes + ch * group_bytes + yy * 16 : -1;
            rc[k] = (yy - halo) << 16 | ((col - halo) & 0xffff);
            off[k] = ((yy - halo) * w + col - halo) * kC + ch * 8;
        }
    }
    // the tile whose first pixel is (y0, x0) of the h x w image at img
    __device__ __forceinline__ void load(const __nv_bfloat16 *img, int y0, int x0, int h, int w,
                                         uint32_t buf) const
    {
        const __nv_bfloat16 *const first = img + (static_cast<long long>(y0) * w + x0) * kC;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            if (at[k] < 0) continue;
            const int gy = y0 + (rc[k] >> 16), gx = x0 + static_cast<short>(rc[k]);
            const bool ok = static_cast<unsigned>(gy) < static_cast<unsigned>(h) &&
                            static_cast<unsigned>(gx) < static_cast<unsigned>(w);
            cp_async16(buf + at[k], ok ? first + off[k] : img, ok);
        }
    }
};

__global__ void __launch_bounds__(kWgThreads, 1) wgrad48_kernel(const WgradArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + kWgOffBar);  // one per buffer
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + kWgStages);
    float *red = reinterpret_cast<float *>(smem + kWgOffRed);
    __shared__ int abort_flag;

    const int tid = threadIdx.x;
    if (tid == 0) {
        abort_flag = 0;
        for (int k = 0; k < kWgStages; ++k) mbar_init(&mbar[k], 1);
        fence_mbar_init();
    }
    if ((tid >> 5) == 0) tmem_alloc(tslot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;

    WgradChunks<kWgGChunks> gc;
    WgradChunks<kWgXChunks> xc;
    gc.init(kTY, kTX, 0, kWgColBytes, kWgGroupBytes, a.w);
    xc.init(kHaloRows, kCols, 1, kHaloColBytes, kGroupBytes, a.w);
    const uint32_t buf0 = smem_u32(smem);
    auto load_tile = [&](int tile, int buf) {  // (an empty group past the end)
        if (tile < a.tiles) {
            int img, y0, x0;
            tile_origin(tile, a.tiles_x, a.tiles_y, img, y0, x0);
            const long long plane = static_cast<long long>(img) * a.h * a.w * kC;
            gc.load(a.g + plane, y0, x0, a.h, a.w, buf0 + buf * kWgBuf);
            xc.load(a.x + plane, y0, x0, a.h, a.w, buf0 + buf * kWgBuf + kGTileBytes);
        }
        cp_async_commit();
    };
    for (int k = 0; k < kWgStages - 1; ++k) load_tile(blockIdx.x + k * gridDim.x, k);
    const int bt = tid - (kWgThreads - kWgBiasThreads);  // bias thread, or negative
    float bsum[8] = {};
    int it = 0;
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, ++it) {
        const int b = it % kWgStages;
        cp_async_wait<kWgStages - 2>();  // this tile has landed
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            tc_fence_after();
            const uint32_t gb = smem_u32(smem + b * kWgBuf), xb = gb + kGTileBytes;
            // base descriptors plus compile-time offsets (as issue_tile_mmas)
            const uint64_t ad0 = smem_desc(gb, kWgColBytes, kWgGroupBytes);
            const uint64_t bd0 = smem_desc(xb, kHaloColBytes, kGroupBytes);
#pragma unroll
            for (int s = 0; s < kTX / 2; ++s) {
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
                    const uint64_t ad = ad0 + static_cast<uint64_t>((s * 2 * kWgColBytes) >> 4);
                    const uint64_t bd =
                        bd0 + static_cast<uint64_t>((dy * 16 + s * 2 * kHaloColBytes) >> 4);
                    mma_bf16(tbase + dy * 3 * kC, ad, bd, kIdescWg, it > 0 || s > 0);
                }
            }
            mma_commit(&mbar[b]);
        }
        if (bt >= 0) {  // bias gradient from the staged G tile: four rows of a column's group
            const uint4 *gs = reinterpret_cast<const uint4 *>(
                smem + b * kWgBuf + (bt >> 1) * kWgGroupBytes + (bt & 1) * 64);
#pragma unroll
            for (int yy = 0; yy < kTY / 2; ++yy) {
                const uint4 u = gs[yy];
                const unsigned wd[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    bsum[2 * k] += __uint_as_float(wd[k] << 16);
                    bsum[2 * k + 1] += __uint_as_float(wd[k] & 0xffff0000u);
                }
            }
        }
        // the previous tile's buffer is free once its MMAs completed (its bias
        // reads ended before this iteration's barrier)
        const int f = (it + kWgStages - 1) % kWgStages;
        bool free = true;
        if (it > 0 && !mbar_wait(&mbar[f], ((it - 1) / kWgStages) & 1, kWaitLimit)) {
            free = false;
            abort_flag = 1;
            if (a.err) atomicOr(a.err, 1u);
        }
        load_tile(free ? tile + (kWgStages - 1) * gridDim.x : a.tiles, f);
    }
    if (bt >= 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            red[((bt >> 1) / 6 * 2 + (bt & 1)) * kC + (bt >> 1) % 6 * 8 + k] = bsum[k];
    }
    __syncthreads();
    float *out = a.partial + static_cast<long long>(blockIdx.x) * kWgPartial;
    const bool ok = !abort_flag && it > 0 &&
                    mbar_wait(&mbar[(it - 1) % kWgStages], ((it - 1) / kWgStages) & 1, kWaitLimit);
    if (!ok && !abort_flag && it > 0 && a.err) atomicOr(a.err, 1u);
    tc_fence_after();
    const int warp = tid >> 5, lane = tid & 31;
    // an M = 64 accumulator's row co is TMEM lane co % 16 of quadrant co / 16 (rows
    // >= 48 discarded): the warps of quadrants 0..2 share the 27 column groups
    if (ok && (warp & 3) < kC / 16) {
        const int co = 16 * (warp & 3) + lane;
        const uint32_t ta = tbase + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
#pragma unroll 1
        for (int c16 = warp >> 2; c16 < 27; c16 += kWgThreads / 128) {  // 432 columns: (dy, dx, ci)
            float v[16];
            tmem_ld16(ta + c16 * 16, v);
            tmem_wait_ld();
            if (lane < 16) {
#pragma unroll
                for (int i = 0; i < 16; ++i) out[(c16 * 16 + i) * kC + co] = v[i];
            }
        }
    } else if (!ok && tid < kC) {
        for (int i = tid; i < kWmid; i += kC) out[i] = 0.0f;
    }
    if (tid < kC) {
        float sum = 0.0f;
        for (int k = 0; k < 2 * kTX; ++k) sum += red[k * kC + tid];
        out[kWmid + tid] = (ok || it == 0) ? sum : 0.0f;
    }
    cp_async_wait_all();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tbase, 512);
    }
}

// Sums of a layer's partial gradients, in double and in a fixed order
// (reproducible). `len` sums over `parts` vectors `len` floats apart, the first
// `wlen` the weights; `mid` weights come as [dy][dx][ci][co]. A block takes 32
// neighbouring sums and its eight warps each an eighth of the parts, so that
// loads are whole lines and no thread waits for a chain of 148 (296) of them:
// with Adam, 7.5 us a layer for 32 crops of 128 x 128 (12 MB of partials) where
// one thread a sum took 17, and a launch of its own for Adam 3.
constexpr int kReduceSums = 32, kReduceThreads = 256;
struct ReduceArgs {
    const float *partial;
    float *w, *b;  // results
    int parts, len, wlen;
    bool mid;
};

__global__ void __launch_bounds__(kReduceThreads) reduce_partials_kernel(const ReduceArgs a)
{
    __shared__ double part[kReduceThreads / 32][kReduceSums];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, nslices = kReduceThreads / 32;
    const int i = blockIdx.x * kReduceSums + lane;
    double s = 0.0;
    if (i < a.len) {
        const float *p = a.partial + i;
        const int from = a.parts * slice / nslices, to = a.parts * (slice + 1) / nslices;
#pragma unroll 8
        for (int q = from; q < to; ++q) s += p[static_cast<long long>(q) * a.len];
    }
    part[slice][lane] = s;
    __syncthreads();
    if (slice != 0 || i >= a.len) return;
    for (int q = 1; q < nslices; ++q) s += part[q][lane];
    float *out;
    if (i >= a.wlen) {
        out = a.b + (i - a.wlen);
    } else if (a.mid) {
        const int col = i / kC, co = i - col * kC;  // col = (dy * 3 + dx) * 48 + ci
        const int tap = col / kC, ci = col - tap * kC;
        out = a.w + (co * kC + ci) * 9 + tap;
    } else {
        out = a.w + i;
    }
    *out = static_cast<float>(s);
}

// Adam on the FP32 master parameters (bias-corrected step size precomputed). One
// launch for all layers once every gradient is there: a step that fails before it
// leaves parameters and moments as they were.
__global__ void adam_kernel(float *param, const float *grad, float *m, float *v, int count, float lr_t,
                            float beta1, float beta2, float eps)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float g = grad[i];
        const float mi = beta1 * m[i] + (1.0f - beta1) * g;
        const float vi = beta2 * v[i] + (1.0f - beta2) * g * g;
        m[i] = mi;
        v[i] = vi;
        param[i] -= lr_t * mi / (sqrtf(vi) + eps);
    }
}

// ---------------------------------------------------------------------------
// FP32-pipe layers.

// Layer 1: [noisy, sigma map] -> 48 channels, ReLU. in = plane with row pitch
// `stride` per image (images `img_stride` elements apart); sigma[img] is the
// noise level (0-1 scale) of the constant second input channel, which is zero
// outside the image like the first.
struct InArgs {
    const float *in;
    long long stride, img_stride;
    const float *sigma;
    const float *wb;  // W1 [48][2][3][3] then b1 [48] (FP32 master copy)
    __nv_bfloat16 *y;
    int n, h, w;
};

// Packed FP32 pairs (fma.rn.f32x2: each half rounded like a scalar FMA).
__device__ __forceinline__ unsigned long long f2pack(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2unpack(unsigned long long v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b,
                                                    unsigned long long c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Layers 1 and 8's pixel kernels give each thread two pixels, 32 apart, of its
// warp's 64: every weight read serves both. Results go through shared memory
// (pixels kPxPitch apart: distinct banks) so that a warp writes its 64 pixels as
// whole lines; straight from the registers, a store's lanes lie 96 bytes apart.
constexpr int kPxThreads = 128, kPxWarps = kPxThreads / 32, kPxPerWarp = 64;
constexpr int kPxPitch = 112;
constexpr int kPxPerCta = kPxWarps * kPxPerWarp;

// Chunk j (16 bytes) of a warp's staged pixels.
__device__ __forceinline__ uint4 staged_chunk(const unsigned char *stage, int j)
{
    return *reinterpret_cast<const uint4 *>(stage + j / 6 * kPxPitch + j % 6 * 16);
}

// acc += x * w. (Scalar: a packed FMA takes the FP32 pipe as long as two and its
// operand (x, x) two moves each time.)
__device__ __forceinline__ void fma4(float4 &acc, float x, const float4 w)
{
    acc.x = fmaf(x, w.x, acc.x);
    acc.y = fmaf(x, w.y, acc.y);
    acc.z = fmaf(x, w.z, acc.z);
    acc.w = fmaf(x, w.w, acc.w);
}

// Layer 1. The noise-level input is constant inside the image, so for a pixel
// whose 3 x 3 neighbourhood is inside, its part is sigma * sum_t W1[c][1][t] (one
// constant per channel); border pixels sum it over their inside taps. Weights are
// kept [tap][channel] in shared memory (128-bit broadcast reads). What bounds it: the FP32
// pipe (28 us of a 1080p plane) and latency. A 1080p plane 101 -> 80 us against one
// pixel a thread, packed FMAs and 16-byte stores from registers (84 with these
// FMAs packed); 32 crops of 128 x 128, where its 2048 units fill 888 CTAs
// unevenly, 35 -> 38.
__global__ void __launch_bounds__(kPxThreads, 6) conv_in_kernel(const InArgs a)
{
    __shared__ __align__(16) float wn[9][kC];  // W1[c][0][t] at [t][c]
    __shared__ __align__(16) float wsg[9][kC]; // W1[c][1][t] at [t][c]
    __shared__ __align__(16) float bias[kC], stot[kC];
    __shared__ __align__(16) unsigned char staging[kPxWarps][kPxPerWarp * kPxPitch];
#pragma unroll
    for (int k = 0; k < (kW1 + kPxThreads - 1) / kPxThreads; ++k) {
        const int i = threadIdx.x + k * kPxThreads;  // W1[c][cin][t]
        const int c = i / 18, r = i - c * 18;
        if (i < kW1) (r < 9 ? wn[r][c] : wsg[r - 9][c]) = a.wb[i];
    }
    for (int c = threadIdx.x; c < kC; c += blockDim.x) bias[c] = a.wb[kW1 + c];
    __syncthreads();
    for (int c = threadIdx.x; c < kC; c += blockDim.x) {
        float st = 0.0f;
        for (int t = 0; t < 9; ++t) st += wsg[t][c];
        stot[c] = st;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *const stage = staging[warp];
    // (pixels of activations that fit in memory count below 2^31)
    const unsigned plane = static_cast<unsigned>(a.h) * a.w, total = plane * a.n;
    for (unsigned base = (blockIdx.x * kPxWarps + warp) * kPxPerWarp; base < total;
         base += gridDim.x * kPxPerCta) {
        float nd[2][9], sd[2];  // noisy at each tap, 0 outside; sigma
        unsigned inside[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned p = min(base + 32 * k + lane, total - 1);
            const unsigned img = p / plane, r = p - img * plane;
            const int y = r / a.w, x = r - y * a.w;
            const float *at = a.in + img * a.img_stride + y * a.stride + x;
            sd[k] = a.sigma[img];
            inside[k] = 0;
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int yy = y + t / 3 - 1, xx = x + t % 3 - 1;
                const bool ok = yy >= 0 && yy < a.h && xx >= 0 && xx < a.w;
                nd[k][t] = ok ? __ldg(at + (t / 3 - 1) * a.stride + (t % 3 - 1)) : 0.0f;
                inside[k] |= (ok ? 1u : 0u) << t;
            }
        }
        // taps of border pixels, for both pixels and all lanes in step (one tap at a
        // time of one pixel at a time took 7 of 18 us on one 128 x 128 image)
        const unsigned edge[2] = {inside[0] == 0x1ffu ? 0u : inside[0], inside[1] == 0x1ffu ? 0u : inside[1]};
        const bool border = __any_sync(0xffffffffu, (edge[0] | edge[1]) != 0);
#pragma unroll 2
        for (int q = 0; q < 6; ++q) {
            uint32_t packed[2][4];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int c = 8 * q + 4 * hf;
                const float4 b4 = *reinterpret_cast<const float4 *>(&bias[c]);
                const float4 s4 = *reinterpret_cast<const float4 *>(&stot[c]);
                float4 acc[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    acc[k] = b4;
                    if (edge[k] == 0) fma4(acc[k], sd[k], s4);
                }
                if (border) {
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
                        const float4 w4 = *reinterpret_cast<const float4 *>(&wsg[t][c]);
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            if (edge[k] >> t & 1) fma4(acc[k], sd[k], w4);
                    }
                }
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(&wn[t][c]);
#pragma unroll
                    for (int k = 0; k < 2; ++k) fma4(acc[k], nd[k][t], w4);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    packed[k][2 * hf] = pack_bf16(acc[k].x, acc[k].y, true);
                    packed[k][2 * hf + 1] = pack_bf16(acc[k].z, acc[k].w, true);
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
                *reinterpret_cast<uint4 *>(stage + (32 * k + lane) * kPxPitch + q * 16) =
                    make_uint4(packed[k][0], packed[k][1], packed[k][2], packed[k][3]);
        }
        __syncwarp();
        uint4 *const dst = reinterpret_cast<uint4 *>(a.y + static_cast<size_t>(base) * kC);
        const int chunks = static_cast<int>(min(total - base, static_cast<unsigned>(kPxPerWarp))) * 6;
#pragma unroll
        for (int i = 0; i < kPxPerWarp * 6 / 32; ++i) {
            const int j = lane + 32 * i;
            if (j < chunks) dst[j] = staged_chunk(stage, j);
        }
        __syncwarp();
    }
}

// Layer 8: 48 -> 1 plus the residual: out = noisy + b8 + conv(X7, W8). With a
// target it also writes dOut = 2 q (out - target) / count and adds
// q (out - target)^2 to *loss, q = (kLossRefSigma / sigma[image])^2: the
// squared error scaled to a common noise level, so that low-noise images
// weigh as much in training as high-noise ones (a plain MSE is dominated by
// the largest sigma, its errors growing as sigma^2).
constexpr float kLossRefSigma = 25.0f / 255.0f;
struct OutArgs {
    const __nv_bfloat16 *x;  // X7 [n][h][w][48]
    const float *noisy;
    long long stride, img_stride;  // of noisy, out, target
    const float *wb;               // W8 [48][3][3] then b8
    float *out;
    const float *target;  // may be null (inference)
    float *dout;          // [n][h][w] (training)
    double *loss;         // (training)
    const float *sigma;   // per image noise level (training: the loss weight)
    float inv_count;
    int n, h, w;
};

// Tiles of 30 x 14 output pixels. The tile with its one-pixel halo is 32 x 16
// = 512 pixels, two per thread (rows hy and hy + 8 of one column): each is
// read and unpacked once, giving its nine per-tap partial sums
// P_t(q) = sum_c W8[c][t] X7[q][c] (channel pairs as packed FMAs, weights
// [tap][channel] in shared memory, each weight load serving both pixels);
// then out(p) = noisy(p) + b8 + sum_t P_t(p + tap offset t).
constexpr int kOutHX = 32, kOutHY = 16;
constexpr int kOutTX = kOutHX - 2, kOutTY = kOutHY - 2;
static_assert(kOutHX * kOutHY == 2 * 256, "two halo pixels per thread of a 256-thread block");

__device__ __forceinline__ void unpack_bf16x8(const uint4 u, unsigned long long (&x)[4])
{
    // channels 8q .. 8q + 7 as (even, odd) pairs
    x[0] = f2pack(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u));
    x[1] = f2pack(__uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    x[2] = f2pack(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xffff0000u));
    x[3] = f2pack(__uint_as_float(u.w << 16), __uint_as_float(u.w & 0xffff0000u));
}

__global__ void __launch_bounds__(256, 2) conv_out_kernel(const OutArgs a)
{
    __shared__ __align__(16) float wt[9][kC];  // W8[c][t] at [t][c]
    __shared__ float part[9][kOutHY * kOutHX];
    __shared__ double red[8];
    for (int i = threadIdx.x; i < 9 * kC; i += blockDim.x) {
        const int t = i / kC, c = i - t * kC;
        wt[t][c] = a.wb[c * 9 + t];
    }
    const float b8 = a.wb[kW8];
    __syncthreads();
    const int tiles_x = (a.w + kOutTX - 1) / kOutTX, tiles_y = (a.h + kOutTY - 1) / kOutTY;
    const long long ntiles = static_cast<long long>(a.n) * tiles_x * tiles_y;
    const int hx = threadIdx.x & (kOutHX - 1), hy0 = threadIdx.x / kOutHX;  // rows hy0, hy0 + 8
    double err2 = 0.0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int img = static_cast<int>(tile / (static_cast<long long>(tiles_x) * tiles_y));
        const int r = static_cast<int>(tile - static_cast<long long>(img) * tiles_x * tiles_y);
        const int ty = r / tiles_x;
        const int y0 = ty * kOutTY, x0 = (r - ty * tiles_x) * kOutTX;
        const int gx = x0 - 1 + hx;
        const uint4 *src[2];
        bool in[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int gy = y0 - 1 + hy0 + 8 * k;
            in[k] = gy >= 0 && gy < a.h && gx >= 0 && gx < a.w;
            src[k] = reinterpret_cast<const uint4 *>(
                a.x + ((static_cast<long long>(img) * a.h + (in[k] ? gy : 0)) * a.w +
                       (in[k] ? gx : 0)) * kC);
        }
        unsigned long long acc[2][9];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int t = 0; t < 9; ++t) acc[k][t] = 0ull;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            unsigned long long x[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k)
                unpack_bf16x8(in[k] ? __ldg(src[k] + q) : make_uint4(0u, 0u, 0u, 0u), x[k]);
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const float4 wa = *reinterpret_cast<const float4 *>(&wt[t][8 * q]);
                const float4 wb = *reinterpret_cast<const float4 *>(&wt[t][8 * q + 4]);
                const unsigned long long w0 = f2pack(wa.x, wa.y), w1 = f2pack(wa.z, wa.w);
                const unsigned long long w2 = f2pack(wb.x, wb.y), w3 = f2pack(wb.z, wb.w);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    acc[k][t] = ffma2(x[k][0], w0, acc[k][t]);
                    acc[k][t] = ffma2(x[k][1], w1, acc[k][t]);
                    acc[k][t] = ffma2(x[k][2], w2, acc[k][t]);
                    acc[k][t] = ffma2(x[k][3], w3, acc[k][t]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                float e, o;
                f2unpack(acc[k][t], e, o);
                part[t][(hy0 + 8 * k) * kOutHX + hx] = e + o;
            }
        __syncthreads();
        for (int i = threadIdx.x; i < kOutTX * kOutTY; i += blockDim.x) {
            const int oy = i / kOutTX, ox = i - oy * kOutTX;
            const int y = y0 + oy, x = x0 + ox;
            if (y >= a.h || x >= a.w) continue;
            float s = b8;
#pragma unroll
            for (int t = 0; t < 9; ++t) s += part[t][(oy + t / 3) * kOutHX + ox + t % 3];
            const long long o = img * a.img_stride + static_cast<long long>(y) * a.stride + x;
            const float v = a.noisy[o] + s;
            a.out[o] = v;
            if (a.target != nullptr) {
                const float e = v - a.target[o];
                const float qs = kLossRefSigma / a.sigma[img], qq = qs * qs;
                a.dout[(static_cast<long long>(img) * a.h + y) * a.w + x] =
                    2.0f * qq * e * a.inv_count;
                err2 += static_cast<double>(qq) * e * e;
            }
        }
        __syncthreads();  // before the next tile overwrites part
    }
    if (a.target == nullptr) return;
    for (int o = 16; o >= 1; o >>= 1) err2 += __shfl_xor_sync(0xffffffffu, err2, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = err2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) s += red[i];
        atomicAdd(a.loss, s);
    }
}

// Backward of layer 8 into layer 7's pre-activation gradient:
// G7[p][ci] = (X7[p][ci] > 0) * sum_t W8[ci][t] dOut[p - (t - center)].
struct OutBackArgs {
    const __nv_bfloat16 *x7;
    const float *dout;
    const float *wb;
    __nv_bfloat16 *g;
    int n, h, w;
};

// What bounds it: latency; then the lines of X7 and G7 (100 MB for 32 crops of
// 128 x 128: 15 us). Those crops 38 -> 29 us against one pixel a thread, scalar
// weight reads and strided 16-byte accesses (32 with scalar FMAs).
__global__ void __launch_bounds__(kPxThreads, 6) out_backward_kernel(const OutBackArgs a)
{
    __shared__ __align__(16) float wt[9][kC];  // W8[c][t] at [t][c]
    __shared__ __align__(16) unsigned char staging[kPxWarps][kPxPerWarp * kPxPitch];
    for (int i = threadIdx.x; i < 9 * kC; i += blockDim.x) {
        const int t = i / kC, c = i - t * kC;
        wt[t][c] = a.wb[c * 9 + t];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *const stage = staging[warp];
    const unsigned plane = static_cast<unsigned>(a.h) * a.w, total = plane * a.n;
    for (unsigned base = (blockIdx.x * kPxWarps + warp) * kPxPerWarp; base < total;
         base += gridDim.x * kPxPerCta) {
        unsigned long long d[2][9];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned p = min(base + 32 * k + lane, total - 1);
            const unsigned r = p % plane;
            const int y = r / a.w, x = r - y * a.w;
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                // out(q) uses x(q + t - 1): x(p) reaches out(p - (t - 1))
                const int yy = y - (t / 3 - 1), xx = x - (t % 3 - 1);
                const bool ok = yy >= 0 && yy < a.h && xx >= 0 && xx < a.w;
                const float v =
                    ok ? a.dout[static_cast<long long>(p) - (t / 3 - 1) * a.w - (t % 3 - 1)] : 0.0f;
                d[k][t] = f2pack(v, v);
            }
        }
#pragma unroll 2
        for (int q = 0; q < 6; ++q) {
            uint32_t packed[2][4];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                unsigned long long g0[2] = {}, g1[2] = {};
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(&wt[t][8 * q + 4 * hf]);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        g0[k] = ffma2(f2pack(w4.x, w4.y), d[k][t], g0[k]);
                        g1[k] = ffma2(f2pack(w4.z, w4.w), d[k][t], g1[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    float v0, v1, v2, v3;
                    f2unpack(g0[k], v0, v1);
                    f2unpack(g1[k], v2, v3);
                    packed[k][2 * hf] = pack_bf16(v0, v1, false);
                    packed[k][2 * hf + 1] = pack_bf16(v2, v3, false);
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
                *reinterpret_cast<uint4 *>(stage + (32 * k + lane) * kPxPitch + q * 16) =
                    make_uint4(packed[k][0], packed[k][1], packed[k][2], packed[k][3]);
        }
        __syncwarp();
        const uint4 *const xs = reinterpret_cast<const uint4 *>(a.x7 + static_cast<size_t>(base) * kC);
        uint4 *const gd = reinterpret_cast<uint4 *>(a.g + static_cast<size_t>(base) * kC);
        const int chunks = static_cast<int>(min(total - base, static_cast<unsigned>(kPxPerWarp))) * 6;
#pragma unroll
        for (int i = 0; i < kPxPerWarp * 6 / 32; ++i) {
            const int j = lane + 32 * i;
            if (j >= chunks) break;
            const uint4 u = xs[j], g = staged_chunk(stage, j);
            auto positive = [](unsigned v) {  // all ones in each half that is > 0
                return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&v),
                                   __float2bfloat162_rn(0.0f));
            };
            gd[j] = make_uint4(g.x & positive(u.x), g.y & positive(u.y), g.z & positive(u.z),
                               g.w & positive(u.w));
        }
        __syncwarp();
    }
}

// Weight and bias gradients of layers 8 and 1, FP32 products and sums:
//   dW8[ci][t] = sum_p dOut[p] X7[p + t - 1][ci], db8 = sum_p dOut[p];
//   dW1[co][cin][t] = sum_p G1[p][co] In_cin[p + t - 1], db1[co] = sum_p G1[p][co].
// Both are sums, per 8-channel group of a 48-channel image V (X7, G1), of V times
// the nine neighbours of a plane u; X7[q] meets dOut[q - (t - 1)], the neighbours
// in reverse. 30 lanes of a warp take five columns of six groups -- V's rows are
// read as 480 contiguous bytes -- and walk kEdgeRows pixels down them, the 3 x 3
// window of u sliding in registers, kEdgeAhead rows of loads at a time, products
// in packed pairs. Layer 1's two planes have blocks of their own. What bounds it:
// latency of the loads and the FP32 pipe. One pixel and 4 (8) channels a thread
// and iteration, each with its nine loads and 64-bit divisions, took 126 (layer 1)
// and 69 us (layer 8) for 32 crops of 128 x 128; this takes 52 and 26 (56 and 27
// with scalar FMAs).
constexpr int kW8Partial = kW8 + 1;
constexpr int kW1Partial = kW1 + kC;
constexpr int kEdgeThreads = 192, kEdgeRows = 16, kEdgeAhead = 4, kEdgeCols = 5;

struct EdgeSums {
    unsigned long long dw[9][4];  // per tap, channel pairs
    unsigned long long v[4];      // sums of V
    float u;                      // sum of u
};

// This warp's share (of `warps`) of the sums; u is sigma[image] everywhere inside
// the image where `constant`.
template <bool REVERSE>
__device__ __forceinline__ void edge_sums(const __nv_bfloat16 *v, const float *u, long long stride,
                                          long long img_stride, const float *sigma, bool constant, int n,
                                          int h, int w, int warp, int warps, int grp, int col, EdgeSums &e)
{
    const int ux = (w + kEdgeCols - 1) / kEdgeCols, uy = (h + kEdgeRows - 1) / kEdgeRows;
    const unsigned long long one = f2pack(1.0f, 1.0f);
    for (long long unit = warp; unit < static_cast<long long>(n) * uy * ux; unit += warps) {
        const int img = static_cast<int>(unit / (uy * ux));
        const int r0 = static_cast<int>(unit - static_cast<long long>(img) * uy * ux);
        const int y0 = r0 / ux * kEdgeRows, x = r0 % ux * kEdgeCols + col;
        if (x >= w) continue;
        const float *const ui = u + img * img_stride;
        const __nv_bfloat16 *const vi = v + (static_cast<long long>(img) * h * w + x) * kC + grp * 8;
        const float sg = constant ? sigma[img] : 0.0f;
        auto at = [&](int yy, int xx) {
            const bool ok = yy >= 0 && yy < h && xx >= 0 && xx < w;
            return !ok ? 0.0f : constant ? sg : __ldg(ui + yy * stride + xx);
        };
        unsigned long long win[3][3];  // rows y - 1 .. y + 1, columns x - 1 .. x + 1
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float f = at(y0 - 1 + j, x - 1 + i);
                win[j][i] = f2pack(f, f);
            }
        const int yend = min(y0 + kEdgeRows, h);
        for (int y = y0; y < yend; y += kEdgeAhead) {
            uint4 rows[kEdgeAhead];
            float below[kEdgeAhead][3];
#pragma unroll
            for (int r = 0; r < kEdgeAhead; ++r) {
                rows[r] = y + r < yend ? __ldg(reinterpret_cast<const uint4 *>(
                                             vi + static_cast<long long>(y + r) * w * kC))
                                       : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int i = 0; i < 3; ++i) below[r][i] = at(y + r + 1, x - 1 + i);
            }
#pragma unroll
            for (int r = 0; r < kEdgeAhead; ++r) {
                if (y + r >= yend) break;
#pragma unroll
                for (int i = 0; i < 3; ++i) win[2][i] = f2pack(below[r][i], below[r][i]);
                unsigned long long xv[4];
                unpack_bf16x8(rows[r], xv);
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const unsigned long long ut = REVERSE ? win[2 - t / 3][2 - t % 3] : win[t / 3][t % 3];
#pragma unroll
                    for (int k = 0; k < 4; ++k) e.dw[t][k] = ffma2(xv[k], ut, e.dw[t][k]);
                }
                if (REVERSE) {
                    float lo, hi;
                    f2unpack(win[1][1], lo, hi);
                    e.u += lo;
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) e.v[k] = ffma2(xv[k], one, e.v[k]);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 3; ++i) win[j][i] = win[j + 1][i];
            }
        }
    }
}

// Sum over a warp's five columns, in lanes 0..5 (lanes 30, 31 hold none; with
// shared atomics for the block's sums the kernels took 73 and 44 us).
__device__ __forceinline__ float column_sum(float v)
{
    return v + __shfl_down_sync(0xffffffffu, v, 6) + __shfl_down_sync(0xffffffffu, v, 12) +
           __shfl_down_sync(0xffffffffu, v, 18) + __shfl_down_sync(0xffffffffu, v, 24);
}

constexpr int kEdgeWarps = kEdgeThreads / 32;

__global__ void __launch_bounds__(kEdgeThreads, 2) wgrad_out_kernel(const __nv_bfloat16 *x7,
                                                                    const float *dout, int n, int h,
                                                                    int w, float *partial)
{
    __shared__ float red[kEdgeWarps][kW8Partial];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane % 6, col = lane / 6;
    EdgeSums e = {};
    if (col < kEdgeCols)
        edge_sums<true>(x7, dout, w, static_cast<long long>(h) * w, nullptr, false, n, h, w,
                        blockIdx.x * kEdgeWarps + warp, gridDim.x * kEdgeWarps, grp, col, e);
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float lo, hi;
            f2unpack(e.dw[t][k], lo, hi);
            lo = column_sum(lo);
            hi = column_sum(hi);
            if (lane < 6) {
                red[warp][(grp * 8 + 2 * k) * 9 + t] = lo;
                red[warp][(grp * 8 + 2 * k + 1) * 9 + t] = hi;
            }
        }
    const float db = column_sum(e.u);
    if (lane == 0) red[warp][kW8] = db;
    __syncthreads();
    for (int i = threadIdx.x; i < kW8Partial; i += blockDim.x) {
        float sum = 0.0f;
#pragma unroll
        for (int q = 0; q < kEdgeWarps; ++q) sum += red[q][i];
        partial[static_cast<long long>(blockIdx.x) * kW8Partial + i] = sum;
    }
}

// Even blocks take the noisy plane (and the bias), odd ones the noise-level plane.
__global__ void __launch_bounds__(kEdgeThreads, 2) wgrad_in_kernel(const InArgs a, const __nv_bfloat16 *g1,
                                                                   float *partial)
{
    __shared__ float red[kEdgeWarps][kC * 10];  // [channel][nine taps, V]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane % 6, col = lane / 6;
    const int cin = blockIdx.x & 1;
    EdgeSums e = {};
    if (col < kEdgeCols)
        edge_sums<false>(g1, a.in, a.stride, a.img_stride, a.sigma, cin == 1, a.n, a.h, a.w,
                         (blockIdx.x >> 1) * kEdgeWarps + warp, (gridDim.x >> 1) * kEdgeWarps, grp, col, e);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int t = 0; t < 10; ++t) {
            float lo, hi;
            f2unpack(t < 9 ? e.dw[t < 9 ? t : 0][k] : e.v[k], lo, hi);
            lo = column_sum(lo);
            hi = column_sum(hi);
            if (lane < 6) {
                red[warp][(grp * 8 + 2 * k) * 10 + t] = lo;
                red[warp][(grp * 8 + 2 * k + 1) * 10 + t] = hi;
            }
        }
    __syncthreads();
    float *const out = partial + static_cast<long long>(blockIdx.x) * kW1Partial;
    for (int i = threadIdx.x; i < kC * 10; i += blockDim.x) {
        const int c = i / 10, t = i - c * 10;
        float sum = 0.0f;
#pragma unroll
        for (int q = 0; q < kEdgeWarps; ++q) sum += red[q][i];
        if (t < 9) {
            out[(c * 2 + cin) * 9 + t] = sum;
            out[(c * 2 + (cin ^ 1)) * 9 + t] = 0.0f;
        } else {
            out[kW1 + c] = cin == 0 ? sum : 0.0f;
        }
    }
}

// BF16 copies of the six 48 -> 48 layers' FP32 weights [co][ci][ky][kx] in the MMA
// operand layouts: `fwd` and `bwd` (flipped, transposed: the data gradient) per tap
// as [co / 8][ci / 8][co % 8][ci % 8] (N = 48); `fwd3` for the N = 144 forward
// kernel, per row tap dy as 144 rows n = column tap * 48 + co of 64 channels ci
// (48 used), 128-byte swizzled (smem_desc_sw128).
__global__ void pack_weights_kernel(const float *params, __nv_bfloat16 *fwd, __nv_bfloat16 *bwd,
                                    __nv_bfloat16 *fwd3)
{
    const int per = 9 * kC * kC;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 6 * per; i += gridDim.x * blockDim.x) {
        const int layer = i / per;
        int r = i - layer * per;
        const float *w = params + off_w(layer + 2);
        const int tap = r / (kC * kC);
        r -= tap * kC * kC;
        // r = element of the packed tap: [n / 8][k / 8][n % 8][k % 8]
        const int ng = r / (6 * 64), kg = (r / 64) % 6, n8 = (r / 8) % 8, k8 = r % 8;
        const int n = ng * 8 + n8, k = kg * 8 + k8;
        const int ky = tap / 3, kx = tap % 3;
        fwd[i] = __float2bfloat16_rn(w[((n * kC + k) * 3 + ky) * 3 + kx]);
        const int n3 = kx * kC + n;
        fwd3[layer * kPack3Elems + ky * kTap3Elems + n3 * 64 + ((k / 8) ^ (n3 & 7)) * 8 + k8] = fwd[i];
        bwd[i] = __float2bfloat16_rn(w[((k * kC + n) * 3 + (2 - ky)) * 3 + (2 - kx)]);
    }
}

}  // namespace pilot
