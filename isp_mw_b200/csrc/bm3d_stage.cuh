// Fused BM3D stage kernel: block matching, 3-D transform, shrinkage, inverse
// transform and shared-memory aggregation for one tile of reference blocks per
// CTA, one reference block per warp at a time.
//
// Reference: BM3D_Base::Kernel (source/BM3D.cpp:80-136, 139-218),
// BM3D_Base::BlockMatching (source/BM3D.cpp:221-236),
// Block::BlockMatchingMulti (include/Block.h:578-615, 658-703),
// BM3D_Basic::CollaborativeFilter (source/BM3D.cpp:339-385),
// BM3D_Final::CollaborativeFilter (source/BM3D.cpp:411-457).
#pragma once

#include <type_traits>

#include "bm3d_device.cuh"
#include "dct.cuh"

namespace bm3d {

// Every translation unit that launches these kernels has its own copy, filled by
// the host when a context is made.
static __constant__ DctTables c_dct;

template <typename T> struct DctTab;
template <> struct DctTab<float> {
    static __device__ __forceinline__ const float *fwd() { return c_dct.fwd_f; }
    static __device__ __forceinline__ const float *inv() { return c_dct.inv_f; }
};
template <> struct DctTab<double> {
    static __device__ __forceinline__ const double *fwd() { return c_dct.fwd_d; }
    static __device__ __forceinline__ const double *inv() { return c_dct.inv_d; }
};

// Transforms along the group axis for two pencils at once. Lengths 8 and 16
// use the butterflies of dct.cuh. In FP64 every other length N has its own
// instantiation of the symmetric matrix form (dct.cuh), reading the
// constant-bank tables at compile-time offsets; FP32 runs those lengths
// through one compact loop instead (zgen, below).
template <typename T, int N>
__device__ __forceinline__ void zfwd_n(T (&a)[kGSMax], T (&b)[kGSMax])
{
    constexpr int O = (N - 1) * N * (2 * N - 1) / 6;  // start of length N: sum of m^2, m < N
    redft10_pair<T, N>(a, b, DctTab<T>::fwd() + O);
}

template <typename T, int N>
__device__ __forceinline__ void zinv_n(T (&a)[kGSMax], T (&b)[kGSMax])
{
    constexpr int O = (N - 1) * N * (2 * N - 1) / 6;
    redft01_pair<T, N>(a, b, DctTab<T>::inv() + O);
}

template <typename V>
__device__ __forceinline__ void zbfly8(V (&a)[kGSMax], bool inverse)
{
    V t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = a[i];
    if (inverse) redft01_8(t);
    else redft10_8(t);
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = t[i];
}

// Forward (REDFT10) transform of two pencils of length n <= 16.
template <typename T>
__device__ __forceinline__ void zdct_fwd2(T (&a)[kGSMax], T (&b)[kGSMax], int n)
{
    switch (n) {
    case 16: redft10_16(a); redft10_16(b); break;
    case 8: zbfly8(a, false); zbfly8(b, false); break;
    case 1: zfwd_n<T, 1>(a, b); break;
    case 2: zfwd_n<T, 2>(a, b); break;
    case 3: zfwd_n<T, 3>(a, b); break;
    case 4: zfwd_n<T, 4>(a, b); break;
    case 5: zfwd_n<T, 5>(a, b); break;
    case 6: zfwd_n<T, 6>(a, b); break;
    case 7: zfwd_n<T, 7>(a, b); break;
    case 9: zfwd_n<T, 9>(a, b); break;
    case 10: zfwd_n<T, 10>(a, b); break;
    case 11: zfwd_n<T, 11>(a, b); break;
    case 12: zfwd_n<T, 12>(a, b); break;
    case 13: zfwd_n<T, 13>(a, b); break;
    case 14: zfwd_n<T, 14>(a, b); break;
    default: zfwd_n<T, 15>(a, b); break;
    }
}

// Backward (REDFT01) transform of two pencils of length n <= 16.
template <typename T>
__device__ __forceinline__ void zdct_inv2(T (&a)[kGSMax], T (&b)[kGSMax], int n)
{
    switch (n) {
    case 16: redft01_16(a); redft01_16(b); break;
    case 8: zbfly8(a, true); zbfly8(b, true); break;
    case 1: zinv_n<T, 1>(a, b); break;
    case 2: zinv_n<T, 2>(a, b); break;
    case 3: zinv_n<T, 3>(a, b); break;
    case 4: zinv_n<T, 4>(a, b); break;
    case 5: zinv_n<T, 5>(a, b); break;
    case 6: zinv_n<T, 6>(a, b); break;
    case 7: zinv_n<T, 7>(a, b); break;
    case 9: zinv_n<T, 9>(a, b); break;
    case 10: zinv_n<T, 10>(a, b); break;
    case 11: zinv_n<T, 11>(a, b); break;
    case 12: zinv_n<T, 12>(a, b); break;
    case 13: zinv_n<T, 13>(a, b); break;
    case 14: zinv_n<T, 14>(a, b); break;
    default: zinv_n<T, 15>(a, b); break;
    }
}

// ---------------------------------------------------------------------------
// Numerator sums in shared memory. FP32 stages keep 64-bit two's-complement
// sums as two arrays of 32-bit words, the low words at p, the high words `hi`
// words after them. A 64-bit shared-memory atomic add has no native form (it
// runs as a compare-and-swap loop), so each word is updated by a native 32-bit
// atomic: the low word's atomic returns the value it replaced, which tells
// whether this addition wrapped it, and that carry goes into the high word
// with the term's own high half. Every wrap of the low word is seen by exactly
// the addition that caused it, so once all additions are done the two words
// hold the sum mod 2^64 -- the value a 64-bit atomic add gives -- whatever the
// order. Nothing reads the sums until the tile's barrier.
//
// The words lie in separate arrays because a warp's additions fall on 32
// unrelated pixels: 32 banks spread them better than the 16 that words of
// interleaved pairs leave.
template <typename T> struct AccWin;
template <> struct AccWin<float> {
    unsigned *p;
    int hi;
    __device__ __forceinline__ AccWin operator+(int i) const { return AccWin{p + i, hi}; }
    __device__ __forceinline__ void zero(int i) const
    {
        p[i] = 0;
        p[i + hi] = 0;
    }
    __device__ __forceinline__ long long get(int i) const
    {
        return static_cast<long long>(static_cast<unsigned long long>(p[i + hi]) << 32 | p[i]);
    }
    __device__ __forceinline__ void add(long long q) const
    {
        const unsigned lo = static_cast<unsigned>(q);
        const unsigned up = static_cast<unsigned>(static_cast<unsigned long long>(q) >> 32);
        const unsigned old = atomicAdd(p, lo);
        atomicAdd(p + hi, up + (old + lo < old ? 1u : 0u));
    }
};
template <> struct AccWin<double> {
    double *p;
    __device__ __forceinline__ AccWin operator+(int i) const { return AccWin{p + i}; }
    __device__ __forceinline__ void zero(int i) const { p[i] = 0.0; }
    __device__ __forceinline__ double get(int i) const { return p[i]; }
};
// n sums at p, as carved by plan_smem (FP32: n low words, then n high words).
template <typename T> __device__ __forceinline__ AccWin<T> make_acc(void *p, int n)
{
    if constexpr (sizeof(T) == 4) return AccWin<T>{static_cast<unsigned *>(p), n};
    else return AccWin<T>{static_cast<double *>(p)};
}

// ---------------------------------------------------------------------------
// One CTA's view of its staged windows.
template <typename T> struct Tile {
    int ry0, rx0, rh, rw;      // staged window origin / size in the plane
    int pitch;
    int bs;                    // block size
    bool origin_inside;        // block (0, 0) lies inside the staged window
    const T *srcw[kMaxPlanes]; // staged src windows
    const T *refw[kMaxPlanes]; // staged ref windows (refw[0] drives matching)
    const T *src0[kMaxPlanes]; // block (0, 0) of src when outside the window
    const T *ref0[kMaxPlanes];
    AccWin<T> accN[kMaxPlanes];   // numerator sums over the window
    AccWin<T> accN0[kMaxPlanes];  // and over block (0, 0) when outside the window
};

// One aggregation term: fixed point for FP32 stages, double for FP64.
__device__ __forceinline__ void acc_add(AccWin<float> w, float v, float scale)
{
    w.add(__float2ll_rn(v * scale));
}
__device__ __forceinline__ void acc_add(AccWin<double> w, double v, float) { atomicAdd(w.p, v); }

// The same for planes with non-finite pixels: a term that has no fixed-point
// value (NaN, +-Inf, or beyond the 2^62 range) marks its pixel instead, and
// the normalisation writes NaN there -- what the reference's float sums give
// once a NaN or an Inf of either sign reaches them (source/BM3D.cpp:130-135).
// Finite terms are converted exactly as acc_add does; with no mark they are
// always converted.
constexpr float kFixedLimit = 4.0e18f;
__device__ __forceinline__ void acc_add_checked(AccWin<float> w, float v, float scale,
                                                unsigned char *mark)
{
    const float x = v * scale;
    if (mark == nullptr || fabsf(x) < kFixedLimit)
        w.add(__float2ll_rn(x));
    else
        *mark = 1;
}
__device__ __forceinline__ void acc_add_checked(AccWin<double> w, double v, float, unsigned char *)
{
    atomicAdd(w.p, v);
}
__device__ __forceinline__ void acc_flush(long long *p, long long v)
{
    atomicAdd(reinterpret_cast<unsigned long long *>(p), static_cast<unsigned long long>(v));
}
__device__ __forceinline__ void acc_flush(double *p, double v) { atomicAdd(p, v); }

// A block's weight, added at the block's origin (py, px) of a plane's weight
// sums. It goes straight to global memory: one reduction per group member
// costs no more than flushing a window of them, and without the window a tile
// needs a third less shared memory and no second zeroing and flushing pass.
__device__ __forceinline__ void weight_add(long long *den, int width, int py, int px, float w,
                                           float scale)
{
    acc_flush(den + static_cast<long long>(py) * width + px, __float2ll_rn(w * scale));
}
__device__ __forceinline__ void weight_add(double *den, int width, int py, int px, double w, float)
{
    acc_flush(den + static_cast<long long>(py) * width + px, w);
}

// Address of pixel (y, x) of the block at plane position (py, px) inside a
// staged window, or inside the (0, 0) copy when the block is (0, 0) and the
// window does not contain it.
template <typename T, typename P>
__device__ __forceinline__ P *block_ptr(const Tile<T> &t, P *win, P *origin, int py, int px,
                                        int &pitch)
{
    if (py == 0 && px == 0 && !t.origin_inside) {
        pitch = t.bs;
        return origin;
    }
    pitch = t.pitch;
    return win + (py - t.ry0) * t.pitch + (px - t.rx0);
}

// The same place of the numerator sums of windows p.
template <typename T>
__device__ __forceinline__ AccWin<T> block_acc(const Tile<T> &t, int p, int py, int px, int &pitch)
{
    if (py == 0 && px == 0 && !t.origin_inside) {
        pitch = t.bs;
        return t.accN0[p];
    }
    pitch = t.pitch;
    return t.accN[p] + ((py - t.ry0) * t.pitch + (px - t.rx0));
}

// True when the block at (py, px) can be addressed: inside the staged window,
// or the (0, 0) block held in its own copy. Group members always are by
// construction; the check keeps a violated invariant from touching memory.
template <typename T>
__device__ __forceinline__ bool block_in_tile(const Tile<T> &t, int py, int px)
{
    if (py == 0 && px == 0 && !t.origin_inside) return true;
    return py >= t.ry0 && px >= t.rx0 && py + t.bs <= t.ry0 + t.rh && px + t.bs <= t.rx0 + t.rw;
}

// A warp's search list while a group is selected: the distance bits of every
// candidate at its place in the reference's list order -- the window grid in
// raster order, then the trailing (0, 0) slot. A rejected candidate (over the
// threshold, or equal to the reference block) has all bits set.
constexpr unsigned kOrdSelf = 0xffffffffu;  // list index that stands for the reference block

template <typename T> struct DistBits;
template <> struct DistBits<float> {
    using type = unsigned;
    static __device__ __forceinline__ unsigned of(float d) { return __float_as_uint(d); }
    static __device__ __forceinline__ float value(unsigned b) { return __uint_as_float(b); }
    // keys between 2^-124 and 2^127: normal, with room for the rounding slack
    static constexpr unsigned kLow = 0x01800000u, kHigh = 0x7f000000u;
    // approximate distances (ssd_row_near): two that differ by more than near_ulps
    // units in the last place are in the order of the exact keys. A unit is at least
    // 2^-24 of the value; the bounds need twice the two sums' roundings (8 x 8
    // blocks: 65 + 33, 11 x 11: 122 + 67) and 4 for keys that round together. All
    // of it holds above kTiny = 2^-100, far from the subnormal range.
    static constexpr unsigned near_ulps(int bs) { return bs <= 8 ? 256u : 512u; }
    static constexpr unsigned kTiny = 0x0d800000u;
    static __device__ __forceinline__ unsigned warp_max(unsigned v)
    {
        return __reduce_max_sync(0xffffffffu, v);
    }
    static __device__ __forceinline__ unsigned warp_min(unsigned v)
    {
        return __reduce_min_sync(0xffffffffu, v);
    }
};
template <> struct DistBits<double> {
    using type = unsigned long long;
    static __device__ __forceinline__ unsigned long long of(double d)
    {
        return static_cast<unsigned long long>(__double_as_longlong(d));
    }
    static __device__ __forceinline__ double value(unsigned long long b)
    {
        return __longlong_as_double(static_cast<long long>(b));
    }
    static constexpr unsigned long long kLow = 0x0040000000000000ull, kHigh = 0x7fe0000000000000ull;
    static constexpr unsigned long long near_ulps(int) { return 0; }
    static constexpr unsigned long long kTiny = 0;
    static __device__ __forceinline__ unsigned long long warp_max(unsigned long long v)
    {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, m);
            v = o > v ? o : v;
        }
        return v;
    }
    static __device__ __forceinline__ unsigned long long warp_min(unsigned long long v)
    {
        return ~warp_max(~v);
    }
};

template <typename T> struct Vec4;
template <> struct Vec4<float> {
    static __device__ __forceinline__ void load(const float *p, float &a, float &b, float &c,
                                                float &d)
    {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        a = v.x; b = v.y; c = v.z; d = v.w;
    }
    static __device__ __forceinline__ void store(float *p, float a, float b, float c, float d)
    {
        *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
    }
    static __device__ __forceinline__ Pair<float> load2(const float *p)
    {
        return Pair<float>{*reinterpret_cast<const unsigned long long *>(p)};
    }
    static __device__ __forceinline__ void store2(float *p, Pair<float> v)
    {
        *reinterpret_cast<unsigned long long *>(p) = v.v;
    }
    static __device__ __forceinline__ void load4(const float *p, Pair<float> &a, Pair<float> &b)
    {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
        a.v = v.x; b.v = v.y;
    }
    static __device__ __forceinline__ void store4(float *p, Pair<float> a, Pair<float> b)
    {
        *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(a.v, b.v);
    }
};
template <> struct Vec4<double> {
    static __device__ __forceinline__ void load(const double *p, double &a, double &b, double &c,
                                                double &d)
    {
        const double2 u = reinterpret_cast<const double2 *>(p)[0];
        const double2 v = reinterpret_cast<const double2 *>(p)[1];
        a = u.x; b = u.y; c = v.x; d = v.y;
    }
    static __device__ __forceinline__ void store(double *p, double a, double b, double c, double d)
    {
        reinterpret_cast<double2 *>(p)[0] = make_double2(a, b);
        reinterpret_cast<double2 *>(p)[1] = make_double2(c, d);
    }
    static __device__ __forceinline__ Pair<double> load2(const double *p)
    {
        const double2 v = *reinterpret_cast<const double2 *>(p);
        return Pair<double>{v.x, v.y};
    }
    static __device__ __forceinline__ void store2(double *p, Pair<double> v)
    {
        *reinterpret_cast<double2 *>(p) = make_double2(v.a, v.b);
    }
    static __device__ __forceinline__ void load4(const double *p, Pair<double> &a, Pair<double> &b)
    {
        a = load2(p);
        b = load2(p + 2);
    }
    static __device__ __forceinline__ void store4(double *p, Pair<double> a, Pair<double> b)
    {
        store2(p, a);
        store2(p + 2, b);
    }
};

// How many of the n (a multiple of 4) values at p, 16-byte aligned in shared
// memory, are below v0 / v1: every lane reads the same words (broadcasts), so
// a lane ranks its values against the whole set with independent compares
// where a sorting network would chain shuffles.
__device__ __forceinline__ void count_below(const unsigned *p, int n, unsigned v0, unsigned v1,
                                            int &c0, int &c1, bool two)
{
    c0 = c1 = 0;
#pragma unroll 2
    for (int j = 0; j < n; j += 4) {
        const uint4 q = *reinterpret_cast<const uint4 *>(p + j);
        c0 += (q.x < v0) + (q.y < v0) + (q.z < v0) + (q.w < v0);
        if (two) c1 += (q.x < v1) + (q.y < v1) + (q.z < v1) + (q.w < v1);
    }
}
__device__ __forceinline__ void count_below(const unsigned long long *p, int n,
                                            unsigned long long v0, unsigned long long v1, int &c0,
                                            int &c1, bool two)
{
    c0 = c1 = 0;
    for (int j = 0; j < n; j += 2) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p + j);
        c0 += (q.x < v0) + (q.y < v0);
        if (two) c1 += (q.x < v1) + (q.y < v1);
    }
}

// Unsigned division by a small number d: k / d == div_magic(k, div_number(d))
// for k * d < 2^32 (d == 1 has no 32-bit number and is passed through).
__device__ __forceinline__ unsigned div_number(int d) { return d > 1 ? 0xffffffffu / d + 1u : 0u; }
__device__ __forceinline__ int div_magic(int k, unsigned m)
{
    return m ? static_cast<int>(__umulhi(static_cast<unsigned>(k), m)) : k;
}

// One reference block's search: its window's grid, where its pixels and its
// candidates' are, and the warp's buffers.
template <typename T> struct Search {
    const T *win, *refb, *slot;  // window place (0, 0), reference block, block (0, 0)
    int pitch, slot_pitch, st;   // row pitches; grid step
    int ngrid, nc;               // grid places in all, columns
    unsigned nc_div;
    int tp, l, j0, i0;           // plane positions of the grid's first place and the block
    int group_size;
    double dist_mul;
    typename DistBits<T>::type limit;  // the matching threshold (dist_limit)
    unsigned near_low, near_high;      // StageArgs'
    typename DistBits<T>::type *dist;
    SortKey<T> *heap;
    BlockPos *list;
    T *lkeys;
};

// Where a list place's pixels are.
template <typename T>
__device__ __forceinline__ const T *list_block(const Search<T> &e, int i, int &pitch)
{
    if (i >= e.ngrid) {
        pitch = e.slot_pitch;
        return e.slot;
    }
    const int rr = div_magic(i, e.nc_div);
    pitch = e.pitch;
    return e.win + rr * e.st * e.pitch + (i - rr * e.nc) * e.st;
}

// The exact distance of a list place, in the reference's order.
template <typename T, int BS>
__device__ __forceinline__ typename DistBits<T>::type exact_dist(const Search<T> &e, int i)
{
    int cp;
    const T *cb = list_block(e, i, cp);
    T acc = T(0);
#pragma unroll 1
    for (int y = 0; y < BS; ++y) {
#pragma unroll
        for (int x = 0; x < BS; ++x) {
            const T d = sub_rn(e.refb[y * e.pitch + x], cb[y * cp + x]);
            acc = add_rn(acc, mul_rn(d, d));
        }
    }
    return DistBits<T>::of(acc);
}

// The same of two places, which may be one: they share the reference block's
// loads, and neither waits for the other's chain of sums.
template <typename T, int BS>
__device__ __forceinline__ void exact_dists(const Search<T> &e, int i, int j, typename DistBits<T>::type &di,
                                            typename DistBits<T>::type &dj)
{
    int pi, pj;
    const T *ci = list_block(e, i, pi), *cj = list_block(e, j, pj);
    T si = T(0), sj = T(0);
#pragma unroll 1
    for (int y = 0; y < BS; ++y) {
#pragma unroll
        for (int x = 0; x < BS; ++x) {
            const T r = e.refb[y * e.pitch + x];
            const T u = sub_rn(r, ci[y * pi + x]), w = sub_rn(r, cj[y * pj + x]);
            si = add_rn(si, mul_rn(u, u));
            sj = add_rn(sj, mul_rn(w, w));
        }
    }
    di = DistBits<T>::of(si);
    dj = DistBits<T>::of(sj);
}

// A candidate's entry in the search list. Distances are sums of squares:
// >= +0, or NaN, whose bits compare above any threshold. A zero distance (the
// reference block itself, or an equal block) is rejected like one over the
// threshold (include/Block.h:606): (bits - 1) wraps to the top for it.
template <typename B>
__device__ __forceinline__ B accept_dist(B bits, B limit, int &nvalid)
{
    const bool ok = bits - 1 < limit;
    nvalid += ok ? 1 : 0;
    return ok ? bits : ~B(0);
}

// The matching threshold as distance bits: d <= thSSE is bits <= limit.
template <typename T> __device__ __forceinline__ typename DistBits<T>::type dist_limit(T thSSE)
{
    return thSSE > T(0) ? DistBits<T>::of(thSSE) : typename DistBits<T>::type(0);
}

// Ordered group of a reference block from its search list, of which this lane
// accepted nvalid. Writes list / lkeys in the reference's group order and
// returns the group size.
//
// What bounds it: latency -- one warp's dependent steps. The list holds
// 32-bit distances; only the few that can be among the best get a key
// (key_from_dist is monotone, so the cut is made on distances, with three
// units in the last place of slack: fewer than that share a key with the
// cut's). Ranks come from broadcast counts (count_below), two dependent
// shared-memory passes instead of two 15-stage shuffle networks. Lanes take
// the list 32 places apart, so that candidates along an edge (one column, or
// one row) fall to different lanes and the cut stays tight (with the lanes'
// own strips the compacted set overflowed on such planes: 0.82 -> 1.09 ms).
// 1080p, sigma 25, against 64-bit keys and two sorting networks: fast basic /
// final 0.355 / 0.461 -> 0.333 / 0.438 ms, np 2.82 / 6.27 -> 2.00 / 5.86 ms
// (the smaller list also lets np's basic stage keep 16 warps).
//
// NEAR, near: the list holds approximate distances (ssd_row_near), accepted up to
// kNear above `limit`. The cut then leaves that much more room, and the
// approximate order stands when no kept distance is within kNear of the next; else
// exact_dist gives the compacted ones'. Returns -1 where the whole list has to be
// exact: a distance at the matching threshold, ties in a full group, ranges where the
// bounds do not hold -- keys that are subnormal or zero tie at distances far apart, so
// every compacted distance has to lie in near_low .. near_high, not the cut's bound alone.
template <typename T, bool NEAR, int BS>
__device__ __forceinline__ int select_once(const Search<T> &e, bool near, int lane, int nvalid,
                                           unsigned &n_fix)
{
    using K = SortKey<T>;
    using DB = DistBits<T>;
    using B = typename DB::type;
    const B none = ~B(0);
    constexpr B kNear = NEAR ? DB::near_ulps(BS) : B(0);
    const int GS = e.group_size, nkeys = e.ngrid + 1;
    const B limit = e.limit;
    const B *const dist = e.dist;
    SortKey<T> *const heap = e.heap;
    BlockPos *const list = e.list;
    T *const lkeys = e.lkeys;
    const int accepted = __reduce_add_sync(0xffffffffu, nvalid);
    const int take = min(GS - 1, accepted);
    // list[0] is the reference block itself (key 0, include/Block.h:685)
    if (lane == 0) {
        list[0] = BlockPos{e.j0, e.i0};
        lkeys[0] = T(0);
    }
    auto place = [&](unsigned idx) {
        if (idx == kOrdSelf) return BlockPos{e.j0, e.i0};
        if (static_cast<int>(idx) >= e.ngrid) return BlockPos{0, 0};
        const int rr = div_magic(static_cast<int>(idx), e.nc_div);
        return BlockPos{e.tp + rr * e.st, e.l + (static_cast<int>(idx) - rr * e.nc) * e.st};
    };
    auto put = [&](int rank, const K &m) {  // rank-th best candidate -> list[rank + 1]
        list[rank + 1] = place(m.idx());
        lkeys[rank + 1] = m.key();
    };
    auto make = [&](B bits, unsigned idx) {
        return bits == none ? K::invalid() : K::make(key_from_dist(DB::value(bits), e.dist_mul), idx);
    };
    bool tie = false;
    if (take > 0) {
        // A window of up to kHeld x 32 places (BMrange 9) is read once and
        // held in registers for both passes; larger ones are read again.
        constexpr int kHeld = 12;
        const bool one = nkeys <= kHeld * kWarp;
        const bool two = GS - 1 > kWarp / 2;
        B v[kHeld];
        auto load = [&](int first) {
#pragma unroll
            for (int k = 0; k < kHeld; ++k) {
                const int i = first + k * kWarp + lane;
                v[k] = i < nkeys ? dist[i] : none;
            }
        };
        // Cut: the (take)-th smallest of the lanes' minima bounds the take best
        // from above (those minima are take distinct candidates). Groups of
        // more than 17 blocks use the lanes' two smallest (64 candidates),
        // which keeps the compacted set within kCand.
        B lmin = none, lmin2 = none;
        for (int first = 0; first < nkeys; first += kHeld * kWarp) {
            load(first);
#pragma unroll
            for (int k = 0; k < kHeld; ++k) {
                if (two) {
                    const B up = v[k] > lmin ? v[k] : lmin;
                    lmin2 = up < lmin2 ? up : lmin2;
                }
                lmin = v[k] < lmin ? v[k] : lmin;
            }
        }
        B *kb = reinterpret_cast<B *>(heap);
        kb[lane] = lmin;
        if (two) kb[lane + kWarp] = lmin2;
        __syncwarp();
        int r0, r1;
        count_below(kb, two ? 2 * kWarp : kWarp, lmin, lmin2, r0, r1, two);
        B tb = r0 < take ? lmin : B(0);
        if (two && r1 < take && lmin2 > tb) tb = lmin2;
        tb = DB::warp_max(tb);
        // The cut leaves slack for distances that share the bound's key. With
        // fewer than take lanes holding a candidate it keeps them all.
        const B slack = 3 + (NEAR && near ? kNear : 0);
        bool sure = true;  // the slack holds (keys are normal)
        auto cut_at = [&](B bound) {
            if (bound >= none - slack) return static_cast<B>(none - 1);
            const B kt = DB::of(key_from_dist(DB::value(bound), e.dist_mul));
            sure = kt >= DB::kLow && kt <= DB::kHigh;
            return static_cast<B>(bound + slack);
        };
        auto count = [&](B top) {  // this lane's elements at or under top
            int c = 0;
            for (int first = 0; first < nkeys; first += kHeld * kWarp) {
                if (!one) load(first);
#pragma unroll
                for (int k = 0; k < kHeld; ++k) c += v[k] <= top ? 1 : 0;
            }
            return c;
        };
        B cut = cut_at(tb);
        int mine = count(cut);
        // Candidates that crowd into few lanes leave the bound too high: halve the
        // range for a lower one that still has take elements under it. (The ordered
        // search that such lists fell back to takes 31 passes over 1089 places; as
        // the last warp of a tile it held up the others.) Both ends move to elements
        // of the list, so that lists of few different distances -- computer graphics --
        // take a step or two instead of 20 to 60.
        int pos = 0, M = 0;  // this lane's end among the compacted ones, and their number
        auto scan = [&] {
            pos = mine;
#pragma unroll
            for (int o = 1; o < kWarp; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, pos, o);
                if (lane >= o) pos += u;
            }
            M = __shfl_sync(0xffffffffu, pos, kWarp - 1);
        };
        scan();
        if (M > kCand) {
            B lo = 0, hi = tb == none ? none - 1 : tb;
            while (hi - lo > (NEAR && near ? kNear : B(1))) {
                const B mid = lo + (hi - lo) / 2;
                B under = 0, over = none;  // the elements next to mid
                int c = 0;
                for (int first = 0; first < nkeys; first += kHeld * kWarp) {
                    if (!one) load(first);
#pragma unroll
                    for (int k = 0; k < kHeld; ++k) {
                        const bool low = v[k] <= mid;
                        c += low ? 1 : 0;
                        if (low && v[k] > under) under = v[k];
                        if (!low && v[k] < over) over = v[k];
                    }
                }
                if (__reduce_add_sync(0xffffffffu, c) < take) {
                    lo = DB::warp_min(over) - 1;
                    continue;
                }
                hi = DB::warp_max(under);
                cut = cut_at(hi);
                mine = count(cut);
                if (__reduce_add_sync(0xffffffffu, mine) <= kCand) break;
            }
            scan();
        }
        if (NEAR && near) {
            // (a cut that keeps all of them leaves them below the threshold)
            if (!sure || limit < DB::kTiny || (cut == none - 1 && limit > e.near_high)) return -1;
            // a distance too close to the threshold to tell matters when it can be
            // kept, or when the group takes every accepted one; either way the cut
            // is up there
            if (cut >= limit - kNear) {
                bool edge = false;
                for (int i = lane; i < nkeys; i += kWarp)
                    edge |= dist[i] - (limit - kNear) <= 2 * kNear;
                if (__any_sync(0xffffffffu, edge)) return -1;
            }
        }
        // Compact the elements at or under the cut into heap[] (any order).
        if (NEAR && near && M > kCand) return -1;
        if (sure && M <= kCand) {
            pos -= mine;
            for (int first = 0; first < nkeys; first += kHeld * kWarp) {
                if (!one) load(first);
#pragma unroll
                for (int k = 0; k < kHeld; ++k)
                    if (v[k] <= cut)
                        heap[pos++] = K::pack(v[k], static_cast<unsigned>(first + k * kWarp + lane));
            }
            __syncwarp();
            const bool more = M > kWarp;
            K v0 = lane < M ? heap[lane] : K::invalid();  // distances for now, not keys
            K v1 = lane + kWarp < M ? heap[lane + kWarp] : K::invalid();
            bool ranked = false;
            if (NEAR && near) {
                B *sorted = kb + kCand;
                __syncwarp();
                kb[lane] = v0.key_bits();
                if (more) kb[lane + kWarp] = v1.key_bits();
                __syncwarp();
                count_below(kb, (M + 3) & ~3, v0.key_bits(), v1.key_bits(), r0, r1, more);
                // distances that are equal share a rank and leave a later one
                // unwritten: the slots start at the lanes' own values' ceiling
                sorted[lane] = none;
                if (more) sorted[lane + kWarp] = none;
                __syncwarp();
                if (lane < M) sorted[r0] = v0.key_bits();
                if (lane + kWarp < M) sorted[r1] = v1.key_bits();
                __syncwarp();
                const B s0 = sorted[lane], n0 = lane + 1 < kCand ? sorted[lane + 1] : none;
                bool close = lane < take && lane + 1 < M && (s0 == none || n0 == none || n0 - s0 <= kNear);
                if (more) {
                    const B s1 = sorted[lane + kWarp];
                    const B n1 = lane + kWarp + 1 < kCand ? sorted[lane + kWarp + 1] : none;
                    close |= lane + kWarp < take && lane + kWarp + 1 < M &&
                             (s1 == none || n1 == none || n1 - s1 <= kNear);
                }
                ranked = !__any_sync(0xffffffffu, close);
                if (__any_sync(0xffffffffu, v0.key_bits() < e.near_low || v1.key_bits() < e.near_low))
                    return -1;
                if (!ranked) {
                    if (lane < M) v0 = K::pack(exact_dist<T, BS>(e, static_cast<int>(v0.idx())), v0.idx());
                    if (lane + kWarp < M) v1 = K::pack(exact_dist<T, BS>(e, static_cast<int>(v1.idx())), v1.idx());
                }
            }
            if (!ranked) {
                if (lane < M) v0 = make(v0.key_bits(), v0.idx());
                if (lane + kWarp < M) v1 = make(v1.key_bits(), v1.idx());
                __syncwarp();
                kb[lane] = v0.key_bits();
                if (more) kb[lane + kWarp] = v1.key_bits();
                __syncwarp();
                count_below(kb, (M + 3) & ~3, v0.key_bits(), v1.key_bits(), r0, r1, more);
                // the ranks are a permutation of 0 .. M - 1 unless keys are equal
                unsigned lo = 0, hi = 0;
                if (lane < M) (r0 < 32 ? lo : hi) |= 1u << (r0 & 31);
                if (lane + kWarp < M) (r1 < 32 ? lo : hi) |= 1u << (r1 & 31);
                int distinct = __popc(__reduce_or_sync(0xffffffffu, lo));
                if (more) distinct += __popc(__reduce_or_sync(0xffffffffu, hi));
                if (distinct != M) {
                    // equal keys rank by list order; a tie counts when it reaches
                    // the kept set: a kept element with an equal one after it
                    __syncwarp();
                    heap[lane] = v0;
                    heap[lane + kWarp] = v1;
                    __syncwarp();
                    bool e0 = false, e1 = false;
                    for (int j = 0; j < M; ++j) {
                        const K o = heap[j];
                        if (o.key_bits() == v0.key_bits()) {
                            if (o < v0) ++r0;
                            else if (v0 < o) e0 = true;
                        }
                        if (o.key_bits() == v1.key_bits()) {
                            if (o < v1) ++r1;
                            else if (v1 < o) e1 = true;
                        }
                    }
                    const bool t0 = lane < M && e0 && r0 < take;
                    const bool t1 = lane + kWarp < M && e1 && r1 < take;
                    tie = __any_sync(0xffffffffu, t0 || t1);
                    // (a list that the group takes whole keeps its order among equal keys)
                    if (NEAR && near && tie && accepted >= GS) return -1;
                }
            }
            if (lane < M && r0 < take) put(r0, v0);
            if (lane + kWarp < M && r1 < take) put(r1, v1);
        } else if (sure) {
            // Many candidates share the cut, so more than the group holds: in all but
            // contrived lists equal keys touch the kept set, and the exact algorithm
            // below places any keys.
            tie = true;
        } else {
            // Rare (keys outside the normal range): repeated warp minimum, whose
            // owner lane advances to the next key of its elements.
            auto next_after = [&](const K &m, bool any) {
                K nxt = K::invalid();
                for (int i = lane; i < nkeys; i += kWarp) {
                    const K u = make(dist[i], static_cast<unsigned>(i));
                    if ((any || m < u) && u < nxt) nxt = u;
                }
                return nxt;
            };
            K cur = next_after(K::invalid(), true);
            T prev_key = T(-1);
            for (int k = 0; k < take; ++k) {
                const K m = warp_min(cur);
                tie |= (m.key() == prev_key);
                prev_key = m.key();
                if (lane == 0) put(k, m);
                if (cur == m) cur = next_after(m, false);
            }
            const K m = warp_min(cur);
            tie |= (m.valid() && m.key() == prev_key);
        }
    }
    __syncwarp();
    // More matches than the group holds: the reference keeps GroupSize of them
    // with std::partial_sort (include/Block.h:690-696), whose placement of
    // equal keys is libstdc++'s heap order, not list order. Redo such groups
    // with that exact algorithm when a tie touches the kept set: lane 0 works
    // the heap, the warp finds the entries that change it (the heap's top only
    // falls, so an entry not below it once is never below it).
    if (accepted + 1 > GS && GS > 1 && tie) {
        auto less = [](const K &p, const K &q) { return p.key() < q.key(); };
        auto adjust = [&](int hole, int len, K value) {
            const int top = hole;
            int child = hole;
            while (child < (len - 1) / 2) {
                child = 2 * (child + 1);
                if (less(heap[child], heap[child - 1])) child--;
                heap[hole] = heap[child];
                hole = child;
            }
            if ((len & 1) == 0 && child == (len - 2) / 2) {
                child = 2 * (child + 1);
                heap[hole] = heap[child - 1];
                hole = child - 1;
            }
            int parent = (hole - 1) / 2;
            while (hole > top && less(heap[parent], value)) {
                heap[hole] = heap[parent];
                hole = parent;
                parent = (hole - 1) / 2;
            }
            heap[hole] = value;
        };
        // heap[] starts with the first GS entries of the reference's match
        // list: the reference block, then matches in list order.
        if (lane == 0) {
            ++n_fix;
            heap[0] = K::make(T(0), kOrdSelf);
        }
        int h = 1;
        for (int first = 0; first < nkeys; first += kWarp) {
            const int i = first + lane;
            const K u = i < nkeys ? make(dist[i], static_cast<unsigned>(i)) : K::invalid();
            unsigned todo = __ballot_sync(0xffffffffu, u.valid());
            if (h < GS) {
                const int at = h + __popc(todo & ((1u << lane) - 1u));
                const bool in = u.valid() && at < GS;
                if (in) heap[at] = u;
                const unsigned took = __ballot_sync(0xffffffffu, in);
                todo &= ~took;
                h += __popc(took);
                if (h == GS) {
                    __syncwarp();
                    if (lane == 0)
                        for (int parent = (GS - 2) / 2;; --parent) {  // __make_heap
                            adjust(parent, GS, heap[parent]);
                            if (parent == 0) break;
                        }
                }
            }
            while (todo) {  // __heap_select
                __syncwarp();
                todo &= __ballot_sync(0xffffffffu, u.valid() && less(u, heap[0]));
                if (todo == 0) break;
                const int from = __ffs(todo) - 1;
                todo &= todo - 1;
                const K w = u.shfl(from);
                if (lane == 0) adjust(0, GS, w);
            }
        }
        __syncwarp();
        if (lane == 0)
            for (int last = GS; last > 1;) {  // __sort_heap
                --last;
                const K u = heap[last];
                heap[last] = heap[0];
                adjust(0, last, u);
            }
        __syncwarp();
        if (lane < GS) {
            list[lane] = place(heap[lane].idx());
            lkeys[lane] = heap[lane].key();
        }
    }
    __syncwarp();
    return take + 1;
}

// The same, the list made exact when its approximate distances do not decide
// (one copy of the selection's code serves both: the stage kernels wait on
// their instruction cache).
template <typename T, bool NEAR, int BS>
__device__ __forceinline__ int select_group(const Search<T> &e, bool near, int lane, int nvalid,
                                            unsigned &n_fix)
{
    for (;;) {
        if (NEAR && !near) {
            __syncwarp();
            nvalid = 0;
            if constexpr (NEAR) {
                // What the approximate pass rejected is past the limit, equal to the
                // reference block or no number either way (bounds that hold above kTiny).
                const bool skip = e.limit >= DistBits<T>::kTiny;
                auto next = [&](int i) {
                    while (i <= e.ngrid && skip && e.dist[i] == ~typename DistBits<T>::type(0)) i += kWarp;
                    return i;
                };
                for (int i = next(lane); __any_sync(0xffffffffu, i <= e.ngrid);) {
                    const int j = i <= e.ngrid ? next(i + kWarp) : i;
                    if (i <= e.ngrid) {
                        typename DistBits<T>::type di, dj;
                        exact_dists<T, BS>(e, i, j <= e.ngrid ? j : i, di, dj);
                        e.dist[i] = accept_dist(di, e.limit, nvalid);
                        if (j <= e.ngrid) e.dist[j] = accept_dist(dj, e.limit, nvalid);
                        i = next(j + kWarp);
                    }
                }
            }
            __syncwarp();
        }
        const int n = select_once<T, NEAR, BS>(e, near, lane, nvalid, n_fix);
        if (n > 0) return n;
        near = false;
    }
}

// Row stride of the reference block's copy: rows of 8 or, for 11, of 12 values
// are whole 16-byte words.
__host__ __device__ constexpr int ref_row_stride(int bs) { return (bs + 3) / 4 * 4; }

// acc += (r - c)^2 over one row of BS values, even columns in the low half, odd
// ones in the high half, squares and sums fused: the ordered, unfused sum of
// ssd_row8 up to rounding, in a third fewer operations. All terms are >= 0, so
// the halves' sum is within (65 + 33) * 2^-24 of the ordered one for 8 x 8 blocks
// and (122 + 67) * 2^-24 for 11 x 11.
template <int BS>
__device__ __forceinline__ Pair<float> ssd_row_near(Pair<float> acc, const Pair<float> (&r)[ref_row_stride(BS) / 2],
                                                    const Pair<float> (&c)[(BS + 1) / 2])
{
#pragma unroll
    for (int x = 0; x < BS / 2; ++x) {
        const Pair<float> d = vsub(r[x], c[x]);
        asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(acc.v) : "l"(d.v));
    }
    if (BS & 1) {
        const float d = __fsub_rn(r[BS / 2].lo(), c[BS / 2].lo());
        acc = Pair<float>::make(__fmaf_rn(d, d, acc.lo()), acc.hi());
    }
    return acc;
}

// Which strip each lane takes in each round over a full window (KS = kStrip):
// entry [round * 32 + lane] is the strip's list place << 16 | its offset in the
// staged window, kTaskSlot for the trailing (0, 0) slot or kTaskIdle. A lane's
// loads of one row touch bank kStrip * pitch * strip + column (+ a constant of
// the instruction), so handing out the strips in raster order puts two lanes of
// most rounds on one bank: lane b takes the strips of bank b instead, and only
// what exceeds the rounds moves to lanes with room. BMrange 9 (95 strips and
// the slot, 3 rounds): 3 strips move, all into the last round, and the first two
// rounds read every row in one wavefront instead of two. Built by one warp
// while the others stage; `spill` is scratch.
constexpr unsigned kTaskSlot = 0xffffffffu, kTaskIdle = 0xfffffffeu;
__device__ __forceinline__ void build_tasks(unsigned *tab, unsigned *spill, int span, int pitch,
                                            int lane)
{
    const int nstrips = (span + kStrip - 1) / kStrip, rounds = task_rounds(span);
    const unsigned below = (1u << lane) - 1u;
    int mine = 0, moved = 0;
    for (int s = 0; s < nstrips; ++s) {
        const int first = (lane - kStrip * pitch * s) & (kWarp - 1);
        for (int c0 = 0; c0 < span; c0 += kWarp) {
            const int c = c0 + first;
            const unsigned task = static_cast<unsigned>(kStrip * s * span + c) << 16 |
                                  static_cast<unsigned>(kStrip * s * pitch + c);
            const bool over = c < span && mine >= rounds;
            if (c < span && !over) tab[mine++ * kWarp + lane] = task;
            const unsigned m = __ballot_sync(0xffffffffu, over);
            if (over) spill[moved + __popc(m & below)] = task;
            moved += __popc(m);
        }
    }
    if (lane == 0) spill[moved] = kTaskSlot;
    ++moved;
    __syncwarp();
    int next = 0;
    for (int r = 0; r < rounds; ++r) {
        const bool room = r >= mine;
        const unsigned m = __ballot_sync(0xffffffffu, room);
        const int k = next + __popc(m & below);
        if (room) tab[r * kWarp + lane] = k < moved ? spill[k] : kTaskIdle;
        next += __popc(m);
    }
}

// ---------------------------------------------------------------------------
// Block matching for reference block (j0, i0) by one warp. What bounds it: the
// FP32 pipe (an ordered, unfused distance is 192 cycles a lane and candidate)
// and, with the warps of a CTA in step, the shared-memory pipe (88 row loads
// per strip, two wavefronts each in raster order). So FP32 distances are first
// taken with fused squares and sums (128 cycles) and strips go to the lanes of
// their banks (build_tasks); either alone gains nothing, both together take the
// 1080p basic / final stage from 0.241 / 0.346 to 0.225 / 0.329 ms (4 x 8 tiles)
// and np on 1283 x 717 from 3.66 to 3.45 ms. The same for 11 x 11 blocks, against
// one candidate a lane: vn's final stage on 960 x 540 1.47 -> 1.13 ms.
// Fills list[0..n) with (y, x) in the reference's group order and returns n.
template <typename T, int KS, int BS = kBS>
__device__ int match_block(const StageArgs<T> &a, const Tile<T> &t, int j0, int i0, int lane,
                           const unsigned *tasks, typename DistBits<T>::type *dist, T *refblk, SortKey<T> *heap,
                           BlockPos *list, T *lkeys, unsigned &n_cand, unsigned &n_fix)
{
    using B = typename DistBits<T>::type;
    if (!a.match) {
        if (lane == 0) {
            list[0] = BlockPos{j0, i0};
            lkeys[0] = T(0);
        }
        __syncwarp();
        return 1;
    }
    const int st = a.bm_step, R = a.range;
    const int right = a.width - BS, bottom = a.height - BS;
    const int l = search_boundary(i0, 0, R, st), r = search_boundary(i0, right, R, st);
    const int tp = search_boundary(j0, 0, R, st), b = search_boundary(j0, bottom, R, st);
    // KS > 1 only with BMstep == 1
    const int nr = KS > 1 ? b - tp + 1 : (b - tp) / st + 1, nc = KS > 1 ? r - l + 1 : (r - l) / st + 1;
    const int ngrid = nr * nc;
    const unsigned nc_div = div_number(nc);

    // The reference block, copied where a row is two 16-byte broadcasts: a
    // strip's candidates use at most KS of its rows at a time, so a lane holds
    // KS rows in registers instead of all eight (1080p basic 0.284 -> 0.268 ms,
    // final 0.374 -> 0.368 ms: fewer registers to shuffle, not more warps -- 20
    // and 24 warps a multiprocessor, at 96 and 80 registers, are no faster).
    const T *rb = t.refw[0] + (j0 - t.ry0) * t.pitch + (i0 - t.rx0);
    constexpr int RS = ref_row_stride(BS);
    for (int k = lane; k < BS * BS; k += kWarp)
        refblk[k / BS * RS + k % BS] = rb[k / BS * t.pitch + k % BS];
    __syncwarp();

    // Candidates: column strips of KS consecutive grid rows per task, plus one
    // task for the trailing (0, 0) slot of the reference's search list.
    const int nstrips = (nr + KS - 1) / KS;
    const int ntasks = nstrips * nc;
    // FP32 lists hold approximate distances first (select_group, NEAR). With BMstep
    // over 1 a list is a quarter as long or less, and what its distances save does not
    // pay for the lists that have to be made exact: final stage of a 1080p plane with
    // BMstep 2 in ordered against approximate distances 266 / 268 us (noise), 360 / 426
    // (computer graphics), 460 / 546 (8-bit values).
    constexpr bool kNearList = sizeof(T) == 4 && KS > 1;
    const B limit = dist_limit(a.thSSE);
    const B accept = kNearList && limit < static_cast<B>(0x7f800000u) ? limit + DistBits<T>::near_ulps(BS) : limit;
    int nvalid = 0;
    constexpr int ROWS = (KS - 1) + BS;
    // a window that the plane's border clips takes its strips in raster order
    const bool full = KS == kStrip && nr == a.span && nc == a.span;
    const T *const win = t.refw[0] + (tp - t.ry0) * t.pitch + (l - t.rx0);
    for (int first = 0; first <= ntasks; first += kWarp) {
        const T *base;
        int bp = t.pitch, at, end = ngrid;  // list place of candidate 0; end of the valid ones
        bool slot;
        if (full) {
            const unsigned task = tasks[first + lane];
            if (task == kTaskIdle) break;  // the last round
            slot = task == kTaskSlot;
            base = win + (task & 0xffffu);
            at = static_cast<int>(task >> 16);
        } else {
            const int task = first + lane;
            if (task > ntasks) break;
            slot = task == ntasks;
            const int strip = div_magic(task, nc_div), cc = task - strip * nc;
            base = win + strip * KS * st * t.pitch + cc * st;
            at = strip * KS * nc + cc;
        }
        if (slot) {
            base = block_ptr(t, t.refw[0], t.ref0[0], 0, 0, bp);
            at = ngrid;
            end = ngrid + 1;
        }
        // Every strip computes all KS candidates over all ROWS window rows,
        // with no data-dependent branch; candidates past the window's last row
        // (at or past `end`) are discarded below. Their rows lie at most KS - 1 rows
        // past a staged window or the (0, 0) copy, which are always followed by
        // other parts of the CTA's shared memory.
        T d[KS];
        if constexpr (kNearList) {
            Pair<float> acc[KS], refv[KS][RS / 2];  // row y of the reference block in refv[y % KS]
#pragma unroll
            for (int q = 0; q < KS; ++q) acc[q] = Pair<float>{0};
#pragma unroll
            for (int w = 0; w < ROWS; ++w) {
                if (w < BS) {
#pragma unroll
                    for (int x = 0; x < RS / 4; ++x)
                        Vec4<float>::load4(refblk + w * RS + 4 * x, refv[w % KS][2 * x],
                                           refv[w % KS][2 * x + 1]);
                }
                Pair<float> row[(BS + 1) / 2];
#pragma unroll
                for (int x = 0; x < (BS + 1) / 2; ++x)
                    row[x] = Pair<float>::make(base[w * bp + 2 * x],
                                               2 * x + 1 < BS ? base[w * bp + 2 * x + 1] : 0.0f);
#pragma unroll
                for (int q = 0; q < KS; ++q) {
                    const int y = w - q;
                    if (y >= 0 && y < BS) acc[q] = ssd_row_near<BS>(acc[q], refv[y % KS], row);
                }
            }
#pragma unroll
            for (int q = 0; q < KS; ++q) d[q] = acc[q].lo() + acc[q].hi();
        } else {
            T refv[KS][BS];
#pragma unroll
            for (int q = 0; q < KS; ++q) d[q] = T(0);
#pragma unroll
            for (int w = 0; w < ROWS; ++w) {
                T row[BS];
                if (w < BS) {
                    T (&r)[BS] = refv[w % KS];
                    Vec4<T>::load(refblk + w * BS, r[0], r[1], r[2], r[3]);
                    Vec4<T>::load(refblk + w * BS + 4, r[4], r[5], r[6], r[7]);
                }
#pragma unroll
                for (int x = 0; x < BS; ++x) row[x] = base[w * bp + x];
#pragma unroll
                for (int q = 0; q < KS; ++q) {
                    const int y = w - q;
                    if (y >= 0 && y < BS) d[q] = ssd_row8(d[q], refv[y % KS], row);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < KS; ++q)
            if (at + q * nc < end)
                dist[at + q * nc] = accept_dist(DistBits<T>::of(d[q]), accept, nvalid);
    }
    __syncwarp();
    n_cand += static_cast<unsigned>(ngrid);  // grid minus self, plus (0, 0)

    Search<T> e;
    e.win = win;
    e.refb = rb;
    e.slot = block_ptr(t, t.refw[0], t.ref0[0], 0, 0, e.slot_pitch);
    e.pitch = t.pitch;
    e.st = st;
    e.ngrid = ngrid;
    e.nc = nc;
    e.nc_div = nc_div;
    e.tp = tp;
    e.l = l;
    e.j0 = j0;
    e.i0 = i0;
    e.group_size = a.group_size;
    e.dist_mul = a.distMul;
    e.limit = limit;
    e.near_low = a.near_low;
    e.near_high = a.near_high;
    e.dist = dist;
    e.heap = heap;
    e.list = list;
    e.lkeys = lkeys;
    // group dumps carry exact keys
    return select_group<T, kNearList, BS>(e, kNearList && a.group_key == nullptr, lane, nvalid, n_fix);
}

// ---------------------------------------------------------------------------
// A warp's group buffer G holds block z at G + z * kGroupStride, element
// (y, x) at y * 8 + x plus a 4-value gap after row 3. The gap puts the two
// lanes that share a block on different shared-memory banks, so the row,
// column and pencil accesses below are all conflict-free.
__device__ __forceinline__ int gidx(int y, int x) { return y * 8 + x + ((y >> 2) << 2); }

// Columns of the forward or inverse 2-D transform, in place in the group buffer.
template <typename T, int MAXN, bool INV>
__device__ __forceinline__ void xy_cols(T *G, int n, int lane)
{
    const int h = lane & 1;
#pragma unroll 1
    for (int z = lane >> 1; z < (MAXN > kGSMax ? n : min(n, kGSMax)); z += kGSMax) {
        T *gz = G + z * kGroupStride;
        Pair<T> c01[8], c23[8];  // columns 4h, 4h + 1 and 4h + 2, 4h + 3
#pragma unroll
        for (int y = 0; y < 8; ++y) Vec4<T>::load4(gz + gidx(y, 4 * h), c01[y], c23[y]);
        if (INV) {
            redft01_8(c01);
            redft01_8(c23);
        } else {
            redft10_8(c01);
            redft10_8(c23);
        }
#pragma unroll
        for (int y = 0; y < 8; ++y) Vec4<T>::store4(gz + gidx(y, 4 * h), c01[y], c23[y]);
    }
    __syncwarp();
}

// Forward 2-D transform (rows then columns) of the n <= MAXN blocks of a group,
// read from a staged window and left in the warp's group buffer. Lane (z, h) =
// (lane / 2, lane % 2) owns rows 4h..4h+3, then columns 4h..4h+3, of blocks z
// and (MAXN 32) z + 16.
template <typename T, int MAXN = kGSMax>
__device__ __forceinline__ void gather_xy_forward(const Tile<T> &t, const T *win, const T *origin,
                                                  const BlockPos *list, int n, int lane, T *G,
                                                  unsigned &n_bad)
{
    const int h = lane & 1;
#pragma unroll 1
    for (int z = lane >> 1; z < (MAXN > kGSMax ? n : min(n, kGSMax)); z += kGSMax) {
        T *gz = G + z * kGroupStride;
        const BlockPos p = list[z];
        const bool ok = block_in_tile(t, p.y, p.x);
        n_bad += ok ? 0 : 1;
        int pitch;
        const T *bp = block_ptr(t, win, origin, ok ? p.y : t.ry0, ok ? p.x : t.rx0, pitch);
#pragma unroll 1
        for (int r = 0; r < 4; ++r) {
            T row[8];
            const int y = 4 * h + r;
#pragma unroll
            for (int x = 0; x < 8; ++x) row[x] = ok ? bp[y * pitch + x] : T(0);
            redft10_8(row);
            Vec4<T>::store(gz + gidx(y, 0), row[0], row[1], row[2], row[3]);
            Vec4<T>::store(gz + gidx(y, 4), row[4], row[5], row[6], row[7]);
        }
    }
    __syncwarp();
    xy_cols<T, MAXN, false>(G, n, lane);
}

// Pencils along the group axis: lane owns positions p = 2 lane and 2 lane + 1,
// i.e. (y, x) = (lane / 4, 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ int pencil_off(int lane) { return gidx(lane >> 2, 2 * (lane & 3)); }

template <typename T>
__device__ __forceinline__ void load_pencils(const T *G, int n, int lane, Pair<T> (&p)[kGSMax])
{
    const int o = pencil_off(lane);
#pragma unroll
    for (int z = 0; z < kGSMax; ++z)
        p[z] = z < n ? Vec4<T>::load2(G + z * kGroupStride + o) : Pair<T>::make(T(0), T(0));
}

template <typename T>
__device__ __forceinline__ void store_pencils(T *G, int n, int lane, const Pair<T> (&p)[kGSMax])
{
    const int o = pencil_off(lane);
#pragma unroll
    for (int z = 0; z < kGSMax; ++z)
        if (z < n) Vec4<T>::store2(G + z * kGroupStride + o, p[z]);
}

// Group-axis transform of the lane's two pencils for the FP32 lengths other
// than 8 and 16: y_k = sum_j m[k][j] x_j, x read from the group buffer, j in
// order, one runtime loop for every such length (a compact body: groups of
// varied lengths would otherwise run many unrolled bodies at once).
__device__ __forceinline__ void zgen(const float *G, int n, int lane, const float *m,
                                     Pair<float> (&p)[kGSMax])
{
    const int o = pencil_off(lane);
    float a[kGSMax], b[kGSMax];
#pragma unroll
    for (int k = 0; k < kGSMax; ++k) {
        a[k] = 0.0f;
        b[k] = 0.0f;
    }
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
        const Pair<float> x = Vec4<float>::load2(G + j * kGroupStride + o);
        const float xa = x.lo(), xb = x.hi();
        const float *mj = m + 16 * j;
#pragma unroll
        for (int k = 0; k < kGSMax; ++k) {
            a[k] = fmaf(mj[k], xa, a[k]);
            b[k] = fmaf(mj[k], xb, b[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < kGSMax; ++k) p[k] = Pair<float>::make(a[k], b[k]);
}

// The compile-time lengths of FP64 on separate pencils.
template <bool INV>
__device__ __forceinline__ void zdct2(Pair<double> (&p)[kGSMax], int n)
{
    double a[kGSMax], b[kGSMax];
#pragma unroll
    for (int k = 0; k < kGSMax; ++k) {
        a[k] = p[k].a;
        b[k] = p[k].b;
    }
    if constexpr (INV) zdct_inv2(a, b, n);
    else zdct_fwd2(a, b, n);
#pragma unroll
    for (int k = 0; k < kGSMax; ++k) p[k] = Pair<double>{a[k], b[k]};
}

// Forward group-axis transform of the pencils held in the group buffer.
template <typename T>
__device__ __forceinline__ void group_fwd(T *G, int n, int lane, Pair<T> (&p)[kGSMax])
{
    if constexpr (sizeof(T) == 4) {
        if (n == 16) {
            load_pencils(G, 16, lane, p);
            redft10_16(p);
        } else if (n == 8) {
            load_pencils(G, 8, lane, p);
            zbfly8(p, false);
        } else {
            zgen(G, n, lane, c_dct.pad_fwd + pad_table_offset(n), p);
        }
    } else {
        load_pencils(G, n, lane, p);
        zdct2<false>(p, n);
    }
}

// Inverse group-axis transform; the result is left in the group buffer.
template <typename T>
__device__ __forceinline__ void group_inv(T *G, int n, int lane, Pair<T> (&p)[kGSMax])
{
    if constexpr (sizeof(T) == 4) {
        if (n == 16) {
            redft01_16(p);
            __syncwarp();
            store_pencils(G, 16, lane, p);
            return;
        }
        if (n == 8) {
            zbfly8(p, true);
        } else {
            store_pencils(G, n, lane, p);
            __syncwarp();
            zgen(G, n, lane, c_dct.pad_inv + pad_table_offset(n), p);
        }
    } else {
        zdct2<true>(p, n);
    }
    __syncwarp();
    store_pencils(G, n, lane, p);
}

// Empirical Wiener weight y^2 / (y^2 + sigma^2) (source/BM3D.cpp:440); the
// FP32 path uses the fast division (within 2 ulp), FP64 the exact one.
__device__ __forceinline__ float wiener_weight(float y2, float s2) { return __fdividef(y2, y2 + s2); }
__device__ __forceinline__ double wiener_weight(double y2, double s2) { return y2 / (y2 + s2); }

// The poison map of plane p when its inputs hold non-finite pixels, else null
// (the normal, unchecked aggregation).
template <typename T>
__device__ __forceinline__ unsigned char *poison_map(const StageArgs<T> &a, int p)
{
    if (a.nonfinite == nullptr || a.poison[p] == nullptr) return nullptr;
    return a.nonfinite[p] != 0 ? a.poison[p] : nullptr;
}

// One 8 x 8 group member whose footprint reaches block (0, 0)'s pixels, or any
// member on a plane with non-finite pixels: per pixel, the scale of its class
// (block (0, 0) or not) and, with a poison map, the check of acc_add_checked.
// gz is the member's transformed block in the group buffer; lane half h
// aggregates rows 4h .. 4h + 3 and h == 0 adds the block weight at the
// member's origin. `plane` indexes the plane's scale and poison map.
template <typename T>
__device__ __forceinline__ void aggregate_member_slow(const StageArgs<T> &a, const Tile<T> &t, int p,
                                                      int plane, BlockPos q, const T *gz, int h,
                                                      T numW, T denW, float scale)
{
    const float scale_c = fixed_scale(a.absmax[plane], a.log2_corner);
    unsigned char *const poison = poison_map(a, plane);
    int pitch;
    const AccWin<T> dn = block_acc(t, p, q.y, q.x, pitch);
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
        const int y = 4 * h + r;
        T v[8];
        Vec4<T>::load(gz + gidx(y, 0), v[0], v[1], v[2], v[3]);
        Vec4<T>::load(gz + gidx(y, 4), v[4], v[5], v[6], v[7]);
        redft01_8(v);
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const bool corner = q.y + y < kBS && q.x + x < kBS;
            unsigned char *mk =
                poison ? poison + static_cast<long long>(q.y + y) * a.width + q.x + x : nullptr;
            acc_add_checked(dn + (y * pitch + x), v[x] * numW, corner ? scale_c : scale, mk);
        }
    }
    if (h == 0) {
        const float sd = (q.y == 0 && q.x == 0) ? scale_c : scale;
        if (poison == nullptr || fabsf(static_cast<float>(denW) * sd) < kFixedLimit)
            weight_add(a.den[plane], a.width, q.y, q.x, denW, sd);
        else  // the block's weight reaches all of its pixels
            for (int i = 0; i < kBS * kBS; ++i)
                poison[static_cast<long long>(q.y + (i >> 3)) * a.width + q.x + (i & 7)] = 1;
    }
}

// Rows of the inverse 2-D transform of the n <= MAXN blocks in the group buffer,
// each aggregated as soon as it is ready: BlockGroup::AddTo / CountTo
// (include/Block.h:1240-1265, 1334-1357). The weight is the same over the block,
// so it is added once, at the block's origin; the normalisation sums origins
// over each pixel's covering blocks. Integer sums make that exactly the
// per-pixel sum.
template <typename T, int MAXN>
__device__ __forceinline__ void aggregate_group(const StageArgs<T> &a, const Tile<T> &t, int p, int pt,
                                                const BlockPos *list, int n, int lane, const T *G,
                                                T numW, T denW, float scale, bool check)
{
    const int h = lane & 1;
#pragma unroll 1
    for (int z = lane >> 1; z < (MAXN > kGSMax ? n : min(n, kGSMax)); z += kGSMax) {
        if (!block_in_tile(t, list[z].y, list[z].x)) continue;
        const BlockPos q = list[z];
        const T *gz = G + z * kGroupStride;
        if (!check && (q.y >= kBS || q.x >= kBS)) {
            int pitch;
            const AccWin<T> dn = block_acc(t, p, q.y, q.x, pitch);
#pragma unroll 1
            for (int r = 0; r < 4; ++r) {
                const int y = 4 * h + r;
                T v[8];
                Vec4<T>::load(gz + gidx(y, 0), v[0], v[1], v[2], v[3]);
                Vec4<T>::load(gz + gidx(y, 4), v[4], v[5], v[6], v[7]);
                redft01_8(v);
#pragma unroll
                for (int x = 0; x < 8; ++x) acc_add(dn + (y * pitch + x), v[x] * numW, scale);
            }
            if (h == 0) weight_add(a.den[pt], a.width, q.y, q.x, denW, scale);
        } else {
            aggregate_member_slow<T>(a, t, p, pt, q, gz, h, numW, denW, scale);
        }
    }
    __syncwarp();
}

// Collaborative filtering of one group on plane p, aggregated into the CTA's
// accumulator windows.
// `check`: the plane holds non-finite pixels (poison_map is not null), so
// every member goes through the checking aggregation.
template <typename T, bool WIENER>
__device__ void filter_group(const StageArgs<T> &a, const Tile<T> &t, int p, const BlockPos *list,
                             int n, int lane, T *G, float scale, unsigned &n_bad, int pt = -1,
                             bool check = false)
{
    // p indexes the tile's windows; pt (default p) the plane's threshold /
    // Wiener tables, which differ when planes share one set of windows
    if (pt < 0) pt = p;
    Pair<T> sp[kGSMax], rp[kGSMax];  // the lane's two pencils of src and ref
    if (WIENER) {
        gather_xy_forward(t, t.refw[p], t.ref0[p], list, n, lane, G, n_bad);
        group_fwd(G, n, lane, rp);
        __syncwarp();
    }
    gather_xy_forward(t, t.srcw[p], t.src0[p], list, n, lane, G, n_bad);
    group_fwd(G, n, lane, sp);

    T denW;
    if (!WIENER) {
        // Hard threshold: |x| <= thr -> 0, else retained (source/BM3D.cpp:361-371).
        // thr depends on how many of (x, y, z) are 0 (source/BM3D.cpp:52-67).
        // pencil lo = (lane / 4, 2 (lane % 4)), pencil hi = (lane / 4, 2 (lane % 4) + 1)
        const int fa = ((lane & 3) == 0) + (lane < 4), fb = (lane < 4);
        const T *thr = a.thr[pt][n - 1];
        int kept = 0;
#pragma unroll
        for (int z = 0; z < kGSMax; ++z) {
            if (z < n) {
                const T ta = thr[fa + (z == 0)], tb = thr[fb + (z == 0)];
                T va = sp[z].lo(), vb = sp[z].hi();
                const T aa = va < T(0) ? -va : va, ab = vb < T(0) ? -vb : vb;
                if (aa <= ta) va = T(0); else ++kept;
                if (ab <= tb) vb = T(0); else ++kept;
                sp[z] = Pair<T>::make(va, vb);
            }
        }
        const int retained = __reduce_add_sync(0xffffffffu, kept);
        denW = retained < 1 ? T(1) : T(1) / static_cast<T>(retained);
    } else {
        // Empirical Wiener shrinkage guided by the basic estimate
        // (source/BM3D.cpp:435-443).
        const T s2 = a.wss[pt][n - 1];
        T l2 = T(0);
#pragma unroll
        for (int z = 0; z < kGSMax; ++z) {
            if (z < n) {
                const T ra = rp[z].lo(), rb = rp[z].hi();
                const T ya2 = ra * ra, yb2 = rb * rb;
                const T wa = wiener_weight(ya2, s2), wb = wiener_weight(yb2, s2);
                sp[z] = vmul(sp[z], Pair<T>::make(wa, wb));
                l2 += wa * wa + wb * wb;
            }
        }
        l2 = warp_sum(l2);
        denW = l2 <= T(0) ? T(1) : T(1) / l2;
    }
    const T numW = static_cast<T>(static_cast<double>(denW) / a.finalAMP[n - 1]);

    group_inv(G, n, lane, sp);
    __syncwarp();
    xy_cols<T, kGSMax, true>(G, n, lane);

    aggregate_group<T, kGSMax>(a, t, p, pt, list, n, lane, G, numW, denW, scale, check);
}

// ---------------------------------------------------------------------------
// CTA-level pieces shared by the register-resident and the generic kernels.

// The CTA's tile of reference positions and its staged window: the union of
// the search windows of the tile's blocks (or the blocks themselves when no
// matching happens).
template <typename T>
__device__ __forceinline__ void tile_window(const StageArgs<T> &a, int tile, int bs, Tile<T> &t,
                                            int &kx0, int &kx1, int &ky0, int &ky1)
{
    const int tx = tile % a.tiles_x, ty = tile / a.tiles_x;
    kx0 = tx * a.tile_x;
    ky0 = ty * a.tile_y;
    kx1 = min(kx0 + a.tile_x, a.nx);
    ky1 = min(ky0 + a.tile_y, a.ny);
    const int right = a.width - bs, bottom = a.height - bs;
    int y0 = 1 << 30, y1 = -1, x0 = 1 << 30, x1 = -1;
    if (a.match) {
        for (int k = ky0; k < ky1; ++k) {
            const int j = ref_pos(k, a.step, bottom);
            y0 = min(y0, search_boundary(j, 0, a.range, a.bm_step));
            y1 = max(y1, search_boundary(j, bottom, a.range, a.bm_step));
        }
        for (int k = kx0; k < kx1; ++k) {
            const int i = ref_pos(k, a.step, right);
            x0 = min(x0, search_boundary(i, 0, a.range, a.bm_step));
            x1 = max(x1, search_boundary(i, right, a.range, a.bm_step));
        }
    } else {
        y0 = ref_pos(ky0, a.step, bottom);
        y1 = ref_pos(ky1 - 1, a.step, bottom);
        x0 = ref_pos(kx0, a.step, right);
        x1 = ref_pos(kx1 - 1, a.step, right);
    }
    t.ry0 = y0;
    t.rx0 = x0;
    t.rh = y1 + bs - y0;
    t.rw = x1 + bs - x0;
    t.pitch = a.region_pitch;
    t.bs = bs;
    t.origin_inside = (y0 == 0 && x0 == 0);
}

// Carve the CTA's shared memory into staged windows, accumulators and the
// (0, 0) copies, following plan_smem.
template <typename T, bool WIENER, int NPL>
__device__ __forceinline__ void carve_tile(const StageArgs<T> &a, const SmemPlan &sp,
                                           unsigned char *smem, Tile<T> &t)
{
    const int bsq = t.bs * t.bs;
    int s = 0;
    T *origin = reinterpret_cast<T *>(smem + sp.off_origin);
    for (int p = 0; p < NPL; ++p) {
        t.srcw[p] = reinterpret_cast<const T *>(smem + sp.region_bytes * s);
        t.src0[p] = origin + bsq * s;
        ++s;
    }
    for (int p = 0; p < NPL; ++p) {
        const bool has_ref = WIENER || p == 0;
        if (!has_ref || (a.ref_alias_src & (1 << p))) {
            t.refw[p] = t.srcw[p];
            t.ref0[p] = t.src0[p];
        } else {
            t.refw[p] = reinterpret_cast<const T *>(smem + sp.region_bytes * s);
            t.ref0[p] = origin + bsq * s;
            ++s;
        }
    }
    for (int p = 0; p < NPL; ++p) {
        t.accN[p] = make_acc<T>(smem + sp.off_acc + sp.acc_bytes * p,
                                static_cast<int>(sp.acc_bytes / sizeof(typename AccOf<T>::type)));
        t.accN0[p] = make_acc<T>(smem + sp.off_origin_acc + sizeof(typename AccOf<T>::type) * bsq * p, bsq);
    }
}

// One element global -> shared without a register round trip (cp.async;
// element-sized, so no alignment beyond the element's own). Completed by
// cp_async_wait_all before the CTA barrier that publishes the windows.
template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src)
{
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(sizeof(T))
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Load the staged windows (and block (0, 0) when outside) and zero the
// accumulators. Ends with __syncthreads().
template <typename T, bool WIENER, int NPL>
__device__ __forceinline__ void stage_tile(const StageArgs<T> &a, const Tile<T> &t)
{
    const int tid = threadIdx.x;
    const int npx = t.rh * t.rw;
    const int bs = t.bs, bsq = bs * bs;
    for (int p = 0; p < NPL; ++p) {
        const bool need_src = !a.bm_only && (a.active & (1 << p));
        const bool need_ref = (p == 0) || (WIENER && need_src);
        const bool ref_sep = need_ref && t.refw[p] != t.srcw[p];
        for (int i = tid; i < npx; i += blockDim.x) {
            const int y = i / t.rw, x = i - y * t.rw;
            const long long g = static_cast<long long>(t.ry0 + y) * a.stride + (t.rx0 + x);
            const int s = y * t.pitch + x;
            if (need_src || (p == 0 && !ref_sep)) cp_async_elem(const_cast<T *>(t.srcw[p]) + s, a.src[p] + g);
            if (ref_sep) cp_async_elem(const_cast<T *>(t.refw[p]) + s, a.ref[p] + g);
            if (need_src) t.accN[p].zero(s);
        }
        if (!t.origin_inside && (need_src || p == 0)) {
            for (int i = tid; i < bsq; i += blockDim.x) {
                const int y = i / bs, x = i - y * bs;
                const long long g = static_cast<long long>(y) * a.stride + x;
                const_cast<T *>(t.src0[p])[i] = __ldg(a.src[p] + g);
                if (ref_sep) const_cast<T *>(t.ref0[p])[i] = __ldg(a.ref[p] + g);
                t.accN0[p].zero(i);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
}

// Flush the accumulator windows into the plane-wide numerator sums.
template <typename T, int NPL>
__device__ __forceinline__ void flush_tile(const StageArgs<T> &a, const Tile<T> &t)
{
    const int tid = threadIdx.x;
    const int npx = t.rh * t.rw;
    const int bs = t.bs, bsq = bs * bs;
    for (int p = 0; p < NPL; ++p) {
        if (!(a.active & (1 << p))) continue;
        for (int i = tid; i < npx; i += blockDim.x) {
            const int y = i / t.rw, x = i - y * t.rw;
            const int s = y * t.pitch + x;
            const auto nv = t.accN[p].get(s);
            const long long g = static_cast<long long>(t.ry0 + y) * a.width + (t.rx0 + x);
            if (nv != 0) acc_flush(a.num[p] + g, nv);
        }
        if (!t.origin_inside) {
            for (int i = tid; i < bsq; i += blockDim.x) {
                const auto nv = t.accN0[p].get(i);
                const int y = i / bs, x = i - y * bs;
                const long long g = static_cast<long long>(y) * a.width + x;
                if (nv != 0) acc_flush(a.num[p] + g, nv);
            }
        }
    }
}

template <typename T>
__device__ __forceinline__ void dump_group(const StageArgs<T> &a, int ky, int kx, int n, int lane,
                                           const BlockPos *list, const T *lkeys)
{
    if (a.group_count == nullptr) return;
    const long long ridx = static_cast<long long>(ky) * a.nx + kx;
    if (lane == 0) a.group_count[ridx] = n;
    for (int k = lane; k < n; k += kWarp) {
        a.group_pos[(ridx * kGSTab + k) * 2 + 0] = list[k].y;
        a.group_pos[(ridx * kGSTab + k) * 2 + 1] = list[k].x;
        if (a.group_key != nullptr) a.group_key[ridx * kGSTab + k] = lkeys[k];
    }
    __syncwarp();  // the keys' bytes become the group buffer
}

// A CTA whose launch gave it less shared memory than its layout needs does
// no work and counts itself in the invariant counter (host-mode calls then
// fail with an internal error) instead of touching memory past its share.
template <typename T>
__device__ __forceinline__ void smem_shortfall(const StageArgs<T> &a)
{
    if (a.bad != nullptr && threadIdx.x == 0) atomicAdd(a.bad, 1ull << 32);
}

template <typename T>
__device__ __forceinline__ void flush_stats(const StageArgs<T> &a, int lane, unsigned n_sum,
                                            unsigned n_sq, unsigned n_cand, unsigned n_fix,
                                            unsigned n_bad)
{
    using U = unsigned long long;
    if (a.stats != nullptr && lane == 0) {
        atomicAdd(a.stats + 0, static_cast<U>(n_sum));
        atomicAdd(a.stats + 1, static_cast<U>(n_sq));
        atomicAdd(a.stats + 2, static_cast<U>(n_cand));
        atomicAdd(a.stats + 3, static_cast<U>(n_fix));
    }
    if (a.bad != nullptr && n_bad) atomicAdd(a.bad, static_cast<U>(n_bad));
}

// ---------------------------------------------------------------------------
// Register-resident stage: BlockSize 8, GroupSize <= 16. One tile per call.
template <typename T, bool WIENER, int NPL, int KS>
__device__ __forceinline__ void stage_tile_body(const StageArgs<T> &a, int tile, unsigned char *smem,
                                                unsigned avail)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int right = a.width - kBS, bottom = a.height - kBS;

    Tile<T> t;
    int kx0, kx1, ky0, ky1;
    tile_window(a, tile, kBS, t, kx0, kx1, ky0, ky1);
    const SmemPlan sp = plan_smem<T>(NPL, WIENER, a.ref_alias_src, a.region_h, a.region_pitch,
                                     a.span, nwarps);
    if (sp.total > avail) {  // launched with less shared memory than the layout needs
        smem_shortfall(a);
        return;
    }
    carve_tile<T, WIENER, NPL>(a, sp, smem, t);
    unsigned *tasks = reinterpret_cast<unsigned *>(smem + sp.off_tasks);
    unsigned char *wbase = smem + sp.off_warps + sp.warp_bytes * warp;  // per-warp scratch
    if (KS == kStrip && warp == 0)
        build_tasks(tasks, reinterpret_cast<unsigned *>(wbase), a.span, t.pitch, lane);
    stage_tile<T, WIENER, NPL>(a, t);

    T *G = reinterpret_cast<T *>(wbase);
    auto *dist = reinterpret_cast<typename DistBits<T>::type *>(wbase);
    T *refblk = reinterpret_cast<T *>(wbase + sp.off_ref);
    SortKey<T> *heap = reinterpret_cast<SortKey<T> *>(wbase + sp.off_heap);
    T *lkeys = reinterpret_cast<T *>(wbase + sp.off_keys);
    BlockPos *list = reinterpret_cast<BlockPos *>(wbase + sp.off_list);

    // per-tile counters (small: 32 bits suffice), flushed once per tile
    unsigned n_sum = 0, n_sq = 0, n_cand = 0, n_fix = 0, n_bad = 0;
    float scale[NPL];
    bool check[NPL];
#pragma unroll
    for (int p = 0; p < NPL; ++p) {
        scale[p] = fixed_scale(a.absmax[p], a.log2_bound);
        check[p] = poison_map(a, p) != nullptr;
    }
    const int tw = kx1 - kx0, nrefs = tw * (ky1 - ky0);
    for (int r = warp; r < nrefs; r += nwarps) {
        const int ky = ky0 + r / tw, kx = kx0 + r % tw;
        const int j0 = ref_pos(ky, a.step, bottom), i0 = ref_pos(kx, a.step, right);
        const int n = match_block<T, KS>(a, t, j0, i0, lane, tasks, dist, refblk, heap, list, lkeys, n_cand,
                                       n_fix);
        n_sum += n;
        n_sq += static_cast<unsigned>(n * n);
        dump_group(a, ky, kx, n, lane, list, lkeys);
        if (!a.bm_only) {
#pragma unroll
            for (int p = 0; p < NPL; ++p)
                if (a.active & (1 << p))
                    filter_group<T, WIENER>(a, t, p, list, n, lane, G, scale[p], n_bad, -1,
                                            check[p]);
        }
        __syncwarp();
    }
    flush_stats(a, lane, n_sum, n_sq, n_cand, n_fix, n_bad);
    if (a.bm_only) return;
    __syncthreads();
    flush_tile<T, NPL>(a, t);
}

// One plane c of a three-plane tile into the single-plane windows: src[c],
// ref[c] where a stage reads it (matching on plane 0; Wiener on every plane),
// zeroed sums. Ends with __syncthreads().
template <typename T, bool WIENER>
__device__ __forceinline__ void stage_plane(const StageArgs<T> &a, const Tile<T> &t, int c)
{
    const int tid = threadIdx.x;
    const int npx = t.rh * t.rw;
    const int bs = t.bs, bsq = bs * bs;
    const bool ref_sep = t.refw[0] != t.srcw[0];
    const bool need_ref = ref_sep && (WIENER || c == 0);
    const bool filt = !a.bm_only && (a.active & (1 << c));
    for (int i = tid; i < npx; i += blockDim.x) {
        const int y = i / t.rw, x = i - y * t.rw;
        const long long g = static_cast<long long>(t.ry0 + y) * a.stride + (t.rx0 + x);
        const int s = y * t.pitch + x;
        cp_async_elem(const_cast<T *>(t.srcw[0]) + s, a.src[c] + g);
        if (need_ref) cp_async_elem(const_cast<T *>(t.refw[0]) + s, a.ref[c] + g);
        if (filt) t.accN[0].zero(s);
    }
    if (!t.origin_inside) {
        for (int i = tid; i < bsq; i += blockDim.x) {
            const int y = i / bs, x = i - y * bs;
            const long long g = static_cast<long long>(y) * a.stride + x;
            const_cast<T *>(t.src0[0])[i] = __ldg(a.src[c] + g);
            if (need_ref) const_cast<T *>(t.ref0[0])[i] = __ldg(a.ref[c] + g);
            t.accN0[0].zero(i);
        }
    }
    cp_async_wait_all();
    __syncthreads();
}

// Flush plane c's accumulator windows (the single-plane windows) into its sums.
template <typename T>
__device__ __forceinline__ void flush_plane(const StageArgs<T> &a, const Tile<T> &t, int c)
{
    const int tid = threadIdx.x;
    const int npx = t.rh * t.rw;
    const int bs = t.bs, bsq = bs * bs;
    for (int i = tid; i < npx; i += blockDim.x) {
        const int y = i / t.rw, x = i - y * t.rw;
        const int s = y * t.pitch + x;
        const auto nv = t.accN[0].get(s);
        const long long g = static_cast<long long>(t.ry0 + y) * a.width + (t.rx0 + x);
        if (nv != 0) acc_flush(a.num[c] + g, nv);
    }
    if (!t.origin_inside) {
        for (int i = tid; i < bsq; i += blockDim.x) {
            const auto nv = t.accN0[0].get(i);
            const int y = i / bs, x = i - y * bs;
            const long long g = static_cast<long long>(y) * a.width + x;
            if (nv != 0) acc_flush(a.num[c] + g, nv);
        }
    }
}

// Three planes sharing the groups matched on plane 0 (BM3D_Base::Kernel's
// 9-plane form, source/BM3D.cpp:139-218), one plane at a time through a
// single plane's windows: plane 0 matches and keeps each reference block's
// group list in shared memory, planes 1 and 2 re-stage their windows and
// filter with those lists. Per plane the arithmetic is that of the
// one-plane tile, so results equal the all-planes-resident form bit for bit
// while the footprint stays that of one plane (full-size tiles).
template <typename T, bool WIENER, int KS>
__device__ __forceinline__ void stage_tile_body_seq3(const StageArgs<T> &a, int tile,
                                                     unsigned char *smem, unsigned avail)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int right = a.width - kBS, bottom = a.height - kBS;

    Tile<T> t;
    int kx0, kx1, ky0, ky1;
    tile_window(a, tile, kBS, t, kx0, kx1, ky0, ky1);
    const SmemPlan sp = plan_smem<T>(3, WIENER, a.ref_alias_src, a.region_h, a.region_pitch,
                                     a.span, nwarps, false, kBS, kGSMax,
                                     a.tile_x * a.tile_y);
    if (sp.total > avail) {  // launched with less shared memory than the layout needs
        smem_shortfall(a);
        return;
    }
    carve_tile<T, WIENER, 1>(a, sp, smem, t);  // every plane goes through windows [0]
    // group lists: position (y - ry0) << 8 | (x - rx0), or 0xffff for a
    // (0, 0) block held outside the window; then one count byte per block
    unsigned short *gpos = reinterpret_cast<unsigned short *>(smem + sp.off_groups);
    unsigned char *gn = reinterpret_cast<unsigned char *>(gpos + a.tile_x * a.tile_y * kGSMax);

    unsigned *tasks = reinterpret_cast<unsigned *>(smem + sp.off_tasks);
    unsigned char *wbase = smem + sp.off_warps + sp.warp_bytes * warp;
    T *G = reinterpret_cast<T *>(wbase);
    auto *dist = reinterpret_cast<typename DistBits<T>::type *>(wbase);
    T *refblk = reinterpret_cast<T *>(wbase + sp.off_ref);
    SortKey<T> *heap = reinterpret_cast<SortKey<T> *>(wbase + sp.off_heap);
    T *lkeys = reinterpret_cast<T *>(wbase + sp.off_keys);
    BlockPos *list = reinterpret_cast<BlockPos *>(wbase + sp.off_list);

    if (KS == kStrip && warp == 0)
        build_tasks(tasks, reinterpret_cast<unsigned *>(wbase), a.span, t.pitch, lane);

    // per-tile counters (small: 32 bits suffice), flushed once per tile
    unsigned n_sum = 0, n_sq = 0, n_cand = 0, n_fix = 0, n_bad = 0;
    const int tw = kx1 - kx0, nrefs = tw * (ky1 - ky0);
    for (int c = 0; c < 3; ++c) {
        const bool filt = !a.bm_only && (a.active & (1 << c));
        if (c > 0 && !filt) continue;
        stage_plane<T, WIENER>(a, t, c);
        const float scale = fixed_scale(a.absmax[c], a.log2_bound);
        const bool check = poison_map(a, c) != nullptr;
        for (int r = warp; r < nrefs; r += nwarps) {
            int n;
            if (c == 0) {
                const int ky = ky0 + r / tw, kx = kx0 + r % tw;
                const int j0 = ref_pos(ky, a.step, bottom), i0 = ref_pos(kx, a.step, right);
                n = match_block<T, KS>(a, t, j0, i0, lane, tasks, dist, refblk, heap, list, lkeys, n_cand,
                                       n_fix);
                n_sum += n;
                n_sq += static_cast<unsigned>(n * n);
                dump_group(a, ky, kx, n, lane, list, lkeys);
                if (lane == 0) gn[r] = static_cast<unsigned char>(n);
                for (int k = lane; k < n; k += kWarp) {
                    const BlockPos q = list[k];
                    const bool outside = q.y == 0 && q.x == 0 && !t.origin_inside;
                    gpos[r * kGSMax + k] = outside ? 0xffff
                                                   : static_cast<unsigned short>(
                                                         ((q.y - t.ry0) << 8) | (q.x - t.rx0));
                }
            } else {
                n = gn[r];
                for (int k = lane; k < n; k += kWarp) {
                    const unsigned v = gpos[r * kGSMax + k];
                    list[k] = v == 0xffffu ? BlockPos{0, 0}
                                           : BlockPos{t.ry0 + static_cast<int>(v >> 8),
                                                      t.rx0 + static_cast<int>(v & 0xffu)};
                }
            }
            __syncwarp();
            if (filt) filter_group<T, WIENER>(a, t, 0, list, n, lane, G, scale, n_bad, c, check);
            __syncwarp();
        }
        __syncthreads();
        if (filt) flush_plane<T>(a, t, c);
        __syncthreads();  // the windows are re-staged for the next plane
    }
    flush_stats(a, lane, n_sum, n_sq, n_cand, n_fix, n_bad);
}

// Registers bound the warps of a CTA: FP32 runs 16 of 128 registers a thread.
// FP64 values take two registers each: at 128 the kernels spill 240-600 bytes a
// thread, so FP64 runs 8 warps of up to 255 (no spills; lc profile, 640 x 480,
// both stages: 0.852 -> 0.660 ms).
template <typename T> __host__ __device__ constexpr int stage_max_warps() { return sizeof(T) == 4 ? 16 : 8; }

template <typename T, bool WIENER, int NPL, int KS>
__global__ void __launch_bounds__(stage_max_warps<T>() * kWarp, 1) stage_kernel(const StageArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned avail = dynamic_smem_bytes();
    if constexpr (NPL == 3) stage_tile_body_seq3<T, WIENER, KS>(a, blockIdx.x, smem, avail);
    else stage_tile_body<T, WIENER, NPL, KS>(a, blockIdx.x, smem, avail);
}

// dst = num / den (source/BM3D.cpp:130-135, include/Image_Type.hpp:319-332).
// Outside block (0, 0) both sums carry the same fixed-point scale, which
// cancels.
__device__ __forceinline__ float ratio(long long n, long long d)
{
    return static_cast<float>(static_cast<double>(n) / static_cast<double>(d));
}
__device__ __forceinline__ double ratio(double n, double d) { return n / d; }

// One plane of a stage, for the per-pixel kernels.
template <typename T> struct PlaneJob {
    typename AccOf<T>::type *num, *den;
    const T *src;
    const T *ref;              // counted for non-finite pixels too when not null
    T *dst;
    long long src_stride, dst_stride;
    int width, height;
    int block_size;
    float *absmax;
    int log2_bound, log2_corner;  // fixed-point bounds of the stage (StageArgs)
    unsigned *nonfinite;       // non-finite src / ref pixels (may be null)
    unsigned char *poison;     // pixels a non-finite term reached (may be null; all zero
                               // between stages: the normalisation clears what it reads)
    // A basic stage that its final stage follows (FP32; null otherwise). The final
    // stage takes num, zeroed by the normalisation as it reads it, weight sums of
    // its own, zeroed together with the basic stage's, |src|'s maximum as it is,
    // and a count of non-finite pixels that starts from the basic stage's and adds
    // the estimate's: it needs no preparation pass.
    long long *den_next;
    unsigned *nonfinite_next;
    unsigned long long *stats;  // the stage's counters, zeroed for the next
};
template <typename T> struct PlaneJobs {
    PlaneJob<T> job[kMaxPlanes];
};

// Tile of the normalisation: 32 x 32 pixels per CTA.
constexpr int kNormTile = 32;

// FP64 sums: dst = num / den for the kNormTile^2 pixels at (y0, x0), with
// den(y, x) the sum of the block weights W at the bs x bs origins whose block
// covers (y, x): y - bs < oy <= y, x - bs < ox <= x. Separable sums over a
// shared-memory copy of W.
template <typename T>
__device__ __forceinline__ void normalize_tile(T *dst, long long dst_stride, const T *num,
                                               const T *wsum, int width, int height, int bs, int y0,
                                               int x0)
{
    constexpr int N = kNormTile, E = N + kBSMax - 1;
    __shared__ T w[E][E];
    __shared__ T hs[E][N];
    const int ext = N + bs - 1;
    for (int i = threadIdx.x; i < ext * ext; i += blockDim.x) {
        const int ly = i / ext, lx = i - ly * ext;
        const int gy = y0 - bs + 1 + ly, gx = x0 - bs + 1 + lx;
        w[ly][lx] = (gy >= 0 && gx >= 0 && gy < height && gx < width)
                        ? wsum[static_cast<long long>(gy) * width + gx]
                        : T(0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ext * N; i += blockDim.x) {
        const int ly = i / N, lx = i - ly * N;
        T v = 0;
        for (int d = 0; d < bs; ++d) v += w[ly][lx + d];
        hs[ly][lx] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N * N; i += blockDim.x) {
        const int ly = i / N, lx = i - ly * N;
        const int gy = y0 + ly, gx = x0 + lx;
        if (gy >= height || gx >= width) continue;
        T d = 0;
        for (int k = 0; k < bs; ++k) d += hs[ly + k][lx];
        dst[gy * dst_stride + gx] = ratio(num[static_cast<long long>(gy) * width + gx], d);
    }
}

// Fixed-point normalisation of one kFixW x kFixH tile of pixels at (y0, x0) by
// 256 threads: the same sums, exact. Block (0, 0)'s pixels and the weight at
// origin (0, 0) carry the scale of log2_corner, everything else that of
// log2_bound (fixed_scale); for those pixels den = (sum of the other weights) *
// ratio + W(0, 0), ratio = corner scale / general scale (a power of two, exact).
// On planes whose prep found non-finite inputs (*nonfinite != 0) the pixels
// marked in `poison` get NaN -- a non-finite term reached them
// (acc_add_checked) -- and the map is cleared as it is read, so it is all zero
// again for the next stage; other planes never touch it. What bounds it: the
// latency of a tile's dependent steps (its loads, two box sums, a division), so
// a tile has few of them and many tiles are resident. Each warp takes every
// eighth row of block weights: all its loads are issued first, then per row a
// lane sums the bs weights left of and at its two columns from a row buffer
// (16-byte loads; the second column's sum is the first's, moved by one). After
// the one barrier a thread sums bs rows of its column for four pixels and
// divides. Numerators are loaded before the barrier.
// 1080p 30.1 -> 15.5 us, 64 x 64 27 -> 4.3 us against warps walking down 32 x 32
// strips with running sums (39 dependent rows each).
constexpr int kFixW = 64, kFixH = 16;
constexpr int kFixRow = 80;  // words of a row buffer: kFixW + kBSMax

// Rows and columns of tiles of a fixed-point plane.
__host__ __device__ inline int fixed_tiles_x(int width) { return (width + kFixW - 1) / kFixW; }
__host__ __device__ inline int fixed_tiles(int width, int height)
{
    return fixed_tiles_x(width) * ((height + kFixH - 1) / kFixH);
}

// Shared memory of a normalisation CTA: box sums of its window's rows, and a
// row buffer per warp.
struct FixedSmem {
    longlong2 hs[(kFixH + kBSMax - 1) * kFixW / 2];
    longlong2 rowbuf[8][kFixRow / 2];
};

// BS: the block size, or 0 to take it from `block_size`.
template <int BS>
__device__ __forceinline__ void normalize_fixed(FixedSmem &sm, const PlaneJob<float> &q, int y0, int x0)
{
    const int width = q.width, height = q.height;
    const long long *const wsum = q.den;
    constexpr int kMost = BS > 0 ? BS : kBSMax;
    const int bs = BS > 0 ? BS : q.block_size;
    long long *const hs = reinterpret_cast<long long *>(sm.hs);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool split = x0 == 0 && y0 == 0;  // the only tile whose sums reach W(0, 0)
    const int rows = kFixH + bs - 1;
    // this thread's pixels: column x, rows yb .. yb + 3
    const int col = tid & (kFixW - 1), yb = y0 + (tid >> 6) * 4, x = x0 + col;
    long long n[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        n[k] = (x < width && yb + k < height) ? q.num[static_cast<long long>(yb + k) * width + x] : 0;
    // weight rows warp, warp + 8, ... of the tile's window: columns
    // x0 - bs + 1 .. x0 + kFixW - 1, three words per lane at most
    constexpr int kRows = (kFixH + kMost - 1 + 7) / 8;
    long long w[kRows][3];
    const int xa = x0 - bs + 1;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int r = warp + 8 * k, gy = y0 - bs + 1 + r;
        const bool in = r < rows && gy >= 0 && gy < height;
        const long long *row = wsum + static_cast<long long>(gy) * width;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int c = j < 2 ? 2 * lane + j : kFixW + lane, gx = xa + c;
            const bool ok = in && gx >= 0 && gx < width && (j < 2 || lane < bs - 1) &&
                            !(split && gy == 0 && gx == 0);
            w[k][j] = ok ? row[gx] : 0;
        }
    }
    long long *const buf = reinterpret_cast<long long *>(sm.rowbuf[warp]);
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
        const int r = warp + 8 * k;
        if (r >= rows) break;  // warp-uniform
        __syncwarp();
        *reinterpret_cast<longlong2 *>(buf + 2 * lane) = make_longlong2(w[k][0], w[k][1]);
        if (lane < kBSMax) buf[kFixW + lane] = w[k][2];
        __syncwarp();
        long long h = 0;
        int d = 0;
#pragma unroll
        for (; d + 1 < bs; d += 2) {
            const longlong2 v = *reinterpret_cast<const longlong2 *>(buf + 2 * lane + d);
            h += v.x + v.y;
        }
        if (d < bs) h += buf[2 * lane + d];
        *reinterpret_cast<longlong2 *>(hs + r * kFixW + 2 * lane) =
            make_longlong2(h, h - w[k][0] + buf[2 * lane + bs]);
    }
    __syncthreads();
    if (x < width && yb < height) {
        const bool marked = q.poison != nullptr && q.nonfinite != nullptr && *q.nonfinite != 0;
        const bool next = q.nonfinite_next != nullptr;
        unsigned bad = 0;
        if (next && split && tid == 0) {
            bad = *q.nonfinite;
            if (q.stats != nullptr)
                for (int k = 0; k < 4; ++k) q.stats[k] = 0;
        }
        const long long *c = hs + (yb - y0) * kFixW + col;
        long long v = 0;
#pragma unroll
        for (int d = 0; d < bs - 1; ++d) v += c[d * kFixW];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int y = yb + k;
            if (y >= height) break;
            v += c[(k + bs - 1) * kFixW];
            float out;
            if (split && y < bs && x < bs) {  // block (0, 0): covered by origin (0, 0)
                const float am = *q.absmax;
                const double cratio = static_cast<double>(fixed_scale(am, q.log2_corner)) /
                                      static_cast<double>(fixed_scale(am, q.log2_bound));
                out = static_cast<float>(static_cast<double>(n[k]) /
                                         (static_cast<double>(v) * cratio +
                                          static_cast<double>(wsum[0])));
            } else {
                out = ratio(n[k], v);
            }
            const long long g = static_cast<long long>(y) * width + x;
            if (marked && q.poison[g]) {
                out = NAN;
                q.poison[g] = 0;
            }
            q.dst[y * q.dst_stride + x] = out;
            if (next) {
                q.num[g] = 0;
                if (!(fabsf(out) <= 3.4028235e38f)) ++bad;
            }
            v -= c[k * kFixW];
        }
        if (bad) atomicAdd(q.nonfinite_next, bad);
    }
}

// Tile `tile` of a plane's normalisation (normalize_tiles in all).
template <typename T> __host__ __device__ inline int normalize_tiles(int width, int height)
{
    if (sizeof(T) == 4) return fixed_tiles(width, height);
    return ((width + kNormTile - 1) / kNormTile) * ((height + kNormTile - 1) / kNormTile);
}
__device__ __forceinline__ void normalize_job(const PlaneJob<float> &q, int tile)
{
    __shared__ FixedSmem sm;
    const int tx = fixed_tiles_x(q.width), ty = tile / tx;
    if (q.block_size == kBS) normalize_fixed<kBS>(sm, q, ty * kFixH, (tile - ty * tx) * kFixW);
    else normalize_fixed<0>(sm, q, ty * kFixH, (tile - ty * tx) * kFixW);
}
__device__ __forceinline__ void normalize_job(const PlaneJob<double> &q, int tile)
{
    const int tx = (q.width + kNormTile - 1) / kNormTile, ty = tile / tx;
    normalize_tile<double>(q.dst, q.dst_stride, q.num, q.den, q.width, q.height, q.block_size,
                           ty * kNormTile, (tile - ty * tx) * kNormTile);
}

// The planes of one stage call (grid.y), one CTA of 256 threads per tile.
template <typename T>
__global__ void __launch_bounds__(256) normalize_kernel(const PlaneJobs<T> jobs)
{
    normalize_job(jobs.job[blockIdx.y], static_cast<int>(blockIdx.x));
}

// Zero one plane's accumulators and fold the largest finite |src| into
// *absmax (which the caller zeroes first; non-negative floats order like their
// bit patterns). With `nonfinite` (FP32 only) it also counts the NaN / Inf
// pixels of src and of ref (when given) into *nonfinite, so that the stage
// kernel checks its terms only on such planes. Rows row0, row0 + row_step, ...
// of the plane, threads along each row.
template <typename T>
__device__ __forceinline__ void prep_plane(const PlaneJob<T> &q, int row0, int row_step)
{
    using Acc = typename AccOf<T>::type;
    Acc *const num = q.num, *const den = q.den;
    long long *const den2 = q.den_next;
    const int width = q.width, height = q.height;
    float m = 0.0f;
    unsigned bad = 0;
    for (int y = row0; y < height; y += row_step) {
        const long long o = static_cast<long long>(y) * width;
        const T *s = q.src + static_cast<long long>(y) * q.src_stride;
        const T *r = q.ref != nullptr ? q.ref + static_cast<long long>(y) * q.src_stride : nullptr;
        if constexpr (sizeof(T) == 4) {
            // two pixels per thread where the row allows 16-byte sum stores
            // and 8-byte source loads (uniform over the CTA)
            const bool vec = (width % 2 == 0) &&
                             ((reinterpret_cast<uintptr_t>(num + o) | reinterpret_cast<uintptr_t>(den + o) |
                               (den2 != nullptr ? reinterpret_cast<uintptr_t>(den2 + o) : 0)) & 15) == 0 &&
                             ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(r)) & 7) == 0;
            if (vec) {
                for (int x = 2 * threadIdx.x; x < width; x += 2 * blockDim.x) {
                    *reinterpret_cast<longlong2 *>(num + o + x) = make_longlong2(0, 0);
                    *reinterpret_cast<longlong2 *>(den + o + x) = make_longlong2(0, 0);
                    if (den2 != nullptr)
                        *reinterpret_cast<longlong2 *>(den2 + o + x) = make_longlong2(0, 0);
                    const float2 v2 = *reinterpret_cast<const float2 *>(s + x);
                    const float v0 = fabsf(v2.x), v1 = fabsf(v2.y);
                    if (v0 <= 3.4028235e38f) m = v0 > m ? v0 : m;  // NaN and Inf are skipped
                    else ++bad;
                    if (v1 <= 3.4028235e38f) m = v1 > m ? v1 : m;
                    else ++bad;
                    if (r != nullptr) {
                        const float2 r2 = *reinterpret_cast<const float2 *>(r + x);
                        if (!(fabsf(r2.x) <= 3.4028235e38f)) ++bad;
                        if (!(fabsf(r2.y) <= 3.4028235e38f)) ++bad;
                    }
                }
                continue;
            }
        }
        for (int x = threadIdx.x; x < width; x += blockDim.x) {
            num[o + x] = 0;
            den[o + x] = 0;
            if (den2 != nullptr) den2[o + x] = 0;
            const float v = fabsf(static_cast<float>(s[x]));
            if (v <= 3.4028235e38f) m = v > m ? v : m;  // NaN and Inf are skipped
            else ++bad;
            if (r != nullptr && !(fabsf(static_cast<float>(r[x])) <= 3.4028235e38f)) ++bad;
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float q = __shfl_xor_sync(0xffffffffu, m, o);
        m = q > m ? q : m;
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (m > 0.0f) atomicMax(reinterpret_cast<int *>(q.absmax), __float_as_int(m));
        if (q.nonfinite != nullptr && bad) atomicAdd(q.nonfinite, bad);
    }
}

// The planes of one stage call (grid.y), one row per CTA at a time.
template <typename T> __global__ void prep_kernel(const PlaneJobs<T> jobs)
{
    prep_plane<T>(jobs.job[blockIdx.y], blockIdx.x, gridDim.x);
}

}  // namespace bm3d
