// Generic BM3D stage kernel: any BlockSize <= 16, GroupSize <= 32, BMrange,
// BMstep -- the reference's other profiles ("np", "high", "vn") and custom
// parameters. One warp per reference block; the group lives in shared memory
// and the separable 3-D transforms run one line per lane: 8-point butterflies
// for BlockSize 8, recursive even/odd splits for full GroupSize-32 groups,
// cosine matrices from global memory otherwise. Block matching keeps the
// reference's exact distance order (BlockSize 8, and 11 in FP32, with step 1 use
// the register-resident kernel's strips); selection, aggregation and the staged
// windows are shared with the register-resident kernel.
//
// Reference: as bm3d_stage.cuh (source/BM3D.cpp:80-457, include/Block.h:578-751).
#pragma once

#include "bm3d_stage.cuh"

namespace bm3d {

// In-place length-n transform of one strided line, by one lane: out[k] =
// sum_j mat[k n + j] in[j] (row k = output k), n <= kGSTab. What bounds it: the
// latency of a chain of n loads and multiply-adds per output (FP64 11 x 11 blocks
// in groups of 32, 300 x 250, basic stage, one output at a time: 1.27 ms, 0.83 so).
template <typename T>
__device__ __forceinline__ void dct_line(T *base, int stride, int n, const T *mat)
{
    if (n == 1) {
        T a = T(0);
        a += __ldg(mat) * base[0];
        base[0] = a;
        return;
    }
    T in[kGSTab];
#pragma unroll
    for (int j = 0; j < kGSTab; ++j) in[j] = j < n ? base[j * stride] : T(0);
    for (int k = 0; k < n; k += 2) {  // two outputs: their chains of sums overlap
        const T *row = mat + k * n, *next = k + 1 < n ? row + n : row;
        T a = T(0), b = T(0);
#pragma unroll
        for (int j = 0; j < kGSTab; ++j)
            if (j < n) {
                a += __ldg(row + j) * in[j];
                b += __ldg(next + j) * in[j];
            }
        base[k * stride] = a;
        if (k + 1 < n) base[(k + 1) * stride] = b;
    }
}

// One 8-point line of an 8 x 8 block, in place, by the butterflies of dct.cuh.
template <typename T>
__device__ __forceinline__ void dct_line8(T *base, int stride, bool inverse)
{
    T v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = base[j * stride];
    if (inverse) redft01_8(v);
    else redft10_8(v);
#pragma unroll
    for (int j = 0; j < 8; ++j) base[j * stride] = v[j];
}

// One 11-point line (FP32), in place, by the symmetric form with
// constant-bank cosines; other precisions never reach it.
template <typename T>
__device__ __forceinline__ void dct_line11(T *base, int stride, bool inverse)
{
    if constexpr (sizeof(T) == 4) {
        T v[11];
#pragma unroll
        for (int j = 0; j < 11; ++j) v[j] = base[j * stride];
        if (inverse) redft01_line<T, 11>(v, c_dct.d11_inv);
        else redft10_line<T, 11>(v, c_dct.d11_fwd);
#pragma unroll
        for (int j = 0; j < 11; ++j) base[j * stride] = v[j];
    }
}

template <typename T>
__device__ void dct_z_generic(T *G, int n, int bs, int lane, const T *tab, const float *pad, bool inverse);

// Separable 3-D transform of an n x bs x bs group (row-major [z][y][x]) with
// the concatenated matrices `tab` (forward REDFT10 or backward REDFT01, as
// `inverse` says): rows, columns, then the group axis. The row-fused block
// sizes (8, and 11 in FP32) do not come here: their rows are transformed as they are
// gathered or aggregated, their other passes in dct_cols_z_fwd /
// dct_z_cols_inv.
template <typename T>
__device__ void dct3_generic(T *G, int n, int bs, int lane, const T *tab, const float *pad, bool inverse)
{
    const int bsq = bs * bs;
    const T *mb = tab + dct_table_offset(bs);
    for (int line = lane; line < n * bs; line += kWarp)  // along x
        dct_line(G + line * bs, 1, bs, mb);
    __syncwarp();
    for (int line = lane; line < n * bs; line += kWarp) {  // along y
        const int z = line / bs, x = line - z * bs;
        dct_line(G + z * bsq + x, bs, bs, mb);
    }
    __syncwarp();
    dct_z_generic(G, n, bs, lane, tab, pad, inverse);
}

// Row-fused block sizes: 8 and 11 (FP32, the "vn" final stage). Rows are
// transformed in registers as they are gathered (gather_rows) or aggregated
// (aggregate_rows); these run the other passes.

// One line of BS points, in place, by the block size's butterflies or
// constant-bank symmetric form.
template <typename T, int BS>
__device__ __forceinline__ void dct_line_bs(T *base, int stride, bool inverse)
{
    if constexpr (BS == 8) dct_line8(base, stride, inverse);
    else dct_line11(base, stride, inverse);
}

// Forward, after gather_rows (which transformed the rows): the columns, then
// the group axis -- the passes and order of dct3_generic.
template <typename T, int BS>
__device__ void dct_cols_z_fwd(T *G, int n, int lane, const T *tab, const float *pad)
{
    constexpr int ZS = BS == 8 ? 72 : BS * BS, RS = BS == 8 ? 9 : BS;
    for (int line = lane; line < n * BS; line += kWarp) {  // along y
        const int z = line / BS, x = line - z * BS;
        dct_line_bs<T, BS>(G + z * ZS + x, RS, false);
    }
    __syncwarp();
    dct_z_generic(G, n, BS, lane, tab, pad, false);
}

// Inverse: the group axis, then the columns; the rows are transformed by
// aggregate_rows as it adds them (the register-resident kernel's inverse
// order).
template <typename T, int BS>
__device__ void dct_z_cols_inv(T *G, int n, int lane, const T *tab, const float *pad)
{
    constexpr int ZS = BS == 8 ? 72 : BS * BS, RS = BS == 8 ? 9 : BS;
    dct_z_generic(G, n, BS, lane, tab, pad, true);
    for (int line = lane; line < n * BS; line += kWarp) {  // along y
        const int z = line / BS, x = line - z * BS;
        dct_line_bs<T, BS>(G + z * ZS + x, RS, true);
    }
    __syncwarp();
}

// Group-axis transform of pencils g0 and g1 (length n < 32, stride zs)
// by matrix columns m of 32 rows: y_k = sum_j m[k][j] x_j, j in order, from the
// buffer into registers. ROWS (16 or 32) bounds n. Sums of all rows advance
// together, so a step is independent loads and multiply-adds; row by row, each
// output waited for its own chain of loads and adds, and one short group could
// take longer than the rest of a tile.
template <int ROWS>
__device__ __forceinline__ void pencils_by_columns(const float *g0, const float *g1, int zs, int n,
                                                   const float *m, Pair<float> (&out)[kGSTab])
{
    float a[ROWS], b[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) a[k] = b[k] = 0.0f;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
        const float x0 = g0[j * zs], x1 = g1[j * zs];
        const float4 *c = reinterpret_cast<const float4 *>(m + 32 * j);
#pragma unroll
        for (int k = 0; k < ROWS; k += 4) {
            const float4 q = __ldg(c + k / 4);
            const float r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[k + i] = fmaf(r[i], x0, a[k + i]);
                b[k + i] = fmaf(r[i], x1, b[k + i]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kGSTab; ++k)
        out[k] = k < ROWS ? Pair<float>::make(a[k < ROWS ? k : 0], b[k < ROWS ? k : 0])
                          : Pair<float>::make(0.0f, 0.0f);
}

// The group-axis pass of a separable 3-D transform (see dct3_generic). FP32: two
// pencils at a time as the halves of pairs, recursive even/odd splits for full
// groups of 32 (dct.cuh), matrix columns for shorter ones.
template <typename T>
__device__ void dct_z_generic(T *G, int n, int bs, int lane, const T *tab, const float *pad, bool inverse)
{
    // along the group: pencil p = (y, x) of every block
    const int bsq = bs * bs;
    const int zs = generic_block_stride(bs), rs = generic_row_stride(bs);
    auto pencil = [&](int line) {
        const int py = line / bs;
        return G + py * rs + (line - py * bs);
    };
    if constexpr (sizeof(T) == 4) {
        using P = Pair<float>;
        const float *m = pad + pad32_offset(n < 32 ? n : 1);
        for (int line = lane; line < bsq; line += 2 * kWarp) {
            float *g0 = pencil(line);
            const bool both = line + kWarp < bsq;
            float *g1 = both ? pencil(line + kWarp) : g0;
            P v[kGSTab];
            if (n == 32) {
#pragma unroll
                for (int j = 0; j < kGSTab; ++j) v[j] = P::make(g0[j * zs], g1[j * zs]);
                if (inverse) redft01_pow2<P, kGSTab>(v);
                else redft10_pow2<P, kGSTab>(v);
            } else if (n <= 16) {
                pencils_by_columns<16>(g0, g1, zs, n, m, v);
            } else {
                pencils_by_columns<32>(g0, g1, zs, n, m, v);
            }
#pragma unroll
            for (int k = 0; k < kGSTab; ++k)
                if (k < n) {
                    g0[k * zs] = v[k].lo();
                    if (both) g1[k * zs] = v[k].hi();
                }
        }
    } else {
        const T *mz = tab + dct_table_offset(n);
        for (int line = lane; line < bsq; line += kWarp) dct_line(pencil(line), zs, n, mz);
    }
    __syncwarp();
}

// Block matching of (j0, i0) for any block size and search step: one lane per
// candidate, sequential row-major distances against a copy of the reference
// block (include/Block.h:589-611), then the shared ordered selection.
template <typename T>
__device__ int match_generic(const StageArgs<T> &a, const Tile<T> &t, int j0, int i0, int lane,
                             typename DistBits<T>::type *dist, T *refblk, SortKey<T> *heap,
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
    const int bs = t.bs, bsq = bs * bs;
    const int st = a.bm_step, R = a.range;
    const int right = a.width - bs, bottom = a.height - bs;
    const int l = search_boundary(i0, 0, R, st), r = search_boundary(i0, right, R, st);
    const int tp = search_boundary(j0, 0, R, st), b = search_boundary(j0, bottom, R, st);
    const int nr = (b - tp) / st + 1, nc = (r - l) / st + 1;
    const int ngrid = nr * nc;
    {
        const T *rb = t.refw[0] + (j0 - t.ry0) * t.pitch + (i0 - t.rx0);
        for (int e = lane; e < bsq; e += kWarp) {
            const int y = e / bs;
            refblk[e] = rb[y * t.pitch + (e - y * bs)];
        }
    }
    __syncwarp();
    const unsigned nc_div = div_number(nc);
    const B limit = dist_limit(a.thSSE);
    int nvalid = 0;
    for (int c = lane; c <= ngrid; c += kWarp) {
        const T *cand;
        int cp;
        if (c < ngrid) {
            const int rr = div_magic(c, nc_div), cc = c - rr * nc;
            const int cy = tp + rr * st, cx = l + cc * st;
            cand = t.refw[0] + (cy - t.ry0) * t.pitch + (cx - t.rx0);
            cp = t.pitch;
        } else {
            cand = block_ptr(t, t.refw[0], t.ref0[0], 0, 0, cp);  // the trailing (0, 0) slot
        }
        T d = T(0);
        if (bs == 11) {  // the same order, unrolled
#pragma unroll
            for (int y = 0; y < 11; ++y)
#pragma unroll
                for (int x = 0; x < 11; ++x) {
                    const T df = sub_rn(refblk[y * 11 + x], cand[y * cp + x]);
                    d = add_rn(d, mul_rn(df, df));
                }
        } else {
            for (int y = 0; y < bs; ++y)
                for (int x = 0; x < bs; ++x) {
                    const T df = sub_rn(refblk[y * bs + x], cand[y * cp + x]);
                    d = add_rn(d, mul_rn(df, df));
                }
        }
        dist[c] = accept_dist(DistBits<T>::of(d), limit, nvalid);
    }
    __syncwarp();
    n_cand += static_cast<unsigned>(ngrid);
    Search<T> e = {};
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
    e.dist = dist;
    e.heap = heap;
    e.list = list;
    e.lkeys = lkeys;
    return select_group<T, false, kBS>(e, false, lane, nvalid, n_fix);
}

// Whether blocks of size bs match by strips of candidates (with BMstep 1).
template <typename T, int BSC> __device__ __forceinline__ bool strip_blocks(int bs)
{
    return BSC == kBS || BSC == 11 || (sizeof(T) == 8 && BSC == 0 && bs == kBS);
}

// Block matching by strips where they apply, else one lane per candidate.
template <typename T, int BSC>
__device__ __forceinline__ int match_any(const StageArgs<T> &a, const Tile<T> &t, bool strips, int j0,
                                         int i0, int lane, const unsigned *tasks,
                                         typename DistBits<T>::type *dist, T *refblk, SortKey<T> *heap,
                                         BlockPos *list, T *lkeys, unsigned &n_cand, unsigned &n_fix)
{
    if constexpr (BSC > 0 || sizeof(T) == 8) {
        if (strips)
            return match_block<T, kStrip, (BSC > 0 ? BSC : kBS)>(a, t, j0, i0, lane, tasks, dist, refblk,
                                                                  heap, list, lkeys, n_cand, n_fix);
    }
    return match_generic<T>(a, t, j0, i0, lane, dist, refblk, heap, list, lkeys, n_cand, n_fix);
}

// Element e of a group stored [z][y][x]: shifts for BlockSize 8, divisions
// otherwise.
__device__ __forceinline__ void group_index(int e, int bs, int bsq, int &z, int &y, int &x)
{
    if (bs == 8) {
        z = e >> 6;
        y = (e >> 3) & 7;
        x = e & 7;
    } else if (bs == 11) {  // constant divisors
        z = e / 121;
        const int rem = e - z * 121;
        y = rem / 11;
        x = rem - y * 11;
    } else {
        z = e / bsq;
        const int rem = e - z * bsq;
        y = rem / bs;
        x = rem - y * bs;
    }
}

// Gather the group's block rows and transform each along x in registers as
// it arrives (the rows pass of the forward transform), into G's layout (row
// stride RS, block stride ZS; row z * BS + y starts at its index times RS).
// Members outside the tile (never, by construction) read as zero blocks and
// are counted in n_bad.
template <typename T, int BS>
__device__ __forceinline__ void gather_rows(const Tile<T> &t, const T *win, const T *win0,
                                            const BlockPos *list, int n, int lane, T *G,
                                            unsigned *n_bad)
{
    constexpr int RS = BS == 8 ? 9 : BS;
    for (int line = lane; line < n * BS; line += kWarp) {  // line = z * BS + y
        const int z = line / BS, y = line - z * BS;
        const BlockPos q = list[z];
        const bool ok = block_in_tile(t, q.y, q.x);
        if (n_bad && !ok && y == 0) ++*n_bad;
        T v[BS];
        if (ok) {
            int pitch;
            const T *bp = block_ptr(t, win, win0, q.y, q.x, pitch);
            bp += y * pitch;
#pragma unroll
            for (int x = 0; x < BS; ++x) v[x] = bp[x];
        } else {
#pragma unroll
            for (int x = 0; x < BS; ++x) v[x] = T(0);
        }
        if constexpr (BS == 8) redft10_8(v);
        else redft10_line<T, BS>(v, c_dct.d11_fwd);
        T *g = G + line * RS;
#pragma unroll
        for (int x = 0; x < BS; ++x) g[x] = v[x];
    }
}

// The rows pass of the inverse transform, each row added to the tile's sums
// as soon as it is transformed (BlockGroup::AddTo / CountTo,
// include/Block.h:1240-1265, 1334-1357); the block weight once per block, at
// its origin. Members reaching block (0, 0)'s pixels, and planes with
// non-finite pixels, take the checking per-term form.
template <typename T, int BS>
__device__ __forceinline__ void aggregate_rows(const StageArgs<T> &a, const Tile<T> &t, int p,
                                               int pt, const BlockPos *list, int n, int lane,
                                               const T *G, T numW, T denW, float scale,
                                               bool check)
{
    constexpr int RS = BS == 8 ? 9 : BS;
    for (int line = lane; line < n * BS; line += kWarp) {  // line = z * BS + y
        const int z = line / BS, y = line - z * BS;
        const BlockPos q = list[z];
        if (!block_in_tile(t, q.y, q.x)) continue;
        T v[BS];
        const T *g = G + line * RS;
#pragma unroll
        for (int x = 0; x < BS; ++x) v[x] = g[x];
        if constexpr (BS == 8) redft01_8(v);
        else redft01_line<T, BS>(v, c_dct.d11_inv);
        int pitch;
        AccWin<T> dn = block_acc(t, p, q.y, q.x, pitch);
        dn = dn + y * pitch;
        if (!check && (q.y >= BS || q.x >= BS)) {
#pragma unroll
            for (int x = 0; x < BS; ++x) acc_add(dn + x, v[x] * numW, scale);
            if (y == 0) weight_add(a.den[pt], a.width, q.y, q.x, denW, scale);
        } else {
            const float scale_c = fixed_scale(a.absmax[pt], a.log2_corner);
            unsigned char *const poison = poison_map(a, pt);
            unsigned char *mk =
                poison ? poison + static_cast<long long>(q.y + y) * a.width + q.x : nullptr;
            for (int x = 0; x < BS; ++x) {
                const bool corner = q.y + y < BS && q.x + x < BS;
                acc_add_checked(dn + x, v[x] * numW, corner ? scale_c : scale,
                                mk ? mk + x : nullptr);
            }
            if (y == 0) {
                const float sd = (q.y == 0 && q.x == 0) ? scale_c : scale;
                if (mk == nullptr || fabsf(static_cast<float>(denW) * sd) < kFixedLimit)
                    weight_add(a.den[pt], a.width, q.y, q.x, denW, sd);
                else  // the block's weight reaches all of its pixels
                    for (int i = 0; i < BS * BS; ++i)
                        mk[static_cast<long long>(i / BS) * a.width + i % BS] = 1;
            }
        }
    }
}

// Collaborative filtering of an FP32 group of 8 x 8 blocks, up to 32 of them, in
// one group buffer of the register-resident kernel's layout and passes (16-byte
// rows, columns in packed pairs). Each lane owns pencils lane and lane + 32 of
// the group axis as the halves of pairs: full groups of 32 stay in registers from
// the last column pass to the first inverse one, and the Wiener weights in 64
// more while the noisy group takes the buffer; shorter groups go through matrix
// columns (pencils_by_columns). What bounds it: issue slots and, at 12 warps of 168 registers,
// latency. Against scalar lines in rows of 9 words (and, for short groups, row by
// row products): np on 1283 x 717 3.33 -> 2.78 ms, its final stage on 64 x 64
// 127 -> 53 us.
template <bool WIENER>
__device__ void filter_group32(const StageArgs<float> &a, const Tile<float> &t, int p,
                               const BlockPos *list, int n, int lane, float *G, float scale,
                               unsigned &n_bad, int pt, bool check)
{
    using P = Pair<float>;
    float *const g0 = G + gidx(lane >> 3, lane & 7);        // pencil lane
    float *const g1 = G + gidx((lane >> 3) + 4, lane & 7);  // pencil lane + 32
    auto by_columns = [&](const float *m, P (&v)[kGSTab]) {
        if (n <= 16) pencils_by_columns<16>(g0, g1, kGroupStride, n, m + pad32_offset(n), v);
        else pencils_by_columns<32>(g0, g1, kGroupStride, n, m + pad32_offset(n), v);
    };
    auto forward = [&](P (&v)[kGSTab]) {
        if (n == kGSTab) {
#pragma unroll
            for (int z = 0; z < kGSTab; ++z)
                v[z] = P::make(g0[z * kGroupStride], g1[z * kGroupStride]);
            redft10_pow2<P, kGSTab>(v);
        } else {
            by_columns(a.pad_fwd, v);
        }
    };
    auto store = [&](const P (&v)[kGSTab]) {
#pragma unroll
        for (int z = 0; z < kGSTab; ++z)
            if (z < n) {
                g0[z * kGroupStride] = v[z].lo();
                g1[z * kGroupStride] = v[z].hi();
            }
    };
    P w[kGSTab];
    float denW;
    if (WIENER) {
        unsigned none = 0;
        gather_xy_forward<float, kGSTab>(t, t.refw[p], t.ref0[p], list, n, lane, G, none);
        forward(w);
        const float s2 = a.wss[pt][n - 1];
        float l2 = 0.0f;
#pragma unroll
        for (int z = 0; z < kGSTab; ++z) {
            if (z < n) {
                const float y0 = w[z].lo(), y1 = w[z].hi();
                const float w0 = wiener_weight(y0 * y0, s2);
                l2 += w0 * w0;
                const float w1 = wiener_weight(y1 * y1, s2);
                l2 += w1 * w1;
                w[z] = P::make(w0, w1);
            }
        }
        l2 = warp_sum(l2);
        denW = l2 <= 0.0f ? 1.0f : 1.0f / l2;
        __syncwarp();
    }
    gather_xy_forward<float, kGSTab>(t, t.srcw[p], t.src0[p], list, n, lane, G, n_bad);
    P v[kGSTab];
    forward(v);
    if (WIENER) {
#pragma unroll
        for (int z = 0; z < kGSTab; ++z)
            if (z < n) v[z] = vmul(v[z], w[z]);
    } else {
        // hard threshold (source/BM3D.cpp:361-371) with thr by #zero indices
        const float *thr = a.thr[pt][n - 1];
        const int f0 = ((lane & 7) == 0) + (lane < 8), f1 = (lane & 7) == 0;
        int kept = 0;
#pragma unroll
        for (int z = 0; z < kGSTab; ++z) {
            if (z < n) {
                float x0 = v[z].lo(), x1 = v[z].hi();
                if (fabsf(x0) <= thr[f0 + (z == 0)]) x0 = 0.0f; else ++kept;
                if (fabsf(x1) <= thr[f1 + (z == 0)]) x1 = 0.0f; else ++kept;
                v[z] = P::make(x0, x1);
            }
        }
        const int retained = __reduce_add_sync(0xffffffffu, kept);
        denW = retained < 1 ? 1.0f : 1.0f / static_cast<float>(retained);
    }
    const float numW = static_cast<float>(static_cast<double>(denW) / a.finalAMP[n - 1]);
    if (n == kGSTab) {
        redft01_pow2<P, kGSTab>(v);
    } else {  // a lane reads back only its own pencils
        store(v);
        by_columns(a.pad_inv, v);
    }
    store(v);
    __syncwarp();
    xy_cols<float, kGSTab, true>(G, n, lane);
    aggregate_group<float, kGSTab>(a, t, p, pt, list, n, lane, G, numW, denW, scale, check);
}

// Collaborative filtering of one group on plane p (generic sizes; BSC as in
// generic_stage_kernel).
template <typename T, bool WIENER, int BSC>
__device__ void filter_generic(const StageArgs<T> &a, const Tile<T> &t, int p, const BlockPos *list,
                               int n, int lane, T *Gs, T *Gr, float scale,
                               unsigned &n_bad, int pt = -1, bool check = false)
{
    // p indexes the tile's windows; pt (default p) the plane's threshold /
    // Wiener tables, which differ when planes share one set of windows
    if (pt < 0) pt = p;
    if constexpr (BSC == kBS) {
        filter_group32<WIENER>(a, t, p, list, n, lane, Gs, scale, n_bad, pt, check);
        return;
    }
    const int bs = BSC > 0 ? BSC : t.bs, bsq = bs * bs, total = n * bsq;
    const int zs = generic_block_stride(bs), rs = generic_row_stride(bs);
    // FP32's 8 and 11 have kernels of their own; FP64's 8 shares this one
    const bool eight = sizeof(T) == 8 && bs == 8;
    constexpr bool kEleven = BSC == 11;
    T denW;
    if (eight) {
        gather_rows<T, 8>(t, t.srcw[p], t.src0[p], list, n, lane, Gs, &n_bad);
        if (WIENER)
            gather_rows<T, 8>(t, t.refw[p], t.ref0[p], list, n, lane, Gr,
                              static_cast<unsigned *>(nullptr));
        __syncwarp();
        dct_cols_z_fwd<T, 8>(Gs, n, lane, a.dct_fwd, a.pad_fwd);
    } else if (kEleven) {
        if constexpr (kEleven) {
            gather_rows<T, 11>(t, t.srcw[p], t.src0[p], list, n, lane, Gs, &n_bad);
            if (WIENER)
                gather_rows<T, 11>(t, t.refw[p], t.ref0[p], list, n, lane, Gr,
                                   static_cast<unsigned *>(nullptr));
            __syncwarp();
            dct_cols_z_fwd<T, 11>(Gs, n, lane, a.dct_fwd, a.pad_fwd);
        }
    } else {
        for (int e = lane; e < total; e += kWarp) {
            int z, y, x;
            group_index(e, bs, bsq, z, y, x);
            const int g = z * zs + y * rs + x;
            const BlockPos q = list[z];
            const bool ok = block_in_tile(t, q.y, q.x);
            if (!ok && y == 0 && x == 0) ++n_bad;
            int pitch;
            const T *bp =
                block_ptr(t, t.srcw[p], t.src0[p], ok ? q.y : t.ry0, ok ? q.x : t.rx0, pitch);
            Gs[g] = ok ? bp[y * pitch + x] : T(0);
            if (WIENER) {
                const T *rp =
                    block_ptr(t, t.refw[p], t.ref0[p], ok ? q.y : t.ry0, ok ? q.x : t.rx0, pitch);
                Gr[g] = ok ? rp[y * pitch + x] : T(0);
            }
        }
        __syncwarp();
        dct3_generic(Gs, n, bs, lane, a.dct_fwd, a.pad_fwd, false);
    }
    if (!WIENER) {
        // hard threshold (source/BM3D.cpp:361-371) with thr by #zero indices
        const T *thr = a.thr[pt][n - 1];
        int kept = 0;
        for (int e = lane; e < total; e += kWarp) {
            int z, y, x;
            group_index(e, bs, bsq, z, y, x);
            const int g = z * zs + y * rs + x;
            const T v = Gs[g];
            const T av = v < T(0) ? -v : v;
            if (av <= thr[(x == 0) + (y == 0) + (z == 0)]) Gs[g] = T(0);
            else ++kept;
        }
        const int retained = __reduce_add_sync(0xffffffffu, kept);
        denW = retained < 1 ? T(1) : T(1) / static_cast<T>(retained);
    } else {
        if (eight) dct_cols_z_fwd<T, 8>(Gr, n, lane, a.dct_fwd, a.pad_fwd);
        else if (kEleven) {
            if constexpr (kEleven) dct_cols_z_fwd<T, 11>(Gr, n, lane, a.dct_fwd, a.pad_fwd);
        } else {
            dct3_generic(Gr, n, bs, lane, a.dct_fwd, a.pad_fwd, false);
        }
        const T s2 = a.wss[pt][n - 1];
        T l2 = T(0);
        for (int e = lane; e < total; e += kWarp) {
            // any one-to-one order works here; the padded layout needs its address
            const int g = eight ? (e >> 6) * 72 + ((e >> 3) & 7) * 9 + (e & 7) : e;
            const T y2 = Gr[g] * Gr[g];
            const T w = wiener_weight(y2, s2);
            Gs[g] *= w;
            l2 += w * w;
        }
        l2 = warp_sum(l2);
        denW = l2 <= T(0) ? T(1) : T(1) / l2;
    }
    const T numW = static_cast<T>(static_cast<double>(denW) / a.finalAMP[n - 1]);
    __syncwarp();
    if (eight) {
        dct_z_cols_inv<T, 8>(Gs, n, lane, a.dct_inv, a.pad_inv);
        aggregate_rows<T, 8>(a, t, p, pt, list, n, lane, Gs, numW, denW, scale, check);
        __syncwarp();
        return;
    }
    if constexpr (kEleven) {
        dct_z_cols_inv<T, 11>(Gs, n, lane, a.dct_inv, a.pad_inv);
        aggregate_rows<T, 11>(a, t, p, pt, list, n, lane, Gs, numW, denW, scale, check);
        __syncwarp();
        return;
    }
    dct3_generic(Gs, n, bs, lane, a.dct_inv, a.pad_inv, true);
    // the block weight once per block, at its origin (as the register-resident kernel)
    for (int e = lane; e < total; e += kWarp) {
        int z, y, x;
        group_index(e, bs, bsq, z, y, x);
        const BlockPos q = list[z];
        if (!block_in_tile(t, q.y, q.x)) continue;
        int pitch;
        AccWin<T> dn = block_acc(t, p, q.y, q.x, pitch);
        if (!check && (q.y >= bs || q.x >= bs)) {
            acc_add(dn + (y * pitch + x), Gs[z * zs + y * rs + x] * numW, scale);
            if (y == 0 && x == 0)
                weight_add(a.den[pt], a.width, q.y, q.x, denW, scale);
        } else {
            // a member reaching block (0, 0)'s pixels (their own scale), or a plane
            // with non-finite pixels (per-term check, marks into the poison map)
            const float scale_c = fixed_scale(a.absmax[pt], a.log2_corner);
            unsigned char *const poison = poison_map(a, pt);
            const bool corner = q.y + y < bs && q.x + x < bs;
            unsigned char *mk =
                poison ? poison + static_cast<long long>(q.y) * a.width + q.x : nullptr;
            acc_add_checked(dn + (y * pitch + x), Gs[z * zs + y * rs + x] * numW,
                            corner ? scale_c : scale,
                            mk ? mk + static_cast<long long>(y) * a.width + x : nullptr);
            if (y == 0 && x == 0) {
                const float sd = (q.y == 0 && q.x == 0) ? scale_c : scale;
                if (mk == nullptr || fabsf(static_cast<float>(denW) * sd) < kFixedLimit)
                    weight_add(a.den[pt], a.width, q.y, q.x, denW, sd);
                else  // the block's weight reaches all of its pixels
                    for (int i = 0; i < bsq; ++i)
                        mk[static_cast<long long>(i / bs) * a.width + i % bs] = 1;
            }
        }
    }
    __syncwarp();
}

template <typename T, bool WIENER, int NPL, int BSC>
__device__ __forceinline__ void generic_tile_body(const StageArgs<T> &a, int tile, unsigned char *smem,
                                                  unsigned avail)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int bs = BSC > 0 ? BSC : a.block_size;
    const int right = a.width - bs, bottom = a.height - bs;

    Tile<T> t;
    int kx0, kx1, ky0, ky1;
    tile_window(a, tile, bs, t, kx0, kx1, ky0, ky1);
    const SmemPlan sp = plan_smem<T>(NPL, WIENER, a.ref_alias_src, a.region_h, a.region_pitch,
                                     a.span, nwarps, true, bs, a.group_size);
    if (sp.total > avail) {  // launched with less shared memory than the layout needs
        smem_shortfall(a);
        return;
    }
    carve_tile<T, WIENER, NPL>(a, sp, smem, t);
    unsigned *tasks = reinterpret_cast<unsigned *>(smem + sp.off_tasks);
    unsigned char *wbase = smem + sp.off_warps + sp.warp_bytes * warp;
    const bool strips = strip_blocks<T, BSC>(bs) && a.bm_step == 1;
    if (strips && warp == 0)
        build_tasks(tasks, reinterpret_cast<unsigned *>(wbase), a.span, t.pitch, lane);
    stage_tile<T, WIENER, NPL>(a, t);

    const int gvals = a.group_size * generic_block_stride(bs);
    T *Gs = reinterpret_cast<T *>(wbase);
    T *Gr = Gs + gvals;
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
        // BlockSize 8 with step 1: the register-resident kernel's strips of
        // four candidates; otherwise one lane per candidate
        const int n = match_any<T, BSC>(a, t, strips, j0, i0, lane, tasks, dist, refblk, heap, list,
                                        lkeys, n_cand, n_fix);
        n_sum += n;
        n_sq += static_cast<unsigned>(n * n);
        dump_group(a, ky, kx, n, lane, list, lkeys);
        if (!a.bm_only) {
#pragma unroll
            for (int p = 0; p < NPL; ++p)
                if (a.active & (1 << p))
                    filter_generic<T, WIENER, BSC>(a, t, p, list, n, lane, Gs, Gr, scale[p], n_bad,
                                              -1, check[p]);
        }
        __syncwarp();
    }
    flush_stats(a, lane, n_sum, n_sq, n_cand, n_fix, n_bad);
    if (a.bm_only) return;
    __syncthreads();
    flush_tile<T, NPL>(a, t);
}

// Three planes sharing the groups matched on plane 0, one plane at a time
// through a single plane's windows (as stage_tile_body_seq3): plane 0 matches
// and keeps each reference block's group list in shared memory, planes 1 and
// 2 re-stage their windows and filter with those lists.
template <typename T, bool WIENER, int BSC>
__device__ __forceinline__ void generic_tile_body_seq3(const StageArgs<T> &a, int tile,
                                                       unsigned char *smem, unsigned avail)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int bs = BSC > 0 ? BSC : a.block_size, GS = a.group_size;
    const int right = a.width - bs, bottom = a.height - bs;

    Tile<T> t;
    int kx0, kx1, ky0, ky1;
    tile_window(a, tile, bs, t, kx0, kx1, ky0, ky1);
    const SmemPlan sp = plan_smem<T>(3, WIENER, a.ref_alias_src, a.region_h, a.region_pitch,
                                     a.span, nwarps, true, bs, GS, a.tile_x * a.tile_y);
    if (sp.total > avail) {  // launched with less shared memory than the layout needs
        smem_shortfall(a);
        return;
    }
    carve_tile<T, WIENER, 1>(a, sp, smem, t);  // every plane goes through windows [0]
    // group lists: position (y - ry0) << 8 | (x - rx0), or 0xffff for a
    // (0, 0) block held outside the window; then one count byte per block
    unsigned short *gpos = reinterpret_cast<unsigned short *>(smem + sp.off_groups);
    unsigned char *gn = reinterpret_cast<unsigned char *>(gpos + a.tile_x * a.tile_y * GS);

    unsigned *tasks = reinterpret_cast<unsigned *>(smem + sp.off_tasks);
    unsigned char *wbase = smem + sp.off_warps + sp.warp_bytes * warp;
    const bool strips = strip_blocks<T, BSC>(bs) && a.bm_step == 1;
    if (strips && warp == 0)
        build_tasks(tasks, reinterpret_cast<unsigned *>(wbase), a.span, t.pitch, lane);
    T *Gs = reinterpret_cast<T *>(wbase);
    T *Gr = Gs + GS * generic_block_stride(bs);
    auto *dist = reinterpret_cast<typename DistBits<T>::type *>(wbase);
    T *refblk = reinterpret_cast<T *>(wbase + sp.off_ref);
    SortKey<T> *heap = reinterpret_cast<SortKey<T> *>(wbase + sp.off_heap);
    T *lkeys = reinterpret_cast<T *>(wbase + sp.off_keys);
    BlockPos *list = reinterpret_cast<BlockPos *>(wbase + sp.off_list);

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
                n = match_any<T, BSC>(a, t, strips, j0, i0, lane, tasks, dist, refblk, heap, list,
                                      lkeys, n_cand, n_fix);
                n_sum += n;
                n_sq += static_cast<unsigned>(n * n);
                dump_group(a, ky, kx, n, lane, list, lkeys);
                if (lane == 0) gn[r] = static_cast<unsigned char>(n);
                for (int k = lane; k < n; k += kWarp) {
                    const BlockPos q = list[k];
                    const bool outside = q.y == 0 && q.x == 0 && !t.origin_inside;
                    gpos[r * GS + k] = outside ? 0xffff
                                               : static_cast<unsigned short>(
                                                     ((q.y - t.ry0) << 8) | (q.x - t.rx0));
                }
            } else {
                n = gn[r];
                for (int k = lane; k < n; k += kWarp) {
                    const unsigned v = gpos[r * GS + k];
                    list[k] = v == 0xffffu ? BlockPos{0, 0}
                                           : BlockPos{t.ry0 + static_cast<int>(v >> 8),
                                                      t.rx0 + static_cast<int>(v & 0xffu)};
                }
            }
            __syncwarp();
            if (filt)
                filter_generic<T, WIENER, BSC>(a, t, 0, list, n, lane, Gs, Gr, scale, n_bad, c, check);
            __syncwarp();
        }
        __syncthreads();
        if (filt) flush_plane<T>(a, t, c);
        __syncthreads();  // the windows are re-staged for the next plane
    }
    flush_stats(a, lane, n_sum, n_sq, n_cand, n_fix, n_bad);
}

// BSC: BlockSize 8 (groups of up to 32) and 11 in FP32 have kernels of their own,
// so that neither's registers and code are the other's: 11 x 11 groups of 32
// leave shared memory for five warps, and that kernel takes up to 255 registers
// a thread. 0 is any size. Against one kernel for all (168 registers, 240 bytes
// of them spilled): np's final stage on 1283 x 717 2.05 -> 1.93 ms, vn's (11 x 11,
// with strips) on 960 x 540 1.47 -> 1.13 ms.
__host__ __device__ constexpr int generic_max_warps(int elem_bytes, int bsc)
{
    return elem_bytes == 8 || bsc == 11 ? 8 : 12;
}
__host__ __device__ constexpr int generic_size_class(int elem_bytes, int bs)
{
    return elem_bytes == 4 && (bs == kBS || bs == 11) ? bs : 0;
}

template <typename T, bool WIENER, int NPL, int BSC>
__global__ void __launch_bounds__(generic_max_warps(sizeof(T), BSC) * kWarp, 1)
    generic_stage_kernel(const StageArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if constexpr (NPL == 3) generic_tile_body_seq3<T, WIENER, BSC>(a, blockIdx.x, smem, dynamic_smem_bytes());
    else generic_tile_body<T, WIENER, NPL, BSC>(a, blockIdx.x, smem, dynamic_smem_bytes());
}

}  // namespace bm3d
