// C ABI of the B200 BM3D path (declared in include/bm3d_b200.h): parameter
// mirroring, per-call constant setup, context scratch and kernel launches.
// The integer / Frame entry points are in bm3d_capi_convert.cu, the batches
// in bm3d_capi_batch.cu.
#include "bm3d_capi_internal.h"

#include <atomic>
#include <type_traits>

static thread_local std::string g_create_error;

static void drain_timing(bm3d_ctx *ctx)
{
    for (int k = 0; k < 2; ++k) {
        for (auto &ev : ctx->pending[k]) {
            float ms = 0;
            if (cudaEventSynchronize(ev.second) == cudaSuccess &&
                cudaEventElapsedTime(&ms, ev.first, ev.second) == cudaSuccess) {
                ctx->time_ms[k] += ms;
                ctx->launches[k] += 1;
            }
            cudaEventDestroy(ev.first);
            cudaEventDestroy(ev.second);
        }
        ctx->pending[k].clear();
    }
}

int bm3d::cuda_fail(bm3d_ctx *ctx, cudaError_t e, const char *what)
{
    char buf[256];
    std::snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    if (ctx) ctx->err = buf;
    else g_create_error = buf;
    return e == cudaErrorMemoryAllocation ? BM3D_ERR_NOMEM : BM3D_ERR_CUDA;
}

// Allocations still to fail on purpose (bm3d_inject_alloc_failures), and those
// that succeed before them.
static std::atomic<int> g_fail_allocs{0}, g_skip_allocs{0};

extern "C" int bm3d_inject_alloc_failures(int count) { return bm3d_inject_alloc_failures_after(0, count); }

extern "C" int bm3d_inject_alloc_failures_after(int skip, int count)
{
    if (skip < 0 || count < 0) return BM3D_ERR_INVALID;
    g_skip_allocs.store(skip);
    g_fail_allocs.store(count);
    return BM3D_OK;
}

// Takes one from a counter above zero.
static bool take_one(std::atomic<int> &counter)
{
    for (int left = counter.load(); left > 0; left = counter.load())
        if (counter.compare_exchange_weak(left, left - 1)) return true;
    return false;
}

// Pilot launches until one is reported as failed; negative: none is.
static std::atomic<int> g_fail_launch{-1};

extern "C" int bm3d_inject_launch_failure_after(int skip)
{
    g_fail_launch.store(skip < 0 ? -1 : skip);
    return BM3D_OK;
}

cudaError_t bm3d::launch_error()
{
    const cudaError_t e = cudaGetLastError();
    if (g_fail_launch.load() < 0 || g_fail_launch.fetch_sub(1) != 0) return e;
    return cudaErrorInvalidConfiguration;
}

int bm3d::ensure(bm3d_ctx *ctx, DevBuf &b, size_t bytes)
{
    if (b.bytes >= bytes) return BM3D_OK;
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
    if (!take_one(g_skip_allocs) && take_one(g_fail_allocs))
        return cuda_fail(ctx, cudaErrorMemoryAllocation, "cudaMalloc (injected failure)");
    const cudaError_t e = cudaMalloc(&b.ptr, bytes);
    if (e != cudaSuccess) {
        b.ptr = nullptr;
        cudaGetLastError();  // the next launch check is not about this
        return cuda_fail(ctx, e, "cudaMalloc");
    }
    b.bytes = bytes;
    return BM3D_OK;
}

int bm3d::ensure_optional(bm3d_ctx *ctx, DevBuf &b, size_t bytes, cudaStream_t s, bool &got)
{
    got = b.bytes >= bytes;
    if (got) return BM3D_OK;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (s != nullptr) CK(ctx, cudaStreamIsCapturing(s, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return BM3D_OK;  // an allocation would end it
    const std::string err = ctx->err;
    const int rc = ensure(ctx, b, bytes);
    got = rc == BM3D_OK;
    if (rc != BM3D_ERR_NOMEM) return rc;
    ctx->err = err;
    return BM3D_OK;
}

cudaError_t bm3d::raise_smem_limit(const void *kern, size_t bytes)
{
    static std::mutex mu;  // read-compare-set must not interleave across threads
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return e;
    if (fa.maxDynamicSharedSizeBytes >= 0 &&
        static_cast<size_t>(fa.maxDynamicSharedSizeBytes) >= bytes)
        return cudaSuccess;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(bytes));
}

#define BM3D_DECLARE_UNIT(name) cudaError_t bm3d_upload_dct_tables_##name(const bm3d::DctTables &);
BM3D_KERNEL_UNITS(BM3D_DECLARE_UNIT)
#undef BM3D_DECLARE_UNIT

namespace bm3d {

cudaError_t upload_dct_tables_all(const DctTables &t)
{
    cudaError_t e = cudaSuccess;
#define BM3D_UPLOAD_UNIT(name) \
    if ((e = bm3d_upload_dct_tables_##name(t)) != cudaSuccess) return e;
    BM3D_KERNEL_UNITS(BM3D_UPLOAD_UNIT)
#undef BM3D_UPLOAD_UNIT
    return e;
}

}  // namespace bm3d

// Cosine matrices in long double, rounded once to each precision; length n
// starts at (n-1) n (2n-1) / 6.
static void make_dct_tables(float *ff, float *fi, double *df, double *di)
{
    const long double pi = 3.141592653589793238462643383279502884L;
    int o = 0;
    for (int n = 1; n <= 16; ++n) {
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) {
                const long double cf = 2.0L * cosl(pi * (2 * j + 1) * k / (2.0L * n));
                const long double ci = j == 0 ? 1.0L : 2.0L * cosl(pi * j * (2 * k + 1) / (2.0L * n));
                ff[o + k * n + j] = static_cast<float>(cf);
                fi[o + k * n + j] = static_cast<float>(ci);
                df[o + k * n + j] = static_cast<double>(cf);
                di[o + k * n + j] = static_cast<double>(ci);
            }
        o += n * n;
    }
}

static bm3d::DctTables g_tab;
static std::once_flag g_tab_once;

static void init_dct_tables()
{
    make_dct_tables(g_tab.fwd_f, g_tab.inv_f, g_tab.fwd_d, g_tab.inv_d);
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int k = 0; k < 11; ++k)
        for (int j = 0; j < 11; ++j) {
            g_tab.d11_fwd[k * 11 + j] = static_cast<float>(2.0L * cosl(pi * (2 * j + 1) * k / 22.0L));
            g_tab.d11_inv[k * 11 + j] =
                static_cast<float>(j == 0 ? 1.0L : 2.0L * cosl(pi * j * (2 * k + 1) / 22.0L));
        }
    // column-major, 16 rows, zero past row n: the same FP32 values
    for (int n = 1; n <= 15; ++n) {
        if (n == 8) continue;
        const int src = (n - 1) * n * (2 * n - 1) / 6, dst = bm3d::pad_table_offset(n);
        for (int j = 0; j < n; ++j)
            for (int k = 0; k < 16; ++k) {
                g_tab.pad_fwd[dst + 16 * j + k] = k < n ? g_tab.fwd_f[src + k * n + j] : 0.0f;
                g_tab.pad_inv[dst + 16 * j + k] = k < n ? g_tab.inv_f[src + k * n + j] : 0.0f;
            }
    }
}

static cudaError_t upload_dct_tables()
{
    std::call_once(g_tab_once, init_dct_tables);
    return upload_dct_tables_all(g_tab);
}

extern "C" int bm3d_ctx_create(bm3d_ctx **out, int device)
{
    if (!out) return BM3D_ERR_INVALID;
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceCount");
    if (device < 0 || device >= count) {
        g_create_error = "bm3d_ctx_create: no such CUDA device";
        return BM3D_ERR_CUDA;
    }
    cudaDeviceProp prop;
    e = cudaGetDeviceProperties(&prop, device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceProperties");
    if (prop.major < 10) {
        g_create_error = "bm3d_ctx_create: this build targets sm_100a (B200)";
        return BM3D_ERR_CUDA;
    }
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaSetDevice");
    bm3d_ctx *ctx = new bm3d_ctx;
    ctx->device = device;
    ctx->sm_count = prop.multiProcessorCount;
    ctx->smem_optin = prop.sharedMemPerBlockOptin;
    e = upload_dct_tables();
    if (e != cudaSuccess) {
        delete ctx;
        return cuda_fail(nullptr, e, "upload_dct_tables");
    }
    e = cudaMalloc(&ctx->head, kHeadBytes);
    if (e != cudaSuccess) {
        delete ctx;
        return cuda_fail(nullptr, e, "cudaMalloc(head)");
    }
    cudaMemset(ctx->head, 0, kHeadBytes);
    ctx->absmax = reinterpret_cast<float *>(ctx->head);
    ctx->nonfinite = reinterpret_cast<unsigned *>(ctx->head) + kMaxPlanes;
    ctx->nonfinite_next = ctx->nonfinite + kMaxPlanes;
    ctx->stats = reinterpret_cast<unsigned long long *>(ctx->head + kHeadStats);
    // cosine matrices of lengths 1..32 for the generic path
    {
        std::vector<float> tf(2 * kDctTableSize + 2 * kPad32Table, 0.0f);
        std::vector<double> td(2 * kDctTableSize);
        const long double pi = 3.141592653589793238462643383279502884L;
        for (int n = 1; n <= kGSTab; ++n) {
            const int o = dct_table_offset(n);
            for (int k = 0; k < n; ++k)
                for (int j = 0; j < n; ++j) {
                    const long double cf = 2.0L * cosl(pi * (2 * j + 1) * k / (2.0L * n));
                    const long double ci = j == 0 ? 1.0L : 2.0L * cosl(pi * j * (2 * k + 1) / (2.0L * n));
                    tf[o + k * n + j] = static_cast<float>(cf);
                    tf[kDctTableSize + o + k * n + j] = static_cast<float>(ci);
                    td[o + k * n + j] = static_cast<double>(cf);
                    td[kDctTableSize + o + k * n + j] = static_cast<double>(ci);
                }
        }
        for (int n = 1; n < kGSTab; ++n) {  // the same, column by column in 32 rows
            const int o = dct_table_offset(n), q = 2 * kDctTableSize + pad32_offset(n);
            for (int k = 0; k < n; ++k)
                for (int j = 0; j < n; ++j) {
                    tf[q + 32 * j + k] = tf[o + k * n + j];
                    tf[q + kPad32Table + 32 * j + k] = tf[kDctTableSize + o + k * n + j];
                }
        }
        e = cudaMalloc(&ctx->gtab_f, tf.size() * sizeof(float));
        if (e == cudaSuccess) e = cudaMalloc(&ctx->gtab_d, td.size() * sizeof(double));
        if (e == cudaSuccess)
            e = cudaMemcpy(ctx->gtab_f, tf.data(), tf.size() * sizeof(float), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
            e = cudaMemcpy(ctx->gtab_d, td.data(), td.size() * sizeof(double), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(ctx->head);
            cudaFree(ctx->gtab_f);
            cudaFree(ctx->gtab_d);
            delete ctx;
            return cuda_fail(nullptr, e, "generic cosine tables");
        }
    }
    *out = ctx;
    return BM3D_OK;
}

extern "C" void bm3d_ctx_destroy(bm3d_ctx *ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    auto fr = [](DevBuf &b) {
        if (b.ptr) cudaFree(b.ptr);
        b.ptr = nullptr;
    };
    for (auto &b : ctx->acc) fr(b);
    for (auto &b : ctx->den_next) fr(b);
    for (auto &b : ctx->basic) fr(b);
    for (auto &b : ctx->stage_in) fr(b);
    for (auto &b : ctx->stage_ref) fr(b);
    for (auto &b : ctx->stage_out) fr(b);
    for (auto &b : ctx->groups) fr(b);
    for (auto &b : ctx->conv) fr(b);
    for (auto &b : ctx->ints) fr(b);
    for (auto &b : ctx->poison) fr(b);
    for (auto &sl : ctx->pipe) {
        fr(sl.in);
        fr(sl.out);
        for (cudaEvent_t e : {sl.in_ready, sl.computed, sl.drained})
            if (e) cudaEventDestroy(e);
    }
    if (ctx->up) cudaStreamDestroy(ctx->up);
    if (ctx->down) cudaStreamDestroy(ctx->down);
    if (ctx->head) cudaFree(ctx->head);
    if (ctx->gtab_f) cudaFree(ctx->gtab_f);
    if (ctx->gtab_d) cudaFree(ctx->gtab_d);
    drain_timing(ctx);
    delete ctx;
}

extern "C" const char *bm3d_last_error(const bm3d_ctx *ctx)
{
    if (ctx) return ctx->err.c_str();
    return g_create_error.c_str();
}

extern "C" int bm3d_set_tiling(bm3d_ctx *ctx, int tile_x, int tile_y, int warps)
{
    if (!ctx || tile_x < 0 || tile_y < 0 || warps < 0 || warps > 16) return BM3D_ERR_INVALID;
    if (tile_x || tile_y || warps) ctx->tiling_set = true;
    if (tile_x) ctx->tile_x = tile_x;
    if (tile_y) ctx->tile_y = tile_y;
    if (warps) ctx->warps = warps;
    return BM3D_OK;
}

// ---------------------------------------------------------------------------
// Parameters: the reference's profile constructors (include/BM3D.h:27-151).

static bool known_profile(const std::string &p)
{
    return p == "fast" || p == "lc" || p == "np" || p == "high" || p == "vn";
}

extern "C" int bm3d_stage_params_thmse_default(const char *profile, int wiener,
                                               bm3d_stage_params *p)
{
    if (!profile || !p || !known_profile(profile)) return BM3D_ERR_INVALID;
    const std::string prof(profile);
    if (!wiener) p->thMSE = prof == "vn" ? 1000 + p->sigma[0] * 150 : 400 + p->sigma[0] * 80;
    else p->thMSE = prof == "vn" ? 400 + p->sigma[0] * 40 : 200 + p->sigma[0] * 10;
    return BM3D_OK;
}

extern "C" int bm3d_stage_params_default(const char *profile, int wiener, const double sigma[3],
                                         bm3d_stage_params *out)
{
    if (!profile || !out || !known_profile(profile)) return BM3D_ERR_INVALID;
    const std::string prof(profile);
    bm3d_stage_params p;
    p.block_size = 8;
    p.bm_range = (prof == "fast" || prof == "lc") ? 9 : 16;
    p.bm_step = 1;
    if (!wiener) {
        p.block_step = 4;
        p.group_size = 16;
        p.lambda = 2.7;
        if (prof == "fast") p.block_step = 8;
        else if (prof == "lc") p.block_step = 6;
        else if (prof == "high") p.block_step = 3;
        else if (prof == "vn") {
            p.block_step = 4;
            p.group_size = 32;
            p.lambda = 2.8;
        }
    } else {
        p.block_step = 3;
        p.group_size = 32;
        p.lambda = 0;
        if (prof == "fast") {
            p.block_step = 7;
            p.group_size = 16;
        } else if (prof == "lc") {
            p.block_step = 5;
            p.group_size = 16;
        } else if (prof == "high") {
            p.block_step = 2;
        } else if (prof == "vn") {
            p.block_size = 11;
            p.block_step = 6;
        }
    }
    for (int i = 0; i < 3; ++i) p.sigma[i] = sigma ? sigma[i] : 10.0;
    bm3d_stage_params_thmse_default(profile, wiener, &p);
    *out = p;
    return BM3D_OK;
}

extern "C" long long bm3d_ref_block_count(const bm3d_stage_params *p, int width, int height)
{
    if (!p || p->block_size <= 0 || p->block_step <= 0 || width < p->block_size ||
        height < p->block_size)
        return -1;
    return static_cast<long long>(ref_count(width - p->block_size, p->block_step)) *
           ref_count(height - p->block_size, p->block_step);
}

// ---------------------------------------------------------------------------
// Stage setup: BM3D_Base ctor (include/BM3D.h:237-259) and BM3D_FilterData
// ctor (source/BM3D.cpp:9-73), evaluated in double exactly as the reference.

static void opp_norms(double norm[3])
{
    const double Yr = static_cast<double>(1.0L / 3.0L), Yg = Yr, Yb = Yr;
    const double Ur = static_cast<double>(1.0L / 2.0L), Ug = 0.0, Ub = static_cast<double>(-1.0L / 2.0L);
    const double Vr = static_cast<double>(1.0L / 4.0L), Vg = static_cast<double>(-1.0L / 2.0L),
                 Vb = static_cast<double>(1.0L / 4.0L);
    norm[0] = std::sqrt(Yr * Yr + Yg * Yg + Yb * Yb);
    norm[1] = std::sqrt(Ur * Ur + Ug * Ug + Ub * Ub);
    norm[2] = std::sqrt(Vr * Vr + Vg * Vg + Vb * Vb);
}

// The register-resident kernel covers BlockSize 8 with GroupSize <= 16 (the
// "fast" and "lc" profiles); everything else up to BlockSize 16 and GroupSize
// 32 runs on the generic kernel.
static bool fast_path(const bm3d_stage_params *p)
{
    return p->block_size == kBS && p->group_size <= kGSMax;
}

Guard bm3d::check_params(const bm3d_stage_params *p, int nplanes)
{
    if (!p) return Guard::Invalid;
    double norm[3];
    opp_norms(norm);
    const double thMSE = p->thMSE * norm[0];
    const bool sig = nplanes == 3 ? (p->sigma[0] <= 0 && p->sigma[1] <= 0 && p->sigma[2] <= 0)
                                  : (p->sigma[0] <= 0);
    if (sig || p->group_size == 0 || p->block_size <= 0 || p->bm_range <= 0 ||
        p->bm_range < p->bm_step || thMSE <= 0)
        return Guard::Copy;
    if (p->group_size < 0 || p->block_step <= 0 || p->bm_step <= 0) return Guard::Invalid;
    if (p->block_size > kBSMax || p->group_size > kGSTab) return Guard::Unsupported;
    return Guard::Run;
}

// The distances whose keys (key_from_dist) are normal, as bits: the least and the
// greatest that approximate matching may rank (DistBits, select_once); keys grow
// with the distance. None: low above high.
static void near_range(double mul, unsigned &low, unsigned &high)
{
    using DB = DistBits<float>;
    auto value = [](unsigned bits) {
        float f;
        std::memcpy(&f, &bits, sizeof(f));
        return f;
    };
    auto first = [&](auto reached) {  // the first distance that `reached` holds for
        unsigned lo = 0, hi = 0x7f800000u;
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo) / 2;
            if (reached(static_cast<float>(static_cast<double>(value(mid)) * mul))) hi = mid;
            else lo = mid + 1;
        }
        return lo;
    };
    low = std::max(DB::kTiny, first([&](float key) { return key >= value(DB::kLow); }));
    high = first([&](float key) { return key > value(DB::kHigh); }) - 1;
}

template <typename T>
void bm3d::fill_tables(StageArgs<T> &a, const bm3d_stage_params *p, bool wiener, int nplanes,
                       double value_range)
{
    double norm[3];
    opp_norms(norm);
    const double thMSE = p->thMSE * norm[0];
    const int GS = p->group_size, BS = p->block_size;
    a.active = 0;
    for (int c = 0; c < nplanes; ++c) {
        if (!(p->sigma[c] > 0)) continue;
        a.active |= 1 << c;
        const double sigma = p->sigma[c] / double(255) * norm[c];
        for (int i = 1; i <= GS; ++i) {
            const double finalAMP = 2 * i * 2 * BS * 2 * BS;
            const double forwardAMP = std::sqrt(finalAMP);
            a.wss[c][i - 1] = static_cast<T>(sigma * forwardAMP * sigma * forwardAMP);
            const double thrBase = sigma * p->lambda * forwardAMP;
            a.thr[c][i - 1][0] = static_cast<T>(thrBase);
            a.thr[c][i - 1][1] = static_cast<T>(thrBase * std::sqrt(double(2)));
            a.thr[c][i - 1][2] = static_cast<T>(thrBase * double(2));
            a.thr[c][i - 1][3] = static_cast<T>(thrBase * std::sqrt(double(8)));
        }
    }
    if (nplanes == 1) a.active = 1;
    for (int i = 1; i <= GS; ++i) a.finalAMP[i - 1] = 2 * i * 2 * BS * 2 * BS;
    (void)wiener;
    // Block::BlockMatchingMulti (include/Block.h:582-584); the plane range is
    // an FLType, promoted to double in the product.
    const T range = static_cast<T>(value_range);
    const double MSE2SSE = static_cast<double>(BS * BS) * range * range / double(255 * 255);
    a.distMul = double(1) / MSE2SSE;
    a.thSSE = static_cast<T>(thMSE * MSE2SSE);
    near_range(a.distMul, a.near_low, a.near_high);
    a.match = (GS == 1 || thMSE <= 0) ? 0 : 1;
}

template <typename T, bool W, int NPL, int KS>
static int launch_one(bm3d_ctx *ctx, StageArgs<T> &a, cudaStream_t s, int warps)
{
    const void *kern = stage_kernel_fn<T, W, NPL, KS>();
    const SmemPlan sp =
        plan_smem<T>(NPL, W, a.ref_alias_src, a.region_h, a.region_pitch, a.span, warps,
                     false, kBS, kGSMax, a.tile_x * a.tile_y);
    CK(ctx, raise_smem_limit(kern, sp.total));
    const int grid = a.tiles_x * ((a.ny + a.tile_y - 1) / a.tile_y);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (ctx->timing && !a.bm_only) {
        CK(ctx, cudaEventCreate(&e0));
        CK(ctx, cudaEventCreate(&e1));
        CK(ctx, cudaEventRecord(e0, s));
    }
    void *args[] = {&a};
    CK(ctx, cudaLaunchKernel(kern, dim3(grid), dim3(warps * kWarp), args, sp.total, s));
    if (e0) {
        CK(ctx, cudaEventRecord(e1, s));
        ctx->pending[W ? 1 : 0].emplace_back(e0, e1);
    }
    return BM3D_OK;
}

template <typename T, bool W, int NPL>
static int launch_ks(bm3d_ctx *ctx, StageArgs<T> &a, cudaStream_t s, int warps)
{
    if (a.bm_step == 1) return launch_one<T, W, NPL, 4>(ctx, a, s, warps);
    return launch_one<T, W, NPL, 1>(ctx, a, s, warps);
}

template <typename T, bool W, int NPL>
static int launch_generic(bm3d_ctx *ctx, StageArgs<T> &a, cudaStream_t s, int warps)
{
    const void *kern = generic_kernel_fn<T, W, NPL, 0>();
    if constexpr (sizeof(T) == 4) {
        const int bsc = generic_size_class(sizeof(T), a.block_size);
        if (bsc == kBS) kern = generic_kernel_fn<T, W, NPL, kBS>();
        else if (bsc == 11) kern = generic_kernel_fn<T, W, NPL, 11>();
    }
    const SmemPlan sp = plan_smem<T>(NPL, W, a.ref_alias_src, a.region_h, a.region_pitch,
                                     a.span, warps, true, a.block_size, a.group_size,
                                     a.tile_x * a.tile_y);
    CK(ctx, raise_smem_limit(kern, sp.total));
    const int grid = a.tiles_x * ((a.ny + a.tile_y - 1) / a.tile_y);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (ctx->timing && !a.bm_only) {
        CK(ctx, cudaEventCreate(&e0));
        CK(ctx, cudaEventCreate(&e1));
        CK(ctx, cudaEventRecord(e0, s));
    }
    void *args[] = {&a};
    CK(ctx, cudaLaunchKernel(kern, dim3(grid), dim3(warps * kWarp), args, sp.total, s));
    if (e0) {
        CK(ctx, cudaEventRecord(e1, s));
        ctx->pending[W ? 1 : 0].emplace_back(e0, e1);
    }
    return BM3D_OK;
}

bool bm3d::fast_args(int block_size, int group_size)
{
    return block_size == kBS && group_size <= kGSMax;
}

template <typename T>
static int launch_stage(bm3d_ctx *ctx, StageArgs<T> &a, bool wiener, int nplanes, cudaStream_t s,
                        int warps)
{
    if (!fast_args(a.block_size, a.group_size)) {
        if (nplanes == 1)
            return wiener ? launch_generic<T, true, 1>(ctx, a, s, warps)
                          : launch_generic<T, false, 1>(ctx, a, s, warps);
        return wiener ? launch_generic<T, true, 3>(ctx, a, s, warps)
                      : launch_generic<T, false, 3>(ctx, a, s, warps);
    }
    if (nplanes == 1)
        return wiener ? launch_ks<T, true, 1>(ctx, a, s, warps) : launch_ks<T, false, 1>(ctx, a, s, warps);
    return wiener ? launch_ks<T, true, 3>(ctx, a, s, warps) : launch_ks<T, false, 3>(ctx, a, s, warps);
}

template <typename T> struct GenericTables;
template <> struct GenericTables<float> {
    static const float *fwd(const bm3d_ctx *c) { return c->gtab_f; }
    static const float *inv(const bm3d_ctx *c) { return c->gtab_f ? c->gtab_f + kDctTableSize : nullptr; }
};
template <> struct GenericTables<double> {
    static const double *fwd(const bm3d_ctx *c) { return c->gtab_d; }
    static const double *inv(const bm3d_ctx *c) { return c->gtab_d ? c->gtab_d + kDctTableSize : nullptr; }
};

// Tile shapes offered to a stage: reference blocks per tile (tx x ty, a multiple
// of the warps, so no warp idles in a tile's last round) and warps per CTA.
struct TileShape {
    int tx, ty, warps;
};

// Window geometry and shared memory of a stage at one tile shape.
template <typename T>
static SmemPlan plan_tile(StageArgs<T> &a, const bm3d_stage_params *p, bool wiener, int nplanes,
                          const TileShape &t)
{
    const int BS = p->block_size;
    const int reach = a.match ? a.range : 0;
    a.region_w = std::min(a.width, (t.tx - 1) * a.step + 2 * reach + BS);
    a.region_h = std::min(a.height, (t.ty - 1) * a.step + 2 * reach + BS);
    a.region_pitch = window_pitch(a.region_w);
    a.tile_x = std::min(t.tx, a.nx);
    a.tile_y = std::min(t.ty, a.ny);
    a.tiles_x = (a.nx + a.tile_x - 1) / a.tile_x;
    return plan_smem<T>(nplanes, wiener, a.ref_alias_src, a.region_h, a.region_pitch, a.span, t.warps,
                        !fast_args(BS, p->group_size), BS, p->group_size, a.tile_x * a.tile_y);
}

// Whether a stage is over the limit on window and list sizes (stage_limit_bytes)
// at its smallest tile.
template <typename T>
static bool over_limit(const bm3d_ctx *ctx, const StageArgs<T> &a, const bm3d_stage_params *p, bool wiener,
                       int nplanes)
{
    const int reach = a.match ? a.range : 0, BS = p->block_size;
    return stage_limit_bytes<T>(nplanes, wiener, a.ref_alias_src, std::min(a.height, 2 * reach + BS),
                                std::min(a.width, 2 * reach + BS), a.span,
                                !fast_args(BS, p->group_size), BS, p->group_size, 1) > ctx->smem_optin;
}

// Predicted time of a stage at one tile shape (microseconds; only the order
// matters). Fast profile: a warp takes 8.5 us for a reference block when its SM
// runs few warps and 12 us with 16; about a third of it is matching, the rest
// follows the group's size. A tile adds staging, flushing and the wait for its last
// warp: about 10 us where other CTAs of the SM overlap it, or by its window in the
// generic kernel, whose 12 warps fill an SM. CTAs run in waves, whose rounding up
// fades once there are several: the sooner in the generic kernels, where a CTA of
// few warps starts as soon as another of its SM ends. Blocks under 8 x 8 take no
// less time than those of 8 x 8. Measured at 64 x 64 .. 3840 x 2160, one shape for all
// sizes (8 x 8, 16 warps) against the shapes this picks, basic / final stage:
// 64 x 64 60 / 67 -> 20 / 23 us, 512 x 512 72 / 88 -> 49 / 65 us, 1280 x 720
// 128 / 197 -> 113 / 177 us, 1920 x 1080 245 / 343 -> 225 / 329 us; generic kernel
// (6 x 4, 12 warps before) np final 300 x 200 212 -> 171 us, vn basic 960 x 540
// 672 -> 650 us.
template <typename T>
static double tile_cost(const bm3d_ctx *ctx, const StageArgs<T> &a, const SmemPlan &sp,
                        const TileShape &t, int nplanes, bool generic)
{
    const size_t sm_smem = ctx->smem_optin + 1024;  // an SM's share; 1 KB of it per CTA is reserved
    const int regs = sizeof(T) == 8 || (generic && a.block_size == 11) ? 256 : generic ? 168 : 128;
    const int by_smem = static_cast<int>(sm_smem / (sp.total + 1024));
    const int by_regs = 65536 / (t.warps * kWarp * regs);
    const int per_sm = std::max(1, std::min(by_smem, by_regs));
    const double tiles = static_cast<double>(a.tiles_x) * ((a.ny + a.tile_y - 1) / a.tile_y);
    const double share = tiles / ctx->sm_count;  // tiles per SM
    const int ctas = std::min(per_sm, std::max(1, static_cast<int>(std::ceil(share))));
    const double px = std::max(1.0, a.block_size * a.block_size / 64.0);
    const double work = px * (0.65 * std::max(16, a.group_size) / 16.0 +
                              0.35 * a.span * a.span / 361.0) * (nplanes == 3 ? 1.9 : 1.0);
    const double round = (8.5 + 0.22 * ctas * t.warps) * work;
    const int rounds = (a.tile_x * a.tile_y + t.warps - 1) / t.warps;
    const double x = share / per_sm;
    const double tail = generic_size_class(sizeof(T), a.block_size) != 0 ? 0.15 : 0.3;  // of a wave
    const double waves = generic && per_sm > 1 ? std::max(1.0, x + tail) : x < 4.0 ? std::ceil(x) : x + 0.5;
    const double window = static_cast<double>(a.region_w) * a.region_h * ctas;
    const double edge = generic ? 3.0 + 1.05e-3 * window : 8.0 + rounds + 0.1 * t.warps;
    return waves * (rounds * round + edge * nplanes);
}

// Geometry, tiling and shared-memory fit.
template <typename T>
static int plan_geometry(bm3d_ctx *ctx, StageArgs<T> &a, const bm3d_stage_params *p, bool wiener,
                         int nplanes, int width, int height, int &warps)
{
    const int BS = p->block_size;
    const bool generic = !fast_args(BS, p->group_size);
    a.width = width;
    a.height = height;
    a.block_size = BS;
    a.step = p->block_step;
    a.group_size = p->group_size;
    a.bm_step = p->bm_step;
    a.range = p->bm_range / p->bm_step * p->bm_step;
    a.nx = ref_count(width - BS, a.step);
    a.ny = ref_count(height - BS, a.step);
    a.span = 2 * (a.range / a.bm_step) + 1;
    if (over_limit(ctx, a, p, wiener, nplanes)) {
        ctx->err = "stage does not fit in shared memory";
        return BM3D_ERR_UNSUPPORTED;
    }
    if (!a.match) a.span = 1;  // no search list (past the limit, which counts one)
    // The launch bounds (register-resident 512 threads in FP32, 256 in FP64;
    // generic 384, and 256 in FP64 and for BlockSize 11) limit the warps; the
    // small shapes are for windows that leave no room for more.
    static const TileShape fast[] = {{2, 2, 4}, {4, 2, 8}, {4, 4, 8}, {4, 8, 8}, {6, 4, 8}, {8, 8, 16}};
    static const TileShape gen[] = {{6, 6, 12}, {6, 4, 12}, {4, 3, 12}, {3, 2, 6}, {2, 2, 4},
                                    {4, 4, 8},  {4, 2, 8},  {5, 2, 5},  {4, 4, 4}};
    static const TileShape gen_tiny[] = {{6, 4, 12}, {2, 2, 4}};
    static const TileShape gen_small[] = {{2, 2, 4}, {2, 2, 2}, {1, 1, 2}, {1, 1, 1}};
    const int max_warps = generic ? generic_max_warps(sizeof(T), generic_size_class(sizeof(T), BS))
                                  : stage_max_warps<T>();
    if (generic || !ctx->tiling_set) {
        TileShape best{0, 0, 0};
        double least = 1e300, within = 0;
        // The model is made for 8 x 8 and (FP32) 11 x 11 blocks in FP32; elsewhere the
        // smallest tile not much above the least cost is taken, because its warps wait
        // least for one another where groups differ in size. FP32 blocks under 8 x 8
        // choose between two shapes that fill the registers with 12 warps (4 x 4 tiles
        // on 4 warps, which cost least, took 2486 us where 6 x 4 on 12 took 1876 and
        // 2 x 2 on 4 2225: 2 x 2 blocks, groups of 32, noise, 320 x 256). Over 198 stages
        // of BlockSize 2 to 16 on 64 x 64, 333 x 200 and 700 x 540, noise and computer
        // graphics, the geometric mean over the best of the shapes is 1.02 (FP32 under
        // 8 x 8; by the least cost 1.12), 1.01 (over; 1.06) and 1.02 (FP64; 1.07).
        const bool plain = generic && generic_size_class(sizeof(T), BS) == 0;
        const bool small = plain && sizeof(T) == 4 && BS < kBS;
        // (FP32 8 x 8 blocks lose by 4 x 4 tiles on 4 warps: four rounds, whose spread
        // nothing evens out; np final stage 700 x 540, computer graphics, up to 1.5 times)
        const bool no_rounds = generic && !plain && BS == kBS;
        auto offer = [&](const TileShape &t) {
            if (t.warps > max_warps || (no_rounds && t.tx * t.ty == 4 * t.warps)) return;
            const SmemPlan sp = plan_tile(a, p, wiener, nplanes, t);
            if (sp.total > ctx->smem_optin) return;
            const double c = tile_cost(ctx, a, sp, t, nplanes, generic);
            const int size = t.tx * t.ty - best.tx * best.ty;
            if (within > 0 ? c <= within && (best.warps == 0 || size < 0 || (size == 0 && c < least)) : c < least) {
                least = c;
                best = t;
            }
        };
        auto offer_all = [&] {
            if (!generic) for (const TileShape &t : fast) offer(t);
            else if (small) for (const TileShape &t : gen_tiny) offer(t);
            else for (const TileShape &t : gen) offer(t);
        };
        offer_all();
        if (plain && best.warps != 0) {
            within = (small ? 1.06 : 1.2) * least;
            best = TileShape{0, 0, 0};
            offer_all();
        }
        if (generic && best.warps == 0)
            for (const TileShape &t : gen_small)
                if (best.warps == 0) offer(t);
        if (best.warps != 0) {
            plan_tile(a, p, wiener, nplanes, best);
            warps = best.warps;
            return BM3D_OK;
        }
        if (generic) {
            ctx->err = "stage does not fit in shared memory";
            return BM3D_ERR_UNSUPPORTED;
        }
    }
    // a set shape, or none of the usual ones fits: the largest that does
    TileShape t{ctx->tile_x, ctx->tile_y, std::min(ctx->warps, max_warps)};
    for (;;) {
        if (plan_tile(a, p, wiener, nplanes, t).total <= ctx->smem_optin) break;
        if (t.warps > 8) {
            t.warps /= 2;
        } else if (t.ty > 1 && t.ty >= t.tx) {
            --t.ty;
        } else if (t.tx > 1) {
            --t.tx;
        } else if (t.warps > 1) {
            t.warps /= 2;
        } else {
            ctx->err = "stage does not fit in shared memory";
            return BM3D_ERR_UNSUPPORTED;
        }
    }
    warps = t.warps;
    return BM3D_OK;
}

// How a stage call relates to another one: a basic stage that also prepares
// the final stage that follows on the same planes, and that final stage
// (PlaneJob's *_next). Saves the final stage's preparation pass and resets. A
// leading stage that finds no room for the final stage's weight sums (8 B per
// pixel) sets None: the stages then run one after the other, with the same results.
enum class Chain { None, Leads, Follows };

// One stage over device-resident planes (all with row pitch `stride`).
template <typename T>
static int run_stage_device(bm3d_ctx *ctx, const bm3d_stage_params *p, bool wiener, int nplanes,
                            T *const dst[], const T *const src[], const T *const ref[], int width,
                            int height, size_t stride, double value_range, cudaStream_t s,
                            Chain &chain, int *gcount = nullptr, int *gpos = nullptr,
                            T *gkey = nullptr, bool bm_only = false)
{
    StageArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    fill_tables(a, p, wiener, nplanes, value_range);
    a.stride = static_cast<long long>(stride);
    a.ref_alias_src = 0;
    for (int c = 0; c < nplanes; ++c) {
        a.src[c] = src[c];
        a.ref[c] = ref[c];
        if (src[c] == ref[c]) a.ref_alias_src |= 1 << c;
    }
    int warps;
    int rc = plan_geometry(ctx, a, p, wiener, nplanes, width, height, warps);
    if (rc != BM3D_OK) return rc;
    a.dct_fwd = GenericTables<T>::fwd(ctx);
    a.dct_inv = GenericTables<T>::inv(ctx);
    a.pad_fwd = ctx->gtab_f + 2 * kDctTableSize;
    a.pad_inv = a.pad_fwd + kPad32Table;
    using Acc = typename AccOf<T>::type;
    const size_t acc_bytes = sizeof(Acc) * static_cast<size_t>(width) * height;
    const long long npx = static_cast<long long>(width) * height;
    const int threads = 256;
    const int blocks = static_cast<int>(std::min<long long>((npx + threads - 1) / threads,
                                                            static_cast<long long>(ctx->sm_count) * 8));
    fixed_point_bounds(p, width, height, a.log2_bound, a.log2_corner);
    a.absmax = ctx->absmax;
    // FP32 sums are fixed point: planes with NaN / Inf pixels take the checking
    // aggregation (FP64 sums are doubles and carry them like the reference's)
    constexpr bool kFixed = std::is_same<Acc, long long>::value;
    const bool follows = chain == Chain::Follows;
    a.nonfinite = !kFixed ? nullptr : follows ? ctx->nonfinite_next : ctx->nonfinite;
    a.stats = ctx->stats;
    a.bad = ctx->stats + 4;
    // per-call state and counters; the invariant counter (stats[4]) is sticky
    if (!follows) CK(ctx, cudaMemsetAsync(ctx->head, 0, kHeadClear, s));
    PlaneJobs<T> jobs;
    std::memset(&jobs, 0, sizeof(jobs));
    int njobs = 0, plane_of[kMaxPlanes];
    for (int c = 0; c < nplanes; ++c) {
        if (!(a.active & (1 << c)) && !bm_only) continue;
        DevBuf &den = follows ? ctx->den_next[c] : ctx->acc[2 * c + 1];
        if ((rc = ensure(ctx, ctx->acc[2 * c], acc_bytes)) != BM3D_OK) return rc;
        if ((rc = ensure(ctx, den, acc_bytes)) != BM3D_OK) return rc;
        a.num[c] = static_cast<Acc *>(ctx->acc[2 * c].ptr);
        a.den[c] = static_cast<Acc *>(den.ptr);
        if (kFixed) {  // starts zeroed; normalisation leaves it zero
            const bool grow = ctx->poison[c].bytes < static_cast<size_t>(npx);
            if ((rc = ensure(ctx, ctx->poison[c], static_cast<size_t>(npx))) != BM3D_OK) return rc;
            if (grow) CK(ctx, cudaMemsetAsync(ctx->poison[c].ptr, 0, ctx->poison[c].bytes, s));
            a.poison[c] = static_cast<unsigned char *>(ctx->poison[c].ptr);
        }
        plane_of[njobs] = c;
        PlaneJob<T> &q = jobs.job[njobs++];
        q.num = a.num[c];
        q.den = a.den[c];
        q.src = src[c];
        q.ref = ref[c] != src[c] ? ref[c] : nullptr;
        q.dst = dst[c];
        q.src_stride = q.dst_stride = static_cast<long long>(stride);
        q.width = width;
        q.height = height;
        q.block_size = a.block_size;
        q.absmax = ctx->absmax + c;
        q.log2_bound = a.log2_bound;
        q.log2_corner = a.log2_corner;
        q.nonfinite = kFixed ? const_cast<unsigned *>(a.nonfinite) + c : nullptr;
        q.poison = a.poison[c];
    }
    for (int j = 0; j < njobs && chain == Chain::Leads; ++j) {
        bool got;
        if ((rc = ensure_optional(ctx, ctx->den_next[plane_of[j]], acc_bytes, s, got)) != BM3D_OK) return rc;
        if (!got) chain = Chain::None;
    }
    for (int j = 0; j < njobs && chain == Chain::Leads; ++j) {
        PlaneJob<T> &q = jobs.job[j];
        q.den_next = static_cast<long long *>(ctx->den_next[plane_of[j]].ptr);
        q.nonfinite_next = ctx->nonfinite_next + plane_of[j];
        if (j == 0) q.stats = ctx->stats;
    }
    // (njobs 0: noise levels that are not numbers pass the guard and select no plane)
    if (!bm_only && !follows && njobs > 0) {
        prep_kernel<T><<<dim3(std::min(height, blocks), njobs), threads, 0, s>>>(jobs);
        CK(ctx, cudaGetLastError());
    }
    a.group_count = gcount;
    a.group_pos = gpos;
    a.group_key = gkey;
    a.bm_only = bm_only ? 1 : 0;
    if ((rc = launch_stage(ctx, a, wiener, nplanes, s, warps)) != BM3D_OK) return rc;
    ctx->last_stream = s;
    if (bm_only || njobs == 0) return BM3D_OK;
    normalize_kernel<T><<<dim3(normalize_tiles<T>(width, height), njobs), 256, 0, s>>>(jobs);
    CK(ctx, cudaGetLastError());
    return BM3D_OK;
}

// Host-mode calls end synchronised; a nonzero invariant counter means a group
// member fell outside its tile's staged window and was skipped.
int bm3d::check_invariants(bm3d_ctx *ctx)
{
    unsigned long long v[kStats];
    CK(ctx, cudaMemcpy(v, ctx->stats, sizeof(v), cudaMemcpyDeviceToHost));
    if (v[4] != 0) {  // low 32 bits: group blocks outside the window; high: CTAs short of smem
        ctx->err = "internal error: " + std::to_string(v[4] & 0xffffffffull) +
                   " group blocks outside the staged window, " + std::to_string(v[4] >> 32) +
                   " tiles launched with too little shared memory";
        return BM3D_ERR_CUDA;
    }
    return BM3D_OK;
}

template <typename T>
static int passthrough(bm3d_ctx *ctx, int nplanes, T *const dst[], const T *const src[], int width,
                       int height, size_t stride, int mem, cudaStream_t s)
{
    for (int c = 0; c < nplanes; ++c) {
        if (dst[c] == src[c]) continue;
        int rc = copy_plane(ctx, dst[c], stride, src[c], stride, width, height,
                            mem == BM3D_MEM_HOST ? cudaMemcpyHostToHost : cudaMemcpyDeviceToDevice, s);
        if (rc != BM3D_OK) return rc;
    }
    if (mem == BM3D_MEM_HOST) CK(ctx, cudaStreamSynchronize(s));
    return BM3D_COPIED;
}

static int check_planes(int nplanes, const void *const dst[], const void *const src[],
                        const void *const ref[], int width, int height, size_t stride, int bs)
{
    if (width < bs || height < bs || stride < static_cast<size_t>(width)) return BM3D_ERR_INVALID;
    for (int c = 0; c < nplanes; ++c)
        if (!dst[c] || !src[c] || (ref && !ref[c])) return BM3D_ERR_INVALID;
    return BM3D_OK;
}

// A stage in either memory kind. In host mode planes go through context
// staging buffers with pitch = width.
template <typename T>
int bm3d::stage_any(bm3d_ctx *ctx, const bm3d_stage_params *p, int wiener, int nplanes,
              T *const dst[], const T *const src[], const T *const ref[], int width, int height,
              size_t stride, double value_range, int mem, void *stream)
{
    if (!ctx) return BM3D_ERR_INVALID;
    if (mem != BM3D_MEM_HOST && mem != BM3D_MEM_DEVICE) return BM3D_ERR_INVALID;
    const Guard g = check_params(p, nplanes);
    if (g == Guard::Invalid) return BM3D_ERR_INVALID;
    int rc = check_planes(nplanes, reinterpret_cast<const void *const *>(dst),
                          reinterpret_cast<const void *const *>(src),
                          reinterpret_cast<const void *const *>(ref), width, height, stride,
                          p->block_size > 0 ? p->block_size : 1);
    if (rc != BM3D_OK) return rc;
    CK(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (g == Guard::Copy) return passthrough(ctx, nplanes, dst, src, width, height, stride, mem, s);
    if (g == Guard::Unsupported) {
        ctx->err = "parameters outside this build (BlockSize <= 16, GroupSize <= 32)";
        return BM3D_ERR_UNSUPPORTED;
    }
    Chain alone = Chain::None;
    if (mem == BM3D_MEM_DEVICE)
        return run_stage_device(ctx, p, wiener != 0, nplanes, dst, src, ref, width, height, stride,
                                value_range, s, alone);
    const size_t plane_bytes = sizeof(T) * static_cast<size_t>(width) * height;
    T *dd[kMaxPlanes];
    const T *ds[kMaxPlanes], *dr[kMaxPlanes];
    for (int c = 0; c < nplanes; ++c) {
        if ((rc = ensure(ctx, ctx->stage_in[c], plane_bytes)) != BM3D_OK) return rc;
        if ((rc = ensure(ctx, ctx->stage_out[c], plane_bytes)) != BM3D_OK) return rc;
        T *in = static_cast<T *>(ctx->stage_in[c].ptr);
        if ((rc = copy_plane(ctx, in, width, src[c], stride, width, height,
                             cudaMemcpyHostToDevice, s)) != BM3D_OK)
            return rc;
        ds[c] = in;
        if (ref[c] == src[c]) {
            dr[c] = in;
        } else {
            if ((rc = ensure(ctx, ctx->stage_ref[c], plane_bytes)) != BM3D_OK) return rc;
            T *r = static_cast<T *>(ctx->stage_ref[c].ptr);
            if ((rc = copy_plane(ctx, r, width, ref[c], stride, width, height,
                                 cudaMemcpyHostToDevice, s)) != BM3D_OK)
                return rc;
            dr[c] = r;
        }
        dd[c] = static_cast<T *>(ctx->stage_out[c].ptr);
        // planes this stage leaves alone (sigma <= 0) keep the caller's contents
        if (nplanes > 1 && !(p->sigma[c] > 0))
            if ((rc = copy_plane(ctx, dd[c], width, dst[c], stride, width, height,
                                 cudaMemcpyHostToDevice, s)) != BM3D_OK)
                return rc;
    }
    rc = run_stage_device(ctx, p, wiener != 0, nplanes, dd, ds, dr, width, height, width,
                          value_range, s, alone);
    if (rc != BM3D_OK) return rc;
    for (int c = 0; c < nplanes; ++c)
        if ((rc = copy_plane(ctx, dst[c], stride, static_cast<const T *>(dd[c]), width, width,
                             height, cudaMemcpyDeviceToHost, s)) != BM3D_OK)
            return rc;
    CK(ctx, cudaStreamSynchronize(s));
    return check_invariants(ctx);
}

extern "C" int bm3d_stage(bm3d_ctx *ctx, const bm3d_stage_params *params, int wiener, float *dst,
                          const float *src, const float *ref, int width, int height,
                          size_t stride, float value_range, int mem, void *stream)
{
    float *d[1] = {dst};
    const float *s[1] = {src}, *r[1] = {ref ? ref : src};
    return stage_any<float>(ctx, params, wiener, 1, d, s, r, width, height, stride, value_range,
                            mem, stream);
}

extern "C" int bm3d_stage_f64(bm3d_ctx *ctx, const bm3d_stage_params *params, int wiener,
                              double *dst, const double *src, const double *ref, int width,
                              int height, size_t stride, double value_range, int mem,
                              void *stream)
{
    double *d[1] = {dst};
    const double *s[1] = {src}, *r[1] = {ref ? ref : src};
    return stage_any<double>(ctx, params, wiener, 1, d, s, r, width, height, stride, value_range,
                             mem, stream);
}

extern "C" int bm3d_stage3(bm3d_ctx *ctx, const bm3d_stage_params *params, int wiener,
                           float *const dst[3], const float *const src[3],
                           const float *const ref[3], int width, int height, size_t stride,
                           float value_range, int mem, void *stream)
{
    if (!dst || !src) return BM3D_ERR_INVALID;
    const float *const *r = ref ? ref : src;
    return stage_any<float>(ctx, params, wiener, 3, dst, src, r, width, height, stride,
                            value_range, mem, stream);
}

template <typename T>
int bm3d::full_any(bm3d_ctx *ctx, const bm3d_stage_params *basic, const bm3d_stage_params *fin,
             int nplanes, T *const dst[], const T *const src[], const T *const ref[], int width,
             int height, size_t stride, double value_range, int mem, void *stream)
{
    if (!ctx || !basic || !fin) return BM3D_ERR_INVALID;
    if (mem != BM3D_MEM_HOST && mem != BM3D_MEM_DEVICE) return BM3D_ERR_INVALID;
    int rc = check_planes(nplanes, reinterpret_cast<const void *const *>(dst),
                          reinterpret_cast<const void *const *>(src), nullptr, width, height,
                          stride, 1);
    if (rc != BM3D_OK) return rc;
    CK(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t plane_bytes = sizeof(T) * static_cast<size_t>(width) * height;
    const size_t dpitch = mem == BM3D_MEM_HOST ? static_cast<size_t>(width) : stride;
    // Device-resident src and dst (context staging in host mode) and the basic
    // estimate, all with row pitch dpitch.
    const T *ds[kMaxPlanes], *dr[kMaxPlanes];
    T *tmp[kMaxPlanes], *dd[kMaxPlanes];
    for (int c = 0; c < nplanes; ++c) {
        if ((rc = ensure(ctx, ctx->basic[c], sizeof(T) * dpitch * height)) != BM3D_OK) return rc;
        tmp[c] = static_cast<T *>(ctx->basic[c].ptr);
    }
    // a distinct ref (the basic stage matches on it; src when absent)
    const bool own_ref = ref != nullptr && ref[0] != nullptr && ref[0] != src[0];
    if (mem == BM3D_MEM_HOST) {
        for (int c = 0; c < nplanes; ++c) {
            if ((rc = ensure(ctx, ctx->stage_in[c], plane_bytes)) != BM3D_OK) return rc;
            if ((rc = ensure(ctx, ctx->stage_out[c], plane_bytes)) != BM3D_OK) return rc;
            T *in = static_cast<T *>(ctx->stage_in[c].ptr);
            if ((rc = copy_plane(ctx, in, width, src[c], stride, width, height,
                                 cudaMemcpyHostToDevice, s)) != BM3D_OK)
                return rc;
            ds[c] = in;
            dr[c] = in;
            dd[c] = static_cast<T *>(ctx->stage_out[c].ptr);
        }
        if (own_ref) {
            if ((rc = ensure(ctx, ctx->stage_ref[0], plane_bytes)) != BM3D_OK) return rc;
            T *r = static_cast<T *>(ctx->stage_ref[0].ptr);
            if ((rc = copy_plane(ctx, r, width, ref[0], stride, width, height,
                                 cudaMemcpyHostToDevice, s)) != BM3D_OK)
                return rc;
            dr[0] = r;
        }
    } else {
        for (int c = 0; c < nplanes; ++c) {
            ds[c] = src[c];
            dr[c] = src[c];
            dd[c] = dst[c];
        }
        if (own_ref) dr[0] = ref[0];
    }
    // Planes a stage does not filter (sigma <= 0), or a stage whose parameters
    // the reference's guard rejects, pass src through: there the basic estimate
    // and dst are copies of src, as in the reference's in-place Frame path
    // (source/BM3D.cpp:512-521).
    const Guard gb = check_params(basic, nplanes), gf = check_params(fin, nplanes);
    auto filtered = [&](const bm3d_stage_params *p, Guard g, int c) {
        return g == Guard::Run && (nplanes == 1 || p->sigma[c] > 0);
    };
    for (int c = 0; c < nplanes; ++c) {
        if (!filtered(basic, gb, c) &&
            (rc = copy_plane(ctx, tmp[c], dpitch, ds[c], dpitch, width, height,
                             cudaMemcpyDeviceToDevice, s)) != BM3D_OK)
            return rc;
        if (!filtered(fin, gf, c) &&
            (rc = copy_plane(ctx, dd[c], dpitch, ds[c], dpitch, width, height,
                             cudaMemcpyDeviceToDevice, s)) != BM3D_OK)
            return rc;
    }
    auto refused = [&](Guard g) {
        if (g == Guard::Invalid) return BM3D_ERR_INVALID;
        if (g == Guard::Unsupported) {
            ctx->err = "parameters outside this build (BlockSize <= 16, GroupSize <= 32)";
            return BM3D_ERR_UNSUPPORTED;
        }
        return BM3D_OK;
    };
    // both stages on the same planes with fixed-point sums: the basic stage's
    // passes prepare the final stage
    bool chained = std::is_same<typename AccOf<T>::type, long long>::value && gb == Guard::Run &&
                   gf == Guard::Run;
    bool any = false;  // (the passes that prepare run on planes that are filtered)
    for (int c = 0; c < nplanes; ++c) {
        chained = chained && filtered(basic, gb, c) == filtered(fin, gf, c);
        any = any || filtered(basic, gb, c);
    }
    chained = chained && any;
    if ((rc = refused(gb)) != BM3D_OK) return rc;
    Chain chain = chained ? Chain::Leads : Chain::None;
    if (gb == Guard::Run) {
        rc = run_stage_device(ctx, basic, false, nplanes, tmp, ds, dr, width, height, dpitch,
                              value_range, s, chain);
        if (rc != BM3D_OK) return rc;
    }
    if ((rc = refused(gf)) != BM3D_OK) return rc;
    if (gf == Guard::Run) {
        const T *tr[kMaxPlanes];
        for (int c = 0; c < nplanes; ++c) tr[c] = tmp[c];
        if (chain == Chain::Leads) chain = Chain::Follows;
        rc = run_stage_device(ctx, fin, true, nplanes, dd, ds, tr, width, height, dpitch,
                              value_range, s, chain);
        if (rc != BM3D_OK) return rc;
    }
    if (mem == BM3D_MEM_HOST) {
        for (int c = 0; c < nplanes; ++c)
            if ((rc = copy_plane(ctx, dst[c], stride, static_cast<const T *>(dd[c]), width, width,
                                 height, cudaMemcpyDeviceToHost, s)) != BM3D_OK)
                return rc;
        CK(ctx, cudaStreamSynchronize(s));
        return check_invariants(ctx);
    }
    return BM3D_OK;
}

extern "C" int bm3d_full(bm3d_ctx *ctx, const bm3d_stage_params *basic,
                         const bm3d_stage_params *final_, float *dst, const float *src,
                         const float *ref, int width, int height, size_t stride,
                         float value_range, int mem, void *stream)
{
    float *d[1] = {dst};
    const float *s[1] = {src}, *r[1] = {ref};
    return full_any<float>(ctx, basic, final_, 1, d, s, r, width, height, stride, value_range,
                           mem, stream);
}

extern "C" int bm3d_full3(bm3d_ctx *ctx, const bm3d_stage_params *basic,
                          const bm3d_stage_params *final_, float *const dst[3],
                          const float *const src[3], const float *const ref[3], int width,
                          int height, size_t stride, float value_range, int mem, void *stream)
{
    if (!dst || !src) return BM3D_ERR_INVALID;
    return full_any<float>(ctx, basic, final_, 3, dst, src, ref, width, height, stride,
                           value_range, mem, stream);
}


// The float drivers the other translation units call.
template void bm3d::fill_tables<float>(StageArgs<float> &, const bm3d_stage_params *, bool, int,
                                 double);
template int bm3d::stage_any<float>(bm3d_ctx *, const bm3d_stage_params *, int, int, float *const[],
                              const float *const[], const float *const[], int, int, size_t,
                              double, int, void *);
template int bm3d::full_any<float>(bm3d_ctx *, const bm3d_stage_params *, const bm3d_stage_params *,
                             int, float *const[], const float *const[], const float *const[],
                             int, int, size_t, double, int, void *);

// The groups of every reference block; keys may be null.
static int dump_groups(bm3d_ctx *ctx, const bm3d_stage_params *p, int wiener, const float *ref,
                       int width, int height, size_t stride, float value_range, int *counts,
                       int *pos_yx, float *keys)
{
    if (!ctx || !p || !ref || !counts || !pos_yx) return BM3D_ERR_INVALID;
    const Guard g = check_params(p, 1);
    if (g == Guard::Invalid || g == Guard::Copy) return BM3D_ERR_INVALID;
    if (g == Guard::Unsupported) return BM3D_ERR_UNSUPPORTED;
    if (width < p->block_size || height < p->block_size || stride < static_cast<size_t>(width))
        return BM3D_ERR_INVALID;
    CK(ctx, cudaSetDevice(ctx->device));
    const long long nref = bm3d_ref_block_count(p, width, height);
    int rc;
    const size_t plane_bytes = sizeof(float) * static_cast<size_t>(width) * height;
    if ((rc = ensure(ctx, ctx->stage_in[0], plane_bytes)) != BM3D_OK) return rc;
    if ((rc = ensure(ctx, ctx->groups[0], sizeof(int) * nref)) != BM3D_OK) return rc;
    if ((rc = ensure(ctx, ctx->groups[1], sizeof(int) * nref * kGSTab * 2)) != BM3D_OK) return rc;
    if (keys && (rc = ensure(ctx, ctx->groups[2], sizeof(float) * nref * kGSTab)) != BM3D_OK) return rc;
    cudaStream_t s = nullptr;
    float *in = static_cast<float *>(ctx->stage_in[0].ptr);
    if ((rc = copy_plane(ctx, in, width, ref, stride, width, height, cudaMemcpyHostToDevice, s)) !=
        BM3D_OK)
        return rc;
    float *d[1] = {in};
    const float *sp[1] = {in};
    Chain alone = Chain::None;
    rc = run_stage_device<float>(ctx, p, wiener != 0, 1, d, sp, sp, width, height, width,
                                 value_range, s, alone, static_cast<int *>(ctx->groups[0].ptr),
                                 static_cast<int *>(ctx->groups[1].ptr),
                                 keys ? static_cast<float *>(ctx->groups[2].ptr) : nullptr, true);
    if (rc != BM3D_OK) return rc;
    CK(ctx, cudaMemcpyAsync(counts, ctx->groups[0].ptr, sizeof(int) * nref, cudaMemcpyDeviceToHost, s));
    CK(ctx, cudaMemcpyAsync(pos_yx, ctx->groups[1].ptr, sizeof(int) * nref * kGSTab * 2,
                            cudaMemcpyDeviceToHost, s));
    if (keys)
        CK(ctx, cudaMemcpyAsync(keys, ctx->groups[2].ptr, sizeof(float) * nref * kGSTab,
                                cudaMemcpyDeviceToHost, s));
    CK(ctx, cudaStreamSynchronize(s));
    return BM3D_OK;
}

extern "C" int bm3d_debug_groups(bm3d_ctx *ctx, const bm3d_stage_params *p, int wiener,
                                 const float *ref, int width, int height, size_t stride,
                                 float value_range, int *counts, int *pos_yx, float *keys)
{
    if (!keys) return BM3D_ERR_INVALID;
    return dump_groups(ctx, p, wiener, ref, width, height, stride, value_range, counts, pos_yx, keys);
}

extern "C" int bm3d_debug_positions(bm3d_ctx *ctx, const bm3d_stage_params *p, int wiener,
                                    const float *ref, int width, int height, size_t stride,
                                    float value_range, int *counts, int *pos_yx)
{
    return dump_groups(ctx, p, wiener, ref, width, height, stride, value_range, counts, pos_yx, nullptr);
}

extern "C" int bm3d_set_kernel_timing(bm3d_ctx *ctx, int on)
{
    if (!ctx) return BM3D_ERR_INVALID;
    CK(ctx, cudaSetDevice(ctx->device));
    drain_timing(ctx);
    ctx->timing = on != 0;
    ctx->time_ms[0] = ctx->time_ms[1] = 0;
    ctx->launches[0] = ctx->launches[1] = 0;
    return BM3D_OK;
}

extern "C" int bm3d_kernel_time(bm3d_ctx *ctx, int wiener, double *ms, long long *launches)
{
    if (!ctx || !ms || !launches) return BM3D_ERR_INVALID;
    CK(ctx, cudaSetDevice(ctx->device));
    drain_timing(ctx);
    *ms = ctx->time_ms[wiener ? 1 : 0];
    *launches = ctx->launches[wiener ? 1 : 0];
    return BM3D_OK;
}

extern "C" int bm3d_last_stats(bm3d_ctx *ctx, unsigned long long out[4])
{
    if (!ctx || !out) return BM3D_ERR_INVALID;
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaStreamSynchronize(ctx->last_stream));
    CK(ctx, cudaMemcpy(out, ctx->stats, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    return BM3D_OK;
}

extern "C" int bm3d_check(bm3d_ctx *ctx)
{
    if (!ctx) return BM3D_ERR_INVALID;
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, cudaStreamSynchronize(ctx->last_stream));
    return check_invariants(ctx);
}

// ---------------------------------------------------------------------------
// Allocation-free stage: bm3d_stage_noalloc.
//
// For callers that must not allocate device memory after start-up, e.g. a
// filter plugin inside a host application that owns every device allocation,
// or a real-time video path where a cudaMalloc (which can synchronise the
// device and can fail under memory pressure) is not allowed per frame. The
// stage kernels' scratch -- the fixed-point numerator and weight planes, the
// per-plane |src| maximum and the counters -- lives in the file-scope array
// below instead of context buffers. Every GPU that loads this library holds
// the array until the process exits.

namespace {

constexpr size_t kNoAllocMaxPixels = size_t(1) << 21;  // 2,097,152 pixels (1920x1080 fits)
constexpr size_t kNoAllocAccBytes = kNoAllocMaxPixels * sizeof(long long);
// num (int64 per pixel) | den (int64 per pixel) | header: absmax (4 floats) at 0,
// non-finite pixel count at 128 | counters (8 x u64) | poison map (1 byte per pixel)
constexpr size_t kNoAllocBytes = 2 * kNoAllocAccBytes + 256 + 256 + kNoAllocMaxPixels;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

struct NoAllocDevice {
    bool ready = false;
    unsigned char *scratch = nullptr;  // device address of g_noalloc_scratch
    int sm_count = 0;
    size_t smem_optin = 0;
};

constexpr int kNoAllocMaxDevices = 64;
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;

// Status for a failed step: CUDA errors map to BM3D_ERR_CUDA, everything else
// to the given code. The message (with the CUDA error text, if any) becomes
// this thread's context-free error, which bm3d_last_error(NULL) returns.
int noalloc_error(const char *what, cudaError_t e = cudaSuccess, int code = BM3D_ERR_INVALID)
{
    if (e != cudaSuccess) {
        char buf[256];
        std::snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
        g_create_error = buf;
        return BM3D_ERR_CUDA;
    }
    g_create_error = what;
    return code;
}

// Set-up once per device, with that device current: the device address of the
// scratch array (the host-side symbol is only a stand-in, not a device
// address), the cosine tables, and the device limits.
int noalloc_setup(int dev, NoAllocDevice **out)
{
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAllocDevice &d = g_noalloc_dev[dev];
    if (d.ready) {
        *out = &d;
        return BM3D_OK;
    }
    int major = 0, sm = 0, optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (e != cudaSuccess) return noalloc_error("cudaDeviceGetAttribute", e);
    if (major < 10)
        return noalloc_error("bm3d_stage_noalloc: this build targets sm_100a (B200)",
                             cudaSuccess, BM3D_ERR_CUDA);
    void *ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) return noalloc_error("cudaGetSymbolAddress(g_noalloc_scratch)", e);
    // the cosine tables live in fixed-size host arrays (no heap), uploaded per device
    if ((e = upload_dct_tables()) != cudaSuccess)
        return noalloc_error("cudaMemcpyToSymbol(cosine tables)", e);
    if ((e = cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) !=
            cudaSuccess)
        return noalloc_error("cudaDeviceGetAttribute", e);
    d.scratch = static_cast<unsigned char *>(ptr);
    d.sm_count = sm;
    d.smem_optin = static_cast<size_t>(optin);
    d.ready = true;
    *out = &d;
    return BM3D_OK;
}

// Offsets inside the scratch array after the two accumulator planes: the
// per-call |src| maximum (256 bytes, cleared by every call), then the counters:
// four statistics (cleared by every call) and the consistency counter, which
// starts at zero when the library loads and is cleared only by
// bm3d_noalloc_check, so it covers every call since the last check.
constexpr size_t kNoAllocAbsmaxOff = 2 * kNoAllocAccBytes;
constexpr size_t kNoAllocNonfiniteOff = kNoAllocAbsmaxOff + 128;
constexpr size_t kNoAllocStatsOff = kNoAllocAbsmaxOff + 256;
constexpr size_t kNoAllocPoisonOff = kNoAllocStatsOff + 256;
constexpr size_t kNoAllocClearBytes = 256 + 4 * sizeof(unsigned long long);

}  // namespace

extern "C" int bm3d_stage_noalloc(const bm3d_stage_params *params, int wiener, float *dst,
                                  const float *src, const float *ref, int width, int height,
                                  size_t stride, float value_range, void *stream)
{
    if (!ref) ref = src;
    if (!params || !dst || !src) return noalloc_error("bm3d_stage_noalloc: null argument");
    const Guard g = check_params(params, 1);
    if (g == Guard::Invalid) return noalloc_error("bm3d_stage_noalloc: invalid parameters");
    // the register-resident kernel only: BlockSize 8, GroupSize <= 16
    if (g == Guard::Unsupported || !fast_path(params))
        return noalloc_error("bm3d_stage_noalloc: only BlockSize 8 with GroupSize <= 16",
                             cudaSuccess, BM3D_ERR_UNSUPPORTED);
    if (width < params->block_size || height < params->block_size ||
        stride < static_cast<size_t>(width))
        return noalloc_error("bm3d_stage_noalloc: width/height below BlockSize or stride < width");
    if (static_cast<size_t>(width) * static_cast<size_t>(height) > kNoAllocMaxPixels)
        return noalloc_error("bm3d_stage_noalloc: plane larger than the 2,097,152-pixel static "
                             "scratch", cudaSuccess, BM3D_ERR_TOO_LARGE);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return noalloc_error("cudaGetDevice", e);
    if (dev < 0 || dev >= kNoAllocMaxDevices) return noalloc_error("bm3d_stage_noalloc: device id");
    NoAllocDevice *d = nullptr;
    int rc = noalloc_setup(dev, &d);
    if (rc != BM3D_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (g == Guard::Copy) {
        if (dst != src &&
            (e = cudaMemcpy2DAsync(dst, stride * sizeof(float), src, stride * sizeof(float),
                                   width * sizeof(float), height, cudaMemcpyDeviceToDevice, s)) !=
                cudaSuccess)
            return noalloc_error("cudaMemcpy2DAsync", e);
        return BM3D_COPIED;
    }

    // The shared scratch: this call's accumulators start from zero below.
    long long *num = reinterpret_cast<long long *>(d->scratch);
    long long *den = reinterpret_cast<long long *>(d->scratch + kNoAllocAccBytes);
    float *absmax = reinterpret_cast<float *>(d->scratch + kNoAllocAbsmaxOff);
    unsigned *nonfinite = reinterpret_cast<unsigned *>(d->scratch + kNoAllocNonfiniteOff);
    unsigned char *poison = d->scratch + kNoAllocPoisonOff;
    unsigned long long *stats = reinterpret_cast<unsigned long long *>(d->scratch + kNoAllocStatsOff);

    StageArgs<float> a;
    std::memset(&a, 0, sizeof(a));
    fill_tables(a, params, wiener != 0, 1, value_range);
    a.stride = static_cast<long long>(stride);
    a.src[0] = src;
    a.ref[0] = ref;
    a.ref_alias_src = src == ref ? 1 : 0;
    bm3d_ctx info;  // device limits and default tiling only; owns no device memory
    info.device = dev;
    info.sm_count = d->sm_count;
    info.smem_optin = d->smem_optin;
    int warps;
    rc = plan_geometry(&info, a, params, wiener != 0, 1, width, height, warps);
    if (rc != BM3D_OK) return noalloc_error(info.err.c_str(), cudaSuccess, rc);
    fixed_point_bounds(params, width, height, a.log2_bound, a.log2_corner);
    a.absmax = absmax;
    a.nonfinite = nonfinite;
    a.poison[0] = poison;
    a.num[0] = num;
    a.den[0] = den;
    a.stats = stats;
    a.bad = stats + 4;

    const long long npx = static_cast<long long>(width) * height;
    const int threads = 256;
    const int blocks = static_cast<int>(
        std::min<long long>((npx + threads - 1) / threads, static_cast<long long>(d->sm_count) * 8));
    // |src| maximum and statistics start at zero; the consistency counter
    // (stats[4]) is left alone so bm3d_noalloc_check sees every call
    if ((e = cudaMemsetAsync(absmax, 0, kNoAllocClearBytes, s)) != cudaSuccess)
        return noalloc_error("cudaMemsetAsync(scratch header)", e);
    PlaneJobs<float> jobs;
    std::memset(&jobs, 0, sizeof(jobs));
    PlaneJob<float> &q = jobs.job[0];
    q.num = num;
    q.den = den;
    q.src = src;
    q.ref = ref != src ? ref : nullptr;
    q.dst = dst;
    q.src_stride = q.dst_stride = a.stride;
    q.width = width;
    q.height = height;
    q.block_size = a.block_size;
    q.absmax = absmax;
    q.log2_bound = a.log2_bound;
    q.log2_corner = a.log2_corner;
    q.nonfinite = nonfinite;
    q.poison = poison;
    prep_kernel<float><<<std::min(height, blocks), threads, 0, s>>>(jobs);
    if ((e = cudaGetLastError()) != cudaSuccess) return noalloc_error("prep_kernel", e);
    rc = launch_stage(&info, a, wiener != 0, 1, s, warps);
    if (rc != BM3D_OK) return noalloc_error(info.err.c_str(), cudaSuccess, rc);
    normalize_kernel<float><<<normalize_tiles<float>(width, height), 256, 0, s>>>(jobs);
    if ((e = cudaGetLastError()) != cudaSuccess) return noalloc_error("normalize_kernel", e);
    return BM3D_OK;
}

extern "C" int bm3d_noalloc_check(void *stream)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return noalloc_error("cudaGetDevice", e);
    if (dev < 0 || dev >= kNoAllocMaxDevices) return noalloc_error("bm3d_noalloc_check: device id");
    NoAllocDevice *d = nullptr;
    int rc = noalloc_setup(dev, &d);
    if (rc != BM3D_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess)
        return noalloc_error("cudaStreamSynchronize", e);
    unsigned long long *bad =
        reinterpret_cast<unsigned long long *>(d->scratch + kNoAllocStatsOff) + 4;
    unsigned long long v = 0;
    if ((e = cudaMemcpy(&v, bad, sizeof(v), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return noalloc_error("cudaMemcpy(consistency counter)", e);
    if (v == 0) return BM3D_OK;
    if ((e = cudaMemset(bad, 0, sizeof(v))) != cudaSuccess)
        return noalloc_error("cudaMemset(consistency counter)", e);
    const std::string msg = "internal error: " + std::to_string(v & 0xffffffffull) +
                            " group blocks outside the staged window, " +
                            std::to_string(v >> 32) +
                            " tiles launched with too little shared memory";
    return noalloc_error(msg.c_str(), cudaSuccess, BM3D_ERR_CUDA);
}

