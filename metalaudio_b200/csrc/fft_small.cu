// __global__ wrappers and launchers for the in-shared-memory transforms (N <= 8192).
#include "bulk_copy.cuh"
#include "fft_plan.h"
#include "host_tables.h"

namespace ma {

struct DevCta {
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int bid() const { return blockIdx.x; }
    __device__ __forceinline__ int nblocks() const { return gridDim.x; }
    __device__ __forceinline__ void sync() { __syncthreads(); }
    __device__ __forceinline__ void bulk_init(uint64_t* bar) { bulk_barrier_init(bar); }
    __device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
        bulk_copy_g2s(dst, src, bytes, bar);
    }
    __device__ __forceinline__ void bulk_expect(uint64_t* bar, uint32_t total_bytes) { bulk_barrier_expect(bar, total_bytes); }
    __device__ __forceinline__ void bulk_part(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
        bulk_copy_part(dst, src, bytes, bar);
    }
    __device__ __forceinline__ bool bulk_wait(uint64_t* bar, uint32_t parity) { return bulk_barrier_wait(bar, parity); }
};

extern __shared__ float4 ma_dyn_smem[];

// Programmatic dependent launch, used by the convolution's streaming step (r2c -> multiply-
// accumulate -> c2r, every block).  A kernel launched with the programmatic-stream-serialization
// attribute may become resident once every CTA of the kernel before it has executed
// launch_dependents; it must execute wait before it touches (or, for r2c, before it completes
// ahead of) anything the earlier kernel produces.  Without the attribute both are no-ops.
//   c2r: wait, then launch_dependents - the next step's r2c starts while this c2r still runs
//        (they share no data), but never before the multiply-accumulate that reads the delay line
//        slot r2c is about to overwrite has completed;
//   r2c: launch_dependents at once, wait only at the very end - so it completes after the c2r
//        before it, and everything later in the stream stays ordered after that c2r as well.
__device__ __forceinline__ void dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// cudaLaunchKernelEx with the attribute (dependent != 0) or a plain launch.
template <typename K, typename P>
static void launch_maybe_dependent(K kernel, int grid, int threads, size_t smem, cudaStream_t stream, const P& p,
                                   int dependent) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, p);  // an error is picked up by after_launch
}

// Kernels of several frames per CTA with a fixed layout but no staging fit five CTAs of 128 threads on an SM.
template <int M, bool ALIGNED, int LAYOUT>
constexpr int r2c_ctas() {
    return CtaShape<M>::FPC > 1 && LAYOUT >= 0 && !(ALIGNED && plan_pairable<M>()) ? 5 : 512 / CtaShape<M>::THREADS;
}

template <int M, bool ALIGNED, int LAYOUT, int MAGK, bool HALF>
__global__ void __launch_bounds__(CtaShape<M>::THREADS, r2c_ctas<M, ALIGNED, LAYOUT>()) r2c_kernel(const R2CParams p) {
    DevCta cta;
    if (p.dependent_launch) dependents_launch();
    r2c_body<M, ALIGNED, LAYOUT, MAGK, DevCta, HALF>(p, cta, reinterpret_cast<float2*>(ma_dyn_smem));
    if (p.dependent_launch) dependency_wait();
}

template <int M, int LAYOUT>
__global__ void __launch_bounds__(CtaShape<M>::THREADS, 512 / CtaShape<M>::THREADS) c2r_kernel(const C2RParams p) {
    DevCta cta;
    if (p.dependent_launch) {
        dependency_wait();
        dependents_launch();
    }
    c2r_body<M, LAYOUT, DevCta>(p, cta, reinterpret_cast<float2*>(ma_dyn_smem));
}

template <int M>
__global__ void __launch_bounds__(FftPlan<M>::T, (512 / FftPlan<M>::T) > 16 ? 16 : (512 / FftPlan<M>::T)) istft_kernel(const C2RParams p) {
    DevCta cta;
    istft_body<M, DevCta>(p, cta, reinterpret_cast<float2*>(ma_dyn_smem));
}

template <int M, int LAYOUT, int OVT, bool PLAIN = false, bool EXACT = PLAIN>
__global__ void __launch_bounds__(FftPlan<M>::T, (512 / FftPlan<M>::T) > 16 ? 16 : (512 / FftPlan<M>::T))
istft_fast_kernel(const C2RParams p) {
    DevCta cta;
    if constexpr (plan_pairable<M>())
        istft_fast_body<M, LAYOUT, OVT, DevCta, PLAIN, EXACT>(p, cta, reinterpret_cast<float2*>(ma_dyn_smem));
}

template <int M, int LAYOUT>
__global__ void __launch_bounds__(CtaShape<M>::THREADS, CtaShape<M>::THREADS == 128 ? 5 : 1) istft_rows_kernel(const C2RParams p) {
    DevCta cta;
    istft_rows_body<M, LAYOUT, DevCta>(p, cta, reinterpret_cast<float2*>(ma_dyn_smem));
}

// Resident CTAs per SM for a kernel (cached per instantiation and device), after raising
// its dynamic shared-memory limit.
template <class K>
static ma_status occupancy(K kernel, int threads, size_t smem, int* per_sm) {
    MA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int n = 0;
    MA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
    *per_sm = n > 0 ? n : 1;
    return MA_OK;
}

template <int M, bool ALIGNED, int LAYOUT, int MAGK, bool HALF = false>
static ma_status launch_r2c_t(ma_fft_plan* plan, R2CParams p) {
    using S = CtaShape<M>;
    static int per_sm[64] = {0};
    ma_context* ctx = plan->ctx;
    int& occ = per_sm[ctx->device & 63];
    constexpr size_t smem = (ALIGNED && LAYOUT >= 0 && plan_pairable<M>()) ? S::SMEM_BYTES_PREFETCH : S::SMEM_BYTES;
    if (occ == 0) MA_TRY(occupancy(r2c_kernel<M, ALIGNED, LAYOUT, MAGK, HALF>, S::THREADS, smem, &occ));
    int64_t want = (p.total_frames + S::FPC - 1) / S::FPC;
    int64_t cap = (int64_t)ctx->sm_count * occ;
    int grid = (int)(want < cap ? want : cap);
    if (grid < 1) return MA_OK;
    // One frame per CTA: nothing to fetch ahead, the threads' own loads arrive sooner than a staged copy.
    if (HALF && want <= cap) p.bulk_ok = 0;
    launch_maybe_dependent(r2c_kernel<M, ALIGNED, LAYOUT, MAGK, HALF>, grid, S::THREADS, smem, ctx->stream, p, p.dependent_launch);
    return after_launch(ctx);
}

template <int M>
static ma_status launch_r2c_variant(ma_fft_plan* plan, const R2CParams& p, bool aligned, int magk) {
    if constexpr (plan_pairable<M>()) {
        if (aligned && magk != -2) {
#define MA_R2C_CASE(L_, K_) \
    if (p.layout == L_ && magk == K_) return launch_r2c_t<M, true, L_, K_>(plan, p);
            MA_R2C_CASE(LAYOUT_HALF_INTERLEAVED, 0)
            MA_R2C_CASE(LAYOUT_HALF_INTERLEAVED, -1)
            MA_R2C_CASE(LAYOUT_HALF_PACKED, 0)
            MA_R2C_CASE(LAYOUT_HALF_PACKED, -1)
            MA_R2C_CASE(LAYOUT_FULL_SPLIT, 0)
            MA_R2C_CASE(LAYOUT_FULL_SPLIT, -1)
            MA_R2C_CASE(LAYOUT_HALF_POLAR, -1)
#undef MA_R2C_CASE
        }
        // the convolution's zero-padded blocks
        if (!aligned && magk == -1 && p.layout == LAYOUT_HALF_PACKED && p.frame_valid == M && p.window == nullptr)
            return launch_r2c_t<M, true, LAYOUT_HALF_PACKED, -1, true>(plan, p);
    }
    if constexpr (M >= 64) {
        if (p.layout == LAYOUT_HALF_INTERLEAVED && magk != -2 && !aligned)
            return magk == 0 ? launch_r2c_t<M, false, LAYOUT_HALF_INTERLEAVED, 0>(plan, p)
                             : launch_r2c_t<M, false, LAYOUT_HALF_INTERLEAVED, -1>(plan, p);
    }
    if constexpr (M >= 64 && !plan_pairable<M>()) {
        if (p.layout == LAYOUT_HALF_INTERLEAVED && magk != -2)
            return magk == 0 ? launch_r2c_t<M, true, LAYOUT_HALF_INTERLEAVED, 0>(plan, p)
                             : launch_r2c_t<M, true, LAYOUT_HALF_INTERLEAVED, -1>(plan, p);
    }
    return aligned ? launch_r2c_t<M, true, -1, -2>(plan, p) : launch_r2c_t<M, false, -1, -2>(plan, p);
}

ma_status launch_r2c_small(ma_fft_plan* plan, R2CParams p) {
    p.twM = plan->d_twM;
    p.twN = plan->d_twN;
    if (p.total_frames <= 0) return MA_OK;
    const int n = plan->n;
    const int64_t last_end = (p.frames_per_signal - 1) * (int64_t)p.hop + n;
    const bool aligned = ((uintptr_t)p.in % 8 == 0) && (p.signal_stride % 2 == 0) && (p.hop % 2 == 0) &&
                         p.frame_valid >= n && last_end <= p.signal_len;
    p.bulk_ok = ((aligned || p.frame_valid == n / 2) && (uintptr_t)p.in % 16 == 0 && p.signal_stride % 4 == 0 && p.hop % 4 == 0 && n % 4 == 0) ? 1 : 0;
    p.error_flag = plan->ctx->d_error_flag;
    ma_status st = MA_ERR_UNSUPPORTED;
    // Aligned launches of the paired plans get kernels with the layout and the magnitude kind
    // fixed at compile time (no per-store branches); everything else decides at run time.
    const int magk = p.mag == nullptr ? -1 : (p.mag_kind == MAG_MAGNITUDE ? 0 : -2);
#define RUN(MM) st = launch_r2c_variant<MM>(plan, p, aligned, magk);
    MA_DISPATCH_M(plan->m, RUN)
#undef RUN
    return st;
}

template <int M, int LAYOUT>
static ma_status launch_c2r_t(ma_fft_plan* plan, const C2RParams& p) {
    using S = CtaShape<M>;
    static int per_sm[64] = {0};
    ma_context* ctx = plan->ctx;
    int& occ = per_sm[ctx->device & 63];
    constexpr size_t smem = (plan_pairable<M>() && (LAYOUT == LAYOUT_HALF_INTERLEAVED || LAYOUT == LAYOUT_HALF_PACKED))
                                ? S::SMEM_BYTES_STAGED
                                : S::SMEM_BYTES;
    if (occ == 0) MA_TRY(occupancy(c2r_kernel<M, LAYOUT>, S::THREADS, smem, &occ));
    const int64_t total = p.n_signals * p.frames_per_signal;
    int64_t want = (total + S::FPC - 1) / S::FPC;
    int64_t cap = (int64_t)ctx->sm_count * occ;
    int grid = (int)(want < cap ? want : cap);
    if (grid < 1) return MA_OK;
    launch_maybe_dependent(c2r_kernel<M, LAYOUT>, grid, S::THREADS, smem, ctx->stream, p, p.dependent_launch);
    return after_launch(ctx);
}

template <int M>
static ma_status launch_c2r_variant(ma_fft_plan* plan, const C2RParams& p) {
    if constexpr (plan_pairable<M>()) {
        // plain batched inverse of a paired plan: layout fixed at compile time
        if (p.tail == nullptr && p.n_partials <= 1 && p.mul == nullptr) {
            if (p.layout == LAYOUT_HALF_INTERLEAVED) return launch_c2r_t<M, LAYOUT_HALF_INTERLEAVED>(plan, p);
            if (p.layout == LAYOUT_HALF_PACKED) return launch_c2r_t<M, LAYOUT_HALF_PACKED>(plan, p);
            if (p.layout == LAYOUT_FULL_SPLIT) return launch_c2r_t<M, LAYOUT_FULL_SPLIT>(plan, p);
        }
    }
    return launch_c2r_t<M, -1>(plan, p);
}

ma_status launch_c2r_small(ma_fft_plan* plan, C2RParams p) {
    p.twM = plan->d_twInv;
    p.twN = plan->d_twN;
    p.error_flag = plan->ctx->d_error_flag;
    if (p.n_signals * p.frames_per_signal <= 0) return MA_OK;
    ma_status st = MA_ERR_UNSUPPORTED;
#define RUN(MM) st = launch_c2r_variant<MM>(plan, p);
    MA_DISPATCH_M(plan->m, RUN)
#undef RUN
    return st;
}

// From this many frames side by side in a CTA the row ring pays; with fewer a CTA per frame fills its warps.
constexpr int kRowsFromSlots = 4;
// Two CTAs per SM at least: smaller hops (many rows) keep the kernel with one frame per CTA.
constexpr int kRowsSmemLimit = 96 << 10;

template <int M>
static size_t istft_rows_smem(int hop) {
    using S = CtaShape<M>;
    const int reach = (2 * M + hop - 1) / hop - 1;
    return ((size_t)S::BUF_STRIDE + M) * sizeof(float2) + (size_t)(S::FPC + reach) * 2 * M * sizeof(float);
}

// Short frames without a thread-private ring (see istft_rows_body).
template <int M, int LAYOUT>
static ma_status launch_istft_rows(ma_fft_plan* plan, const C2RParams& p, size_t smem, int* cached_occ) {
    using S = CtaShape<M>;
    ma_context* ctx = plan->ctx;
    if (*cached_occ == 0) {
        MA_CUDA(cudaFuncSetAttribute(istft_rows_kernel<M, LAYOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmemLimit));
        int n = 0;
        MA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, istft_rows_kernel<M, LAYOUT>, S::THREADS, smem));
        *cached_occ = n > 0 ? n : 1;
    }
    // One wave of equal ranges, each at least one batch of the CTA's slots with the frames rebuilt in front of it.
    const int reach = (2 * M + p.hop - 1) / p.hop - 1;
    const int64_t total = p.n_signals * p.frames_per_signal, least = S::FPC > reach ? S::FPC - reach : 1;
    const int64_t want = (total + least - 1) / least, cap = (int64_t)ctx->sm_count * *cached_occ;
    istft_rows_kernel<M, LAYOUT><<<(unsigned)(want < cap ? want : cap), S::THREADS, smem, ctx->stream>>>(p);
    return after_launch(ctx);
}

// The fast kernels (see istft_fast_body).  Contiguous ranges of the global frame list, one wave of them: a range pays
// for `reach` lead-in frames, yet the wave lasts as long as one range, so fewer, longer ranges only leave SMs idle
// (8 signals of 332 frames, 4096 points, hop 1024: 55 ranges of 48 frames 110 us, 532 of 5 frames 69 us).
template <int M, int LAYOUT, int OVT, bool PLAIN = false, bool EXACT = PLAIN>
static ma_status launch_istft_fast(ma_fft_plan* plan, const C2RParams& p) {
    constexpr int T = FftPlan<M>::T;
    constexpr size_t smem = (size_t)IstftFastShape<M, OVT, PLAIN>::SMEM_BYTES;
    static int per_sm[64] = {0};
    ma_context* ctx = plan->ctx;
    int& occ = per_sm[ctx->device & 63];
    if (occ == 0) MA_TRY(occupancy(istft_fast_kernel<M, LAYOUT, OVT, PLAIN, EXACT>, T, smem, &occ));
    const int64_t total = p.frames_per_signal * p.n_signals, cap = (int64_t)ctx->sm_count * occ;
    istft_fast_kernel<M, LAYOUT, OVT, PLAIN, EXACT><<<(unsigned)(total < cap ? total : cap), T, smem, ctx->stream>>>(p);
    return after_launch(ctx);
}

template <int M>
static ma_status launch_istft_t(ma_fft_plan* plan, C2RParams& p) {
    constexpr int T = FftPlan<M>::T;
    const bool fast = istft_fast_ok<M>(p);
    if constexpr (plan_pairable<M>()) {
        if (fast && istft_plain<M>(p)) return launch_istft_fast<M, LAYOUT_HALF_PACKED, 2, true>(plan, p);
    }
    if constexpr (CtaShape<M>::FPC >= kRowsFromSlots) {
        const size_t rows_smem = istft_rows_smem<M>(p.hop);
        // The fast kernel's CTA is one frame's threads: less than a warp below 1024 points (256 points, hop 64: STFT and
        // iSTFT of 256 x 300000 samples 1800 us with it, 1423 us with the rows).  Only the plain overlap-add of
        // convolution blocks, which stages packed rows, is the faster one at any length.  Hops that the fast kernel
        // could serve there leave few enough rows for the limit (31 of 256 samples).
        if ((!fast || T < 32) && rows_smem <= kRowsSmemLimit) {
            return p.layout == LAYOUT_HALF_INTERLEAVED
                       ? launch_istft_rows<M, LAYOUT_HALF_INTERLEAVED>(plan, p, rows_smem, &plan->rows_occ[0])
                       : launch_istft_rows<M, -1>(plan, p, rows_smem, &plan->rows_occ[1]);
        }
    }
    if constexpr (plan_pairable<M>() && T >= 32) {
        // Overlap counts of 4 and, in the interleaved layout, 2 are fixed at compile time (register ring); hops that
        // do not divide the frame come in the interleaved layout only (istft_fast_ok).
        if (fast && 4 * p.hop == 2 * M) {
            if (p.layout == LAYOUT_HALF_INTERLEAVED) return launch_istft_fast<M, LAYOUT_HALF_INTERLEAVED, 4>(plan, p);
            if (p.layout == LAYOUT_HALF_PACKED) return launch_istft_fast<M, LAYOUT_HALF_PACKED, 4>(plan, p);
            return launch_istft_fast<M, LAYOUT_HALF_POLAR, 4>(plan, p);
        }
        if (fast) {
            if (p.layout == LAYOUT_HALF_PACKED) return launch_istft_fast<M, LAYOUT_HALF_PACKED, 0>(plan, p);
            if (p.layout == LAYOUT_HALF_POLAR) return launch_istft_fast<M, LAYOUT_HALF_POLAR, 0>(plan, p);
            if (p.hop == M) return launch_istft_fast<M, LAYOUT_HALF_INTERLEAVED, 2>(plan, p);
            if ((2 * M) % p.hop != 0) return launch_istft_fast<M, LAYOUT_HALF_INTERLEAVED, 0, false, true>(plan, p);
            return launch_istft_fast<M, LAYOUT_HALF_INTERLEAVED, 0>(plan, p);
        }
    }
    constexpr size_t smem = 2 * smem_elems_per_fft<M, 1>() * sizeof(float2) + 2 * M * sizeof(float);
    static int per_sm[64] = {0};
    ma_context* ctx = plan->ctx;
    int& occ = per_sm[ctx->device & 63];
    if (occ == 0) MA_TRY(occupancy(istft_kernel<M>, T, smem, &occ));
    // Chunks per signal: two waves of CTAs where the lead-in frames stay a small fraction of a chunk, at least
    // one wave in any case.
    const int64_t F = p.frames_per_signal, cap = (int64_t)ctx->sm_count * occ;
    const int reach = (2 * M + p.hop - 1) / p.hop - 1;
    const int64_t min_len = reach > 0 ? 16 * (int64_t)reach : 1;
    int64_t chunks = (2 * cap + p.n_signals - 1) / p.n_signals;
    if (chunks > F / min_len) chunks = F / min_len;
    if (chunks < cap / p.n_signals) chunks = cap / p.n_signals < F ? cap / p.n_signals : F;
    if (chunks < 1) chunks = 1;
    p.chunks_per_signal = (int32_t)chunks;
    const int64_t total = chunks * p.n_signals;
    istft_kernel<M><<<(unsigned)(total < cap ? total : cap), T, smem, ctx->stream>>>(p);
    return after_launch(ctx);
}

// One thread per position, each a chain of up to N/hop sums over independent loads.  As a host loop these sums kept
// the first iSTFT of a plan waiting; first call then and now: 8192 points, hop 1 127 -> 2.4 ms; hop 16 10.7 -> 2.8 ms;
// 4096 points, hop 64 0.92 -> 0.39 ms; hop 1024 (8 signals of 332 frames) 141 -> 73 us.
__global__ void __launch_bounds__(128) window_sum_edges_kernel(const float* __restrict__ window, int n, int hop, float floor,
                                                               float* __restrict__ edges) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i < 2 * n) edges[i] = window_sum_entry(window, i, n, hop, floor);
}

// Rebuilds the window-sum tables when the floor changes: the interior (host_tables.h) and its reciprocals on the
// host, the ends on the device.
static ma_status update_norm_table(ma_fft_plan* plan, int hop, float floor) {
    if (plan->norm_floor == floor) return MA_OK;
    window_sum_edges_kernel<<<(unsigned)((2 * plan->n + 127) / 128), 128, 0, plan->ctx->stream>>>(plan->d_window, plan->n, hop, floor,
                                                                                               plan->d_norm + 2 * hop);
    MA_TRY(after_launch(plan->ctx));
    std::vector<float> tab =
        make_norm_table(plan->h_window.empty() ? nullptr : plan->h_window.data(), plan->n, hop, floor);
    tab.resize(2 * (size_t)hop);
    for (int r = 0; r < hop; ++r) tab[(size_t)(hop + r)] = 1.0f / tab[(size_t)r];
    MA_CUDA(cudaMemcpyAsync(plan->d_norm, tab.data(), sizeof(float) * tab.size(), cudaMemcpyHostToDevice, plan->ctx->stream));
    MA_CUDA(cudaStreamSynchronize(plan->ctx->stream));
    plan->norm_floor = floor;
    return MA_OK;
}

ma_status launch_istft_small(ma_fft_plan* plan, C2RParams p) {
    p.twM = plan->d_twInv;
    p.twN = plan->d_twN;
    if (p.n_signals <= 0 || p.frames_per_signal <= 0) return MA_OK;
    if (!(p.window == nullptr && p.floor < 0.f)) {
        if (p.hop != plan->hop) return MA_ERR_INVALID_ARGUMENT;
        MA_TRY(update_norm_table(plan, p.hop, p.floor));
    }
    p.norm_mid = plan->d_norm;
    p.norm_mid_inv = plan->d_norm + plan->hop;
    p.norm_edge = plan->d_norm + 2 * plan->hop;
    p.window_syn = p.window != nullptr ? reinterpret_cast<const float4*>(plan->d_window_syn) : nullptr;
    p.error_flag = plan->ctx->d_error_flag;
    ma_status st = MA_ERR_UNSUPPORTED;
#define RUN(MM) st = launch_istft_t<MM>(plan, p);
    MA_DISPATCH_M(plan->m, RUN)
#undef RUN
    return st;
}

// Magnitude family over bins 0..N/2 of full-N split spectra.
__global__ void magnitude_kernel(const float* __restrict__ re, const float* __restrict__ im,
                                 float* __restrict__ out, int64_t batch, int n, int kind, float db_scale) {
    const int kh = n / 2 + 1;
    const int64_t total = batch * kh;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t g = i / kh;
        const int k = (int)(i - g * kh);
        const float2 x = make_float2(__ldg(re + g * n + k), __ldg(im + g * n + k));
        out[i] = mag_value(x, kind, db_scale);
    }
}

ma_status launch_magnitude(ma_fft_plan* plan, const float* re, const float* im, float* out, int64_t batch,
                           int kind, float db_scale) {
    ma_context* ctx = plan->ctx;
    const int64_t total = batch * (plan->n / 2 + 1);
    if (total <= 0) return MA_OK;
    int64_t want = (total + 255) / 256;
    int64_t cap = (int64_t)ctx->sm_count * 8;
    int grid = (int)(want < cap ? want : cap);
    magnitude_kernel<<<grid, 256, 0, ctx->stream>>>(re, im, out, batch, plan->n, kind, db_scale);
    return after_launch(ctx);
}

}  // namespace ma
