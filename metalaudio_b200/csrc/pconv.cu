// Uniformly partitioned overlap-add convolution with a frequency-domain delay line (FDL).
//
// Data in HBM (all float2, "packed" half spectra: B complex bins per 2B-point block, bin 0
// holding (DC, Nyquist)):
//   H     [n_irs][P][B]      partition spectra of every impulse response
//   ring  [C][P][B]          delay line of the last P input-block spectra per channel
//   tl    [C][P-1+T][B]      whole-signal call: history followed by all T block spectra
//   Y     [C][T][B]          whole-signal call: accumulated output spectra
// Kernels:
//   r2c (fft_small.cu)       input blocks -> spectra (zero-padded to 2B in the loader)
//   pconv_mac_kernel         Y[c] = sum_p X[c][t-p] * H[ir(c)][p]; streams the delay line once,
//                            channels that share an IR are tiled so each H element is loaded
//                            once per tile and reused from registers
//   c2r / istft (fft_small)  inverse transform + block overlap-add
#include <cuda_pipeline.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <new>
#include <type_traits>
#include <vector>

#include "bulk_copy.cuh"
#include "copy_threads.h"
#include "fft_plan.h"
#include "host_pipe.h"
#include "pconv_tiling.h"
#include "tensor_map.h"

struct ma_pconv {
    ma_context* ctx = nullptr;
    int block = 0;      // B
    int channels = 0;   // C
    ma_fft_plan* plan = nullptr;  // N = 2B
    int64_t taps = 0;
    int partitions = 0;  // P
    int n_irs = 0;
    int share = 1;       // channels per tile that share one IR (1, 2 or 4)
    float2* d_h = nullptr;
    int32_t* d_ch2ir = nullptr;
    float2* d_ring = nullptr;
    float* d_tail = nullptr;
    int write_index = 0;
    int splits = 1;              // partition splits of the streaming step
    float2* d_partial = nullptr; // [splits][C][B]
    int64_t reserved_len = 0;
    float2* d_timeline = nullptr;
    float2* d_y = nullptr;
    // Whole-signal calls that start on a clear delay line need not keep the caller's block size: they run on
    // a coarser partition of the same taps (whole_block), built by ma_pconv_reserve.  Where the caller's own
    // block is the better one, or the only one there is memory for, w_plan and d_hw are plan and d_h.
    std::unique_ptr<float[]> h_taps;  // [n_irs][taps_stride], from set_kernels until the coarse spectra and their buffers exist
    float* d_taps = nullptr;      // [n_irs][taps_stride], beside the coarse spectra (pconv_rescue_kernel)
    int32_t* d_marks = nullptr;   // [channels]: the call that last met a non-finite sample in the channel
    int32_t mark = 0;             // number of the latest coarse call
    int w_block = 0, w_partitions = 0;
    ma_fft_plan* w_plan = nullptr;
    float2* d_hw = nullptr;
    // float2 per channel of the coarse timeline.  The w_partitions - 1 rows in front of each channel's are zero, in stream
    // order, whenever no call is using the buffer otherwise (clear_prefix).
    int64_t w_stride = 0;
    bool clear = true;            // every delay-line spectrum a later call can reach, and the tail, are zero
    bool step_captured = false;   // a graph holds steps of this object: its replays fill the delay line unseen
};

namespace ma {

struct MacParams {
    const float2* x;        // delay line or timeline
    int64_t x_chan_stride;  // float2 units
    const float2* h;
    const int32_t* ch2ir;
    float2* out;
    int64_t out_split_stride, out_chan_stride, out_t_stride;  // float2 units
    int block;       // B
    int partitions;  // P
    int w0;          // slot of partition 0 for t = 0
    int wrap;        // P for the ring, 0 for the timeline
    int splits;
    int p_per_split;
    int bin_tiles;
    int bpt;         // threads covering one spectrum tile (power of two <= 128)
    int dependent_launch;  // streaming step: launched with programmatic stream serialization
    int cluster;           // CTAs per thread-block cluster along the splits (1: none): their partial sums are
                           // added up through distributed shared memory and rank 0 alone writes
};

constexpr int kMacThreads = 128;

template <int VEC>
struct VecT;
template <>
struct VecT<1> { using type = float2; };
template <>
struct VecT<2> { using type = float4; };

// One CTA: CT channels sharing an IR, one tile of bins, one range of partitions, one block
// index t (blockIdx.y).  Threads along bins (VEC bins each); when a spectrum tile needs fewer
// than 128 threads the remaining thread rows take interleaved partitions and are reduced
// through shared memory.  STREAM selects evict-first loads for the delay line (read once).
template <int CT, int VEC, bool STREAM>
__global__ void __launch_bounds__(kMacThreads) pconv_mac_kernel(const MacParams q) {
    using V = typename VecT<VEC>::type;
    __shared__ float2 red[kMacThreads * CT * VEC];
    if (q.dependent_launch) {  // streaming step: the new delay-line slot comes from the kernel before this one
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    const int tid = threadIdx.x;
    const int bpt = q.bpt;
    const int kb = tid & (bpt - 1);
    const int pl = tid / bpt;
    const int PL = kMacThreads / bpt;
    int bx = blockIdx.x;
    const int split = bx % q.splits;
    bx /= q.splits;
    const int bt = bx % q.bin_tiles;
    const int ctile = bx / q.bin_tiles;
    const int t = blockIdx.y;
    const int c0 = ctile * CT;
    const int e = (bt * bpt + kb) * VEC;  // first bin of this thread
    const bool dc = (e == 0);
    const int B = q.block;
    const int p_beg = split * q.p_per_split;
    int p_end = p_beg + q.p_per_split;
    if (p_end > q.partitions) p_end = q.partitions;

    const float2* hb = q.h + (int64_t)__ldg(q.ch2ir + c0) * q.partitions * B + e;
    const float2* xb = q.x + (int64_t)c0 * q.x_chan_stride + e;
    const int w = q.w0 + t;

    float2 acc[CT][VEC];
#pragma unroll
    for (int c = 0; c < CT; ++c)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[c][v] = make_float2(0.f, 0.f);

#pragma unroll 4
    for (int p = p_beg + pl; p < p_end; p += PL) {
        const V hv = __ldg(reinterpret_cast<const V*>(hb + (int64_t)p * B));
        float2 h[VEC];
        h[0] = make_float2(reinterpret_cast<const float*>(&hv)[0], reinterpret_cast<const float*>(&hv)[1]);
        if constexpr (VEC == 2)
            h[1] = make_float2(reinterpret_cast<const float*>(&hv)[2], reinterpret_cast<const float*>(&hv)[3]);
        // bin 0 carries (DC, Nyquist): component-wise product instead of a complex one
        const float ha = dc ? 0.f : h[0].y;
        const float hc = dc ? h[0].y : h[0].x;
        int slot = w - p;
        if (slot < 0) slot += q.wrap;
        const float2* xp = xb + (int64_t)slot * B;
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            const V* src = reinterpret_cast<const V*>(xp + (int64_t)c * q.x_chan_stride);
            V xv;
            if (STREAM) xv = __ldcs(src);
            else xv = __ldg(src);
            const float* xf = reinterpret_cast<const float*>(&xv);
            acc[c][0].x = fmaf(xf[0], h[0].x, acc[c][0].x);
            acc[c][0].x = fmaf(-xf[1], ha, acc[c][0].x);
            acc[c][0].y = fmaf(xf[0], ha, acc[c][0].y);
            acc[c][0].y = fmaf(xf[1], hc, acc[c][0].y);
            if constexpr (VEC == 2) {
                acc[c][1].x = fmaf(xf[2], h[1].x, acc[c][1].x);
                acc[c][1].x = fmaf(-xf[3], h[1].y, acc[c][1].x);
                acc[c][1].y = fmaf(xf[2], h[1].y, acc[c][1].y);
                acc[c][1].y = fmaf(xf[3], h[1].x, acc[c][1].y);
            }
        }
    }

    if (PL > 1) {
#pragma unroll
        for (int c = 0; c < CT; ++c)
#pragma unroll
            for (int v = 0; v < VEC; ++v) red[(c * VEC + v) * kMacThreads + tid] = acc[c][v];
        __syncthreads();
        if (pl == 0) {
            for (int r = 1; r < PL; ++r) {
#pragma unroll
                for (int c = 0; c < CT; ++c)
#pragma unroll
                    for (int v = 0; v < VEC; ++v) {
                        const float2 o = red[(c * VEC + v) * kMacThreads + r * bpt + kb];
                        acc[c][v].x += o.x;
                        acc[c][v].y += o.y;
                    }
            }
        }
    }
    int out_split = split;
    bool writer = pl == 0;
    if (q.cluster > 1) {
        // The cluster's CTAs hold consecutive splits of one tile.  Each leaves its sums in its own shared
        // memory; after the cluster barrier rank 0 adds the others' in rank order (a fixed order: results
        // do not depend on timing) through distributed shared memory and writes one partial spectrum for
        // the whole cluster.  The second barrier keeps every CTA's shared memory alive until rank 0 has
        // read it.  Cluster barriers are hardware barriers among co-scheduled CTAs, not spin waits.
        uint32_t rank;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        if (PL > 1) __syncthreads();  // the intra-CTA reduction above is done with `red`
        if (pl == 0) {
#pragma unroll
            for (int c = 0; c < CT; ++c)
#pragma unroll
                for (int v = 0; v < VEC; ++v) red[(c * VEC + v) * kMacThreads + tid] = acc[c][v];
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank == 0 && pl == 0) {
            for (int r = 1; r < q.cluster; ++r) {
#pragma unroll
                for (int c = 0; c < CT; ++c)
#pragma unroll
                    for (int v = 0; v < VEC; ++v) {
                        const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(&red[(c * VEC + v) * kMacThreads + tid]));
                        uint32_t remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(r));
                        float2 o;
                        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(o.x), "=f"(o.y) : "r"(remote) : "memory");
                        acc[c][v].x += o.x;
                        acc[c][v].y += o.y;
                    }
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        writer = pl == 0 && rank == 0;
        out_split = split / q.cluster;
    }
    if (writer) {
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            float2* o = q.out + (int64_t)out_split * q.out_split_stride + (int64_t)(c0 + c) * q.out_chan_stride +
                        (int64_t)t * q.out_t_stride + e;
#pragma unroll
            for (int v = 0; v < VEC; ++v) o[v] = acc[c][v];
        }
    }
}

// Whole-signal form of the same multiply-accumulate, tiled over time.  With every block
// spectrum of the call already in the timeline, output blocks are independent, and TT consecutive
// outputs of one (channel, bin) reuse the same partition spectra: a thread keeps TT accumulators
// and a sliding window of TT timeline values in registers, and per partition takes ONE new
// timeline value and ONE partition value for TT complex multiply-accumulates (4*TT FMAs).
// A CTA is 4 warps = 4 consecutive time tiles of one channel and 32 bins (lanes along bins).
// Its warps need the same partition rows and overlapping timeline rows, so both are staged in
// shared memory by 16-byte asynchronous copies, a chunk of TT partitions ahead: the timeline
// rows in a ring of 128 rows (each row enters once per CTA), the partition rows double-buffered.
// That leaves about 0.25 byte of L2 traffic per complex multiply-accumulate and makes the FMA
// pipe the limiter.  One barrier per chunk (1024 FMAs per thread apart).
// A complex product is two packed two-wide multiply-adds into two component-wise sums: no operand has to be
// swapped or negated (32 partitions of 4096 bins, 512 channels x 288 blocks: 4.33 -> 4.0 ms against sums
// of complex products, for which the swapped rows were rebuilt at every use).
// TWO_LEVEL: every kFlushChunks chunks the running sums are added into a second set of
// accumulators and cleared, so no float32 sum runs over more than TT*kFlushChunks partitions
// (blocked summation: the rounding error of thousands of partitions grows with the block
// length, not with the partition count).
constexpr int kFlushChunks = 16;
template <int TT, bool TWO_LEVEL>
__global__ void __launch_bounds__(128) pconv_mac_tiled_kernel(const MacParams q, int t_total, int64_t tl_len) {
    using TL = MacTiling<TT>;
    constexpr int RING = TL::kRing;
    __shared__ __align__(16) float2 xs[RING][32];
    __shared__ __align__(16) float2 hs[2][TT][32];
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int B = q.block, P = q.partitions;
    const int bin_tiles = B >> 5;
    const int bt = blockIdx.x % bin_tiles;
    const int c = blockIdx.x / bin_tiles;
    const bool dc = (bt == 0 && lane == 0);
    const int t0_cta = blockIdx.y * 4 * TT;
    if (t0_cta >= t_total) return;
    const float2* xc = q.x + (int64_t)c * q.x_chan_stride + bt * 32;
    const float2* hc = q.h + (int64_t)__ldg(q.ch2ir + c) * P * B + bt * 32;
    const int64_t base0 = TL::base0(P, t0_cta);          // timeline row of the CTA's first output at p = 0
    const int64_t base = base0 + warp * TT;              // ... of this warp's first output

    // 16-byte copies: a row of 32 bins is 16 segments
    auto load_x_rows = [&](int64_t first, int count) {
        for (int idx = tid; idx < count * 16; idx += 128) {
            const int64_t row = first + (idx >> 4);
            const int seg = idx & 15;
            const int64_t src = TL::fetch_row(row, tl_len);  // clamped into the channel's own timeline
            __pipeline_memcpy_async(&xs[row & (RING - 1)][seg * 2], xc + src * B + seg * 2, 16);
        }
    };
    auto load_h_rows = [&](int buf, int p0) {
        for (int idx = tid; idx < TT * 16; idx += 128) {
            const int pr = p0 + (idx >> 4);
            const int seg = idx & 15;
            if (pr < P) __pipeline_memcpy_async(&hs[buf][idx >> 4][seg * 2], hc + (int64_t)pr * B + seg * 2, 16);
        }
    };

    load_x_rows(TL::chunk0_first(P, t0_cta), TL::kChunk0Rows);  // rows of chunk 0: [base0-TT+1, base0+4TT-1]
    load_h_rows(0, 0);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();

    // x*h as two component-wise sums, ar = sum (xr, xi) * hr and ai = sum (xr, xi) * hi; re = ar.x - ai.y and
    // im = ar.y + ai.x at the end.  Packed operands are used as they lie in the window.
    float2 ar[TT], ai[TT], xw[TT];
    float2 acc2[TWO_LEVEL ? TT : 1];
#pragma unroll
    for (int i = 0; i < TT; ++i) {
        ar[i] = make_float2(0.f, 0.f);
        ai[i] = make_float2(0.f, 0.f);
        if constexpr (TWO_LEVEL) acc2[i] = make_float2(0.f, 0.f);
        xw[i] = xs[(base + i) & (RING - 1)][lane];
    }
    int buf = 0;
    int since_flush = 0;
    for (int p0 = 0; p0 < P; p0 += TT) {
        if (p0 + TT < P) {  // stage the next chunk while this one is consumed
            load_x_rows(TL::lookahead_first(P, t0_cta, p0), TT);
            load_h_rows(buf ^ 1, p0 + TT);
        }
        __pipeline_commit();
        // one chunk of TT partitions; FULL: all of them exist, so no per-partition test
        auto chunk = [&](auto full) {
            constexpr bool FULL = decltype(full)::value;
            const float2* hrow = &hs[buf][0][lane];
#pragma unroll
            for (int j = 0; j < TT; ++j) {
                const int p = p0 + j;
                if (FULL || p < P) {
                    // slot (i - j) mod TT holds timeline row base + i - p; the row base - p enters at i = 0
                    if (j > 0 || p0 > 0) xw[(TT - j) % TT] = xs[(base - p) & (RING - 1)][lane];
                    const float2 h = hrow[j * 32];
                    const float hi = dc ? 0.f : h.y;   // bin 0 carries (DC, Nyquist): component-wise product
                    const float2 hr2 = make_float2(h.x, dc ? h.y : h.x), hi2 = make_float2(hi, hi);
#pragma unroll
                    for (int i = 0; i < TT; ++i) {
                        ar[i] = pfma(xw[(i - j + TT) % TT], hr2, ar[i]);
                        ai[i] = pfma(xw[(i - j + TT) % TT], hi2, ai[i]);
                    }
                }
            }
        };
        if (p0 + TT <= P) chunk(std::true_type{});
        else chunk(std::false_type{});
        if constexpr (TWO_LEVEL) {
            if (++since_flush == kFlushChunks) {
                since_flush = 0;
#pragma unroll
                for (int i = 0; i < TT; ++i) {
                    acc2[i].x += ar[i].x - ai[i].y;
                    acc2[i].y += ar[i].y + ai[i].x;
                    ar[i] = make_float2(0.f, 0.f);
                    ai[i] = make_float2(0.f, 0.f);
                }
            }
        }
        __pipeline_wait_prior(0);
        __syncthreads();
        buf ^= 1;
    }
    const int t0 = t0_cta + warp * TT;
    float2* o = q.out + (int64_t)c * q.out_chan_stride + (int64_t)t0 * q.out_t_stride + bt * 32 + lane;
#pragma unroll
    for (int i = 0; i < TT; ++i)
        if (t0 + i < t_total) {
            float2 y = make_float2(ar[i].x - ai[i].y, ar[i].y + ai[i].x);
            if constexpr (TWO_LEVEL) y = make_float2(y.x + acc2[i].x, y.y + acc2[i].y);
            o[(int64_t)i * q.out_t_stride] = y;
        }
}

// The same for few partitions (the coarse whole-signal calls: 8 to 64), where the kernel above spends as many
// instructions on staging its ring as on products.  Everything a CTA reads fits shared memory at once: the
// 16 * warps + P - 1 timeline rows and the P partition rows of its 32 bins, each one box of a tensor map that one
// thread asks the TMA unit for.  Rows behind the timeline arrive as zeros; they feed outputs that are not
// stored.  Neighbouring CTAs are neighbouring time tiles, so the rows they share come from L2.  32 partitions of
// 4096 bins, 512 channels x 288 blocks: 4.00 -> 3.17 ms (1.2e13 of the 1.9e13 products per second the FMA pipe allows).
struct MacBoxParams {
    const int32_t* ch2ir;
    float2* out;
    int64_t out_chan_stride, out_t_stride;  // float2 units
    int bin_tiles, partitions, t_tiles, t_total;
    int32_t* error_flag;
};
constexpr int kBoxMostPartitions = 64;

// Partitions J .. TT-1 of a chunk; the row that enters the window for the next one is fetched under the products.
template <int J, class Products, int TT>
__device__ __forceinline__ void box_chunk(const Products& products, const float2* hrow, const float2* xnew, float2 (&xw)[TT]) {
    const float2 x_next = xnew[-(J + 1) * 32];
    products(hrow[J * 32], std::integral_constant<int, J>{});
    xw[TT - 1 - J] = x_next;
    if constexpr (J + 1 < TT) box_chunk<J + 1>(products, hrow, xnew, xw);
}

template <int TT>
__global__ void __launch_bounds__(128, 4) pconv_mac_box_kernel(const MacBoxParams q, const __grid_constant__ CUtensorMap x_map,
                                                               const __grid_constant__ CUtensorMap h_map) {
    extern __shared__ __align__(128) float2 box_smem[];
    __shared__ uint64_t bar;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int P = q.partitions, rows = warps * TT + P - 1;
    // a spare row in front: the last partition's look-ahead reads it and drops the value
    float2* const xs = box_smem + 32;          // [rows][32]: timeline rows t0_cta ..
    float2* const hs = xs + rows * 32;         // [P][32]
    unsigned blk = blockIdx.x;
    const int t_tile = (int)(blk % (unsigned)q.t_tiles);
    blk /= (unsigned)q.t_tiles;
    const int bt = (int)(blk % (unsigned)q.bin_tiles), c = (int)(blk / (unsigned)q.bin_tiles);
    const int t0_cta = t_tile * warps * TT;
    if (threadIdx.x == 0) {
        bulk_barrier_init(&bar);
        bulk_barrier_expect(&bar, (uint32_t)((rows + P) * 32 * sizeof(float2)));
        bulk_tensor_load_3d(xs, &x_map, bt * 64, t0_cta, c, &bar);
        bulk_tensor_load_3d(hs, &h_map, bt * 64, 0, __ldg(q.ch2ir + c), &bar);
    }
    __syncthreads();  // the barrier is initialised before anyone polls it
    if (!bulk_barrier_wait(&bar, 0)) *q.error_flag = 1;
    const bool dc = bt == 0 && lane == 0;
    const float2* xrow = xs + (P - 1 + warp * TT) * 32 + lane;  // row of this warp's first output at p = 0
    float2 ar[TT], ai[TT], xw[TT];
#pragma unroll
    for (int i = 0; i < TT; ++i) {
        ar[i] = make_float2(0.f, 0.f);
        ai[i] = make_float2(0.f, 0.f);
        xw[i] = xrow[i * 32];
    }
    auto products = [&](const float2 h, auto rotation) {
        constexpr int J = decltype(rotation)::value;
        const float hi = dc ? 0.f : h.y;  // bin 0 carries (DC, Nyquist): component-wise product
        const float2 hr2 = make_float2(h.x, dc ? h.y : h.x), hi2 = make_float2(hi, hi);
#pragma unroll
        for (int i = 0; i < TT; ++i) {
            ar[i] = pfma(xw[(i - J + TT) % TT], hr2, ar[i]);
            ai[i] = pfma(xw[(i - J + TT) % TT], hi2, ai[i]);
        }
    };
    // whole chunks of TT partitions: the window rotates through the registers
    int p = 0;
#pragma unroll 1
    for (; p + TT <= P; p += TT) {
        const float2* hrow = hs + p * 32 + lane;
        const float2* xnew = xrow - p * 32;
        box_chunk<0>(products, hrow, xnew, xw);
    }
    // the remainder: the window moves up by registers
#pragma unroll 1
    for (; p < P; ++p) {
        products(hs[p * 32 + lane], std::integral_constant<int, 0>{});
#pragma unroll
        for (int i = TT - 1; i > 0; --i) xw[i] = xw[i - 1];
        xw[0] = xrow[-(p + 1) * 32];
    }
    const int t0 = t0_cta + warp * TT;
    float2* o = q.out + (int64_t)c * q.out_chan_stride + (int64_t)t0 * q.out_t_stride + bt * 32 + lane;
#pragma unroll
    for (int i = 0; i < TT; ++i) {
        if (t0 + i < q.t_total) *o = make_float2(ar[i].x - ai[i].y, ar[i].y + ai[i].x);
        o += q.out_t_stride;
    }
}

constexpr int kTwoLevelFrom = 2048;

// Launches the box kernel; MA_ERR_UNSUPPORTED when these parameters are not its (see launch_mac_tiled).
static ma_status launch_mac_box(ma_pconv* pc, const MacParams& q, int channels, int64_t t_count, int64_t tl_len) {
    constexpr int TT = 16;
    ma_context* ctx = pc->ctx;
    if (q.partitions > kBoxMostPartitions || q.block % 32 != 0 || tl_len > (int64_t)1 << 30) return MA_ERR_UNSUPPORTED;
    // Warps per CTA: four, or fewer where that leaves less of the last time tile empty.
    int warps = 4;
    auto padded = [&](int w) { return (t_count + w * TT - 1) / (w * TT) * (w * TT); };
    for (int w = 3; w >= 1; --w)
        if (padded(w) * 16 < padded(warps) * 15) warps = w;
    const int64_t t_tiles = padded(warps) / (warps * TT), grid = t_tiles * (q.block / 32) * channels;
    if (grid > 0x7fffffff) return MA_ERR_UNSUPPORTED;
    const int rows = warps * TT + q.partitions - 1;
    CUtensorMap xm, hm;
    if (!tile_tensor_map(reinterpret_cast<const float*>(q.x), 2 * q.block, tl_len, channels, 2 * q.x_chan_stride, 64, rows, &xm) ||
        !tile_tensor_map(reinterpret_cast<const float*>(q.h), 2 * q.block, q.partitions, pc->n_irs, 2 * (int64_t)q.partitions * q.block, 64,
                         q.partitions, &hm))
        return MA_ERR_UNSUPPORTED;
    MacBoxParams b{};
    b.ch2ir = q.ch2ir;
    b.out = q.out;
    b.out_chan_stride = q.out_chan_stride;
    b.out_t_stride = q.out_t_stride;
    b.bin_tiles = q.block / 32;
    b.partitions = q.partitions;
    b.t_tiles = (int)t_tiles;
    b.t_total = (int)t_count;
    b.error_flag = ctx->d_error_flag;
    const size_t smem = (size_t)(rows + q.partitions + 1) * 32 * sizeof(float2);
    static std::atomic<bool> raised[64];
    if (!raised[ctx->device & 63].load(std::memory_order_acquire)) {
        const int most = (4 * TT + 2 * kBoxMostPartitions) * 32 * (int)sizeof(float2);
        MA_CUDA(cudaFuncSetAttribute(pconv_mac_box_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        raised[ctx->device & 63].store(true, std::memory_order_release);
    }
    pconv_mac_box_kernel<TT><<<(unsigned)grid, warps * 32, smem, ctx->stream>>>(b, xm, hm);
    return after_launch(ctx);
}

static ma_status launch_mac_tiled(ma_pconv* pc, const MacParams& q, int channels, int64_t t_count, int64_t tl_len) {
    constexpr int TT = 16;
    ma_context* ctx = pc->ctx;
    const ma_status boxed = launch_mac_box(pc, q, channels, t_count, tl_len);
    if (boxed != MA_ERR_UNSUPPORTED) return boxed;
    const int bin_tiles = q.block >> 5;
    const int64_t t_ctas = (t_count + 4 * TT - 1) / (4 * TT);
    int64_t done = 0;
    while (done < t_ctas) {  // grid.y limit
        int64_t ny = t_ctas - done;
        if (ny > 32768) ny = 32768;
        MacParams qq = q;
        const int64_t t_first = done * 4 * TT;
        qq.out = q.out + t_first * q.out_t_stride;
        qq.x = q.x + t_first * q.block;  // shifts the timeline origin by t_first rows
        dim3 grid((unsigned)(bin_tiles * channels), (unsigned)ny, 1);
        // Blocked summation once a running sum would cover more than kTwoLevelFrom partitions.
        if (q.partitions >= kTwoLevelFrom)
            pconv_mac_tiled_kernel<TT, true><<<grid, 128, 0, ctx->stream>>>(qq, (int)(t_count - t_first), tl_len - t_first);
        else
            pconv_mac_tiled_kernel<TT, false><<<grid, 128, 0, ctx->stream>>>(qq, (int)(t_count - t_first), tl_len - t_first);
        MA_TRY(after_launch(ctx));
        done += ny;
    }
    return MA_OK;
}

template <int CT, int VEC, bool STREAM>
static ma_status launch_mac_t(ma_context* ctx, const MacParams& q, int chan_tiles, int64_t t_count) {
    int64_t done = 0;
    while (done < t_count) {
        int64_t ny = t_count - done;
        if (ny > 32768) ny = 32768;
        MacParams qq = q;
        qq.w0 = q.w0 + (int)done;
        qq.out = q.out + done * q.out_t_stride;
        dim3 grid((unsigned)(chan_tiles * q.bin_tiles * q.splits), (unsigned)ny, 1);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kMacThreads);
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[2];
        int n_attr = 0;
        if (q.dependent_launch) {
            attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
            ++n_attr;
        }
        if (q.cluster > 1) {  // consecutive splits of a tile (consecutive blockIdx.x) form a cluster
            attr[n_attr].id = cudaLaunchAttributeClusterDimension;
            attr[n_attr].val.clusterDim.x = (unsigned)q.cluster;
            attr[n_attr].val.clusterDim.y = 1;
            attr[n_attr].val.clusterDim.z = 1;
            ++n_attr;
        }
        cfg.attrs = attr;
        cfg.numAttrs = n_attr;
        (void)cudaLaunchKernelEx(&cfg, pconv_mac_kernel<CT, VEC, STREAM>, qq);  // an error is picked up by after_launch
        MA_TRY(after_launch(ctx));
        done += ny;
    }
    return MA_OK;
}

static ma_status launch_mac(ma_pconv* pc, MacParams q, int channels, bool stream, int64_t t_count) {
    const int B = q.block;
    const int vec = B >= 2 ? 2 : 1;
    const int bp = B / vec;  // threads per spectrum
    q.bpt = bp < kMacThreads ? bp : kMacThreads;
    q.bin_tiles = bp / q.bpt;
    const int ct = pc->share;
    const int chan_tiles = channels / ct;
    ma_context* ctx = pc->ctx;
#define MAC_CASE(CT_, VEC_)                                                                        \
    if (ct == CT_ && vec == VEC_)                                                                  \
        return stream ? launch_mac_t<CT_, VEC_, true>(ctx, q, chan_tiles, t_count)                 \
                      : launch_mac_t<CT_, VEC_, false>(ctx, q, chan_tiles, t_count);
    MAC_CASE(1, 1) MAC_CASE(2, 1) MAC_CASE(4, 1) MAC_CASE(1, 2) MAC_CASE(2, 2) MAC_CASE(4, 2)
#undef MAC_CASE
    return MA_ERR_UNSUPPORTED;
}

// Streaming step with many partition splits: adds the partial spectra up, split 0 first, and
// leaves the total in slot 0, one thread per 16 bytes with eight loads in flight.  The inverse
// transform behind it then reads one spectrum per channel; walking `splits` partials inside that
// kernel costs a memory round trip per partial on a handful of CTAs, which with few channels per
// GPU (many splits) was the longest part of a step.  Same summation order as that walk.
__global__ void __launch_bounds__(256) pconv_sum_partials_kernel(float4* __restrict__ partial, int64_t n4,
                                                                 int64_t split_stride4, int splits) {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the multiply-accumulate before this kernel has finished
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n4) return;
    float4 acc = __ldcg(partial + i);
#pragma unroll 8
    for (int sp = 1; sp < splits; ++sp) {
        const float4 v = __ldcg(partial + sp * split_stride4 + i);
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
    }
    partial[i] = acc;
}

// Thread-block cluster size of the streaming step's multiply-accumulate: with many partition splits, groups
// of eight (four, two) consecutive splits reduce their sums on chip and write one partial spectrum.
static int step_cluster(int splits) {
    // Measured (block 256, 512 partitions): 16 / 64 / 128 channels 21.4 / 27.4 / 35.3 -> 14.8 / 24.1 / 33.4 us
    // per step; below 16 splits (256 channels and more) clusters cost 2-4 %, so those keep one CTA each.
    if (splits < 16) return 1;
    for (int s : {8, 4, 2})
        if (splits % s == 0) return s;
    return 1;
}

// Partial spectra are summed by their own kernel from this many splits up.
constexpr int kSumKernelFromSplits = 16;  // measured: 9 splits are faster summed inside the inverse kernel, 19 and 37 by this one

// Ordered copies between the ring and the timeline.
// to_timeline: tl[c][j] = ring[c][(w - (P-1-j)) mod P], j < P-1.
// to_ring:     ring[c][j] = tl[c][first + j], j < P.
__global__ void pconv_history_kernel(float2* __restrict__ ring, float2* __restrict__ tl, int64_t tl_chan_stride,
                                     int P, int B, int w, int64_t first, int to_timeline, int channels) {
    const int rows = to_timeline ? P - 1 : P;
    const int64_t total = (int64_t)channels * rows * B;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % B);
        const int64_t r = i / B;
        const int j = (int)(r % rows);
        const int64_t c = r / rows;
        if (to_timeline) {
            int slot = w - (P - 1 - j);
            slot %= P;
            if (slot < 0) slot += P;
            tl[c * tl_chan_stride + (int64_t)j * B + k] = ring[(c * P + slot) * B + k];
        } else {
            ring[(c * P + j) * B + k] = tl[c * tl_chan_stride + (first + j) * B + k];
        }
    }
}

// Largest block of the whole-signal calls: 8192-point transforms, the longest that fit shared memory.
constexpr int kWholeBlock = 4096;
constexpr int kWholePartitions = 8;

static void free_signal_buffers(ma_pconv* pc) {
    if (pc->d_timeline) (void)cudaFree(pc->d_timeline);
    if (pc->d_y) (void)cudaFree(pc->d_y);
    pc->d_timeline = nullptr;
    pc->d_y = nullptr;
    pc->reserved_len = 0;
}

static int64_t taps_stride(int64_t taps) { return (taps + 3) & ~(int64_t)3; }

// Partition spectra: the taps are the "signals", partitions the "frames" at hop `block`, each
// frame's samples beyond `block` (and beyond the end of the response) read as zero.
static ma_status partition_spectra(ma_pconv* pc, ma_fft_plan* plan, const float* d_taps, int block, int partitions, float2* h) {
    R2CParams p{};
    p.in = d_taps;
    p.signal_stride = taps_stride(pc->taps);
    p.frames_per_signal = partitions;
    p.total_frames = (int64_t)partitions * pc->n_irs;
    p.signal_len = pc->taps;
    p.hop = block;
    p.frame_valid = block;
    p.out_a = reinterpret_cast<float*>(h);
    p.out_signal_stride = (int64_t)partitions * block;
    p.out_frame_stride = block;
    p.layout = LAYOUT_HALF_PACKED;
    p.mag_kind = MAG_NONE;
    return launch_r2c_small(plan, p);
}

// The taps on the device, rows taps_stride apart: the host copy as one transfer, or the caller's rows.
static ma_status upload_taps(ma_pconv* pc, const float* irs, float* d_taps) {
    const int64_t stride = taps_stride(pc->taps);
    if (pc->h_taps != nullptr) return copy_h2d(pc->ctx, d_taps, pc->h_taps.get(), sizeof(float) * (size_t)(stride * pc->n_irs));
    for (int i = 0; i < pc->n_irs; ++i)
        MA_TRY(copy_h2d(pc->ctx, d_taps + i * stride, irs + i * pc->taps, sizeof(float) * (size_t)pc->taps));
    return MA_OK;
}

static void free_coarse(ma_pconv* pc) {
    if (pc->w_plan && pc->w_plan != pc->plan) (void)ma_fft_plan_destroy(pc->w_plan);
    if (pc->d_hw && pc->d_hw != pc->d_h) (void)cudaFree(pc->d_hw);
    if (pc->d_taps) (void)cudaFree(pc->d_taps);
    if (pc->d_marks) (void)cudaFree(pc->d_marks);
    pc->w_plan = nullptr;
    pc->d_hw = nullptr;
    pc->d_taps = nullptr;
    pc->d_marks = nullptr;
}

// Block size of whole-signal calls.  The multiply-accumulate costs one complex product per output bin and
// partition, i.e. it shrinks with the number of partitions, while the transforms' cost per sample hardly
// depends on their length up to 8192 points.  The shorter sums also round less, which pays for the longer
// transforms' rounding as long as there are sums to shorten: at least kWholePartitions partitions stay.
// Measured, 512 channels x 2^20 samples, 131072 taps: 512 partitions of 256 samples 64.2 ms, error 4.4e-7; 64 of 2048
// samples 10.4 ms (transforms 3.4, products 7.1), 2.9e-7; 32 of 4096 samples 8.7 ms (4.2, 4.3), 2.7e-7.
static int whole_block(int block, int64_t taps) {
    int b = block;
    while (b < kWholeBlock && 2 * (int64_t)b * kWholePartitions <= taps) b *= 2;
    return b;
}

// ---- non-finite samples in a coarse whole-signal call
//
// A transform turns one non-finite sample into a non-finite block, so on the coarse partition (blocks of W, PW of them)
// output block j is lost when input blocks j - PW .. j hold one, on the caller's own (B, P) when blocks j - P .. j do.
// Outputs that only the coarse blocks lose are computed here from the samples themselves, so that such a sample spoils
// what it always did.  The forward transforms mark the channels they met one in; without a mark the kernel returns after
// a look at the marks.  It costs such a call 1.5 us, launched early behind the inverse transform (4 us plainly).  A
// marked channel costs a scan of its samples and `taps` multiply-adds for each of at most 3 W outputs per non-finite
// sample: 512 channels x 2^20 samples, 131072 taps 7.3 ms clean, 9.3 ms with one such sample, 131 ms with one in every
// channel (the caller's own block of 256 takes 64 ms in every case).
struct RescueParams {
    const float* in;
    int64_t len, in_stride;
    const float* taps;           // [n_irs][taps_stride]
    int64_t n_taps, taps_stride;
    const int32_t* ch2ir;
    float* out;
    int64_t out_stride, full;
    const int32_t* marks;        // [channels]: `mark` where this call met a non-finite sample
    int32_t mark;
    int channels;
    int block, coarse;           // B, W (both powers of two, B <= W)
    int64_t reach, coarse_reach; // P * B, PW * W
};
constexpr int kRescueThreads = 256, kRescueOutputs = 4 * kRescueThreads, kRescueTaps = 256;
constexpr int kRescueWords = (kRescueOutputs + kWholeBlock) / 32;

__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }

__global__ void __launch_bounds__(kRescueThreads) pconv_rescue_kernel(const RescueParams p) {
    __shared__ uint32_t bad[kRescueWords];   // samples from the chunk's first output position on
    __shared__ int64_t before;               // the last non-finite sample in front of it, or -1
    __shared__ __align__(16) float xs[kRescueOutputs + kRescueTaps];
    __shared__ __align__(16) float hs[kRescueTaps];
    const int tid = threadIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // launched behind the inverse transform (programmatic)
    bool mine = false;
    for (int c = tid; c < p.channels; c += kRescueThreads) mine |= p.marks[c] == p.mark;
    if (!__syncthreads_or(mine)) return;
    const int64_t chunks = (p.full + kRescueOutputs - 1) / kRescueOutputs;
    for (int c = 0; c < p.channels; ++c) {
        if (p.marks[c] != p.mark) continue;
        const float* x = p.in + c * p.in_stride;
        const float* h = p.taps + (int64_t)p.ch2ir[c] * p.taps_stride;
        // channels that lose the same positions, as when all stop at once, still meet different CTAs
        for (int64_t chunk = (blockIdx.x + 61u * (unsigned)c) % gridDim.x; chunk < chunks; chunk += gridDim.x) {
            const int64_t o0 = chunk * kRescueOutputs;
            const int64_t last_o = (o0 + kRescueOutputs < p.full ? o0 + kRescueOutputs : p.full) - 1;
            // samples that the chunk's coarse blocks depend on: [lo, o0) and [o0, hi)
            const int64_t lo = (o0 & -(int64_t)p.coarse) - p.coarse_reach;
            const int64_t hi = (last_o & -(int64_t)p.coarse) + p.coarse;
            __syncthreads();  // the previous chunk's readers are done
            if (tid == 0) before = -1;
            for (int w = tid; w < kRescueWords; w += kRescueThreads) bad[w] = 0;
            __syncthreads();
            int64_t last = -1;
            for (int64_t s = (lo > 0 ? lo : 0) + tid; s < hi && s < p.len; s += kRescueThreads) {
                if (!not_finite(x[s])) continue;
                if (s < o0) last = s;
                else atomicOr(&bad[(s - o0) >> 5], 1u << ((s - o0) & 31));
            }
            if (last >= 0) atomicMax((long long*)&before, (long long)last);
            __syncthreads();
            // the last non-finite sample in front of `end`, which lies in (o0, hi]
            auto last_before = [&](int64_t end) {
                int bits = (int)(end - o0);
                int w = (bits - 1) >> 5;
                uint32_t word = bad[w] & (0xffffffffu >> (31 - ((bits - 1) & 31)));
                while (word == 0 && w > 0) word = bad[--w];
                return word != 0 ? o0 + 32 * w + 31 - __clz(word) : before;
            };
            bool need[4], any = false;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int64_t o = o0 + 4 * tid + r;
                need[r] = false;
                if (o < p.full) {
                    const int64_t j = o & -(int64_t)p.coarse, i = o & -(int64_t)p.block;
                    const int64_t lost = last_before(j + p.coarse), lost_anyway = last_before(i + p.block);
                    need[r] = lost >= 0 && lost >= j - p.coarse_reach && !(lost_anyway >= 0 && lost_anyway >= i - p.reach);
                }
                any |= need[r];
            }
            if (!__syncthreads_or(any)) continue;
            double sum[4] = {0.0, 0.0, 0.0, 0.0};
            for (int64_t n0 = 0; n0 < p.n_taps && n0 <= last_o; n0 += kRescueTaps) {
                const int count = p.n_taps - n0 < kRescueTaps ? (int)(p.n_taps - n0) : kRescueTaps;
                __syncthreads();
                if (tid < count) hs[tid] = h[n0 + tid];
                const int64_t first = o0 - n0 - kRescueTaps;  // sample of xs[0]
                for (int k = tid; k < kRescueOutputs + kRescueTaps; k += kRescueThreads) {
                    const int64_t s = first + k;
                    xs[k] = s >= 0 && s < p.len ? x[s] : 0.f;
                }
                __syncthreads();
                float part[4] = {0.f, 0.f, 0.f, 0.f};
                const float* const xo = xs + kRescueTaps + 4 * tid;  // output 4*tid at tap 0
                float4 hi4 = *reinterpret_cast<const float4*>(xo);
                int n = 0;
                for (; n + 4 <= count; n += 4) {  // a window of eight samples: four outputs, four taps
                    const float4 lo4 = *reinterpret_cast<const float4*>(xo - n - 4), h4 = *reinterpret_cast<const float4*>(hs + n);
                    const float win[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        part[r] = fmaf(h4.x, win[4 + r], part[r]);
                        part[r] = fmaf(h4.y, win[3 + r], part[r]);
                        part[r] = fmaf(h4.z, win[2 + r], part[r]);
                        part[r] = fmaf(h4.w, win[1 + r], part[r]);
                    }
                    hi4 = lo4;
                }
                for (; n < count; ++n) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) part[r] = fmaf(hs[n], xo[r - n], part[r]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) sum[r] += (double)part[r];
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (need[r]) p.out[c * p.out_stride + o0 + 4 * tid + r] = (float)sum[r];
        }
    }
}

// Without the memory for more the caller's own block size serves the whole-signal calls.
static void use_own_block(ma_pconv* pc) {
    free_coarse(pc);
    pc->w_block = pc->block;
    pc->w_partitions = pc->partitions;
    pc->w_plan = pc->plan;
    pc->d_hw = pc->d_h;
}

// Plan and partition spectra of the whole-signal calls; MA_ERR_ALLOC without the memory for them.
static ma_status build_coarse(ma_pconv* pc) {
    ma_context* ctx = pc->ctx;
    pc->w_block = whole_block(pc->block, pc->taps);
    pc->w_partitions = (int)((pc->taps + pc->w_block - 1) / pc->w_block);
    if (pc->w_block == pc->block || pc->h_taps == nullptr) {
        use_own_block(pc);
        return MA_OK;
    }
    ma_status st = fault_at(ctx, MA_FAULT_RESERVE_SPECTRA);
    if (st == MA_OK) st = ma_fft_plan_create(ctx, 2 * pc->w_block, nullptr, pc->w_block, &pc->w_plan);
    if (st == MA_OK) {
        cudaError_t e = cudaMalloc((void**)&pc->d_hw, sizeof(float2) * (size_t)pc->w_partitions * pc->w_block * (size_t)pc->n_irs);
        if (e == cudaSuccess) e = cudaMalloc((void**)&pc->d_taps, sizeof(float) * (size_t)(taps_stride(pc->taps) * pc->n_irs));
        if (e == cudaSuccess) e = cudaMalloc((void**)&pc->d_marks, sizeof(int32_t) * (size_t)pc->channels);
        if (e == cudaSuccess) e = cudaMemsetAsync(pc->d_marks, 0, sizeof(int32_t) * (size_t)pc->channels, ctx->stream);
        if (e != cudaSuccess) st = cuda_fail(e);
    }
    if (st == MA_OK) st = upload_taps(pc, nullptr, pc->d_taps);
    if (st == MA_OK) st = partition_spectra(pc, pc->w_plan, pc->d_taps, pc->w_block, pc->w_partitions, pc->d_hw);
    if (st == MA_OK) {
        const cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) st = cuda_fail(e);
    }
    if (st != MA_OK) free_coarse(pc);
    return st;
}

// Zeroes the rows in front of every channel's coarse timeline: after the allocation, and after calls that lay the
// buffer out by the caller's block size.  Kept as a state of the stream, not of the host, so that recorded calls may
// be replayed between others.
static ma_status clear_prefix(ma_pconv* pc) {
    if (pc->w_partitions == 1) return MA_OK;
    MA_CUDA(cudaMemset2DAsync(pc->d_timeline, sizeof(float2) * (size_t)pc->w_stride, 0,
                              sizeof(float2) * (size_t)(pc->w_partitions - 1) * (size_t)pc->w_block, (size_t)pc->channels,
                              pc->ctx->stream));
    return MA_OK;
}

// The timeline and product buffers for outputs of up to `full` samples.  Both partitions share them: the
// caller's block size serves calls that continue a stream.
static ma_status alloc_signal_buffers(ma_pconv* pc, int64_t full) {
    MA_TRY(fault_at(pc->ctx, MA_FAULT_RESERVE_BUFFERS));
    auto blocks = [&](int b) { return (full + b - 1) / b; };
    const int64_t own_row = (pc->partitions - 1 + blocks(pc->block)) * pc->block;
    pc->w_stride = (pc->w_partitions - 1 + blocks(pc->w_block)) * pc->w_block;
    const int64_t tl_row = own_row > pc->w_stride ? own_row : pc->w_stride;
    const int64_t own_y = blocks(pc->block) * pc->block, w_y = blocks(pc->w_block) * pc->w_block;
    cudaError_t e = cudaMalloc((void**)&pc->d_timeline, sizeof(float2) * (size_t)pc->channels * (size_t)tl_row);
    if (e == cudaSuccess)
        e = cudaMalloc((void**)&pc->d_y, sizeof(float2) * (size_t)pc->channels * (size_t)(own_y > w_y ? own_y : w_y));
    const ma_status st = e == cudaSuccess ? clear_prefix(pc) : cuda_fail(e);
    if (st != MA_OK) free_signal_buffers(pc);
    return st;
}

// The host copy that ma_pconv_reserve lays out in coarse blocks; without the memory for it whole-signal calls keep the
// caller's block size.  Fresh pages make one thread's copy slow: four share it from 2 MiB up, and
// it makes the uploads one transfer (128 responses of 65536 taps: setting them 5.4 -> 6.4 ms, 8.6 with one thread and
// a transfer per row; with the reservation 7 -> 10.5 ms, 16 that way).
static void keep_taps(ma_pconv* pc, const float* irs) {
    const int64_t taps = pc->taps, stride = taps_stride(taps), count = taps * pc->n_irs;
    pc->h_taps.reset(new (std::nothrow) float[(size_t)(stride * pc->n_irs)]);
    float* const to = pc->h_taps.get();
    if (to == nullptr) return;
    auto part = [&](int64_t at, int64_t end) {
        while (at < end) {
            const int64_t row = at / taps, off = at - row * taps, n = end - at < taps - off ? end - at : taps - off;
            std::memcpy(to + row * stride + off, irs + at, sizeof(float) * (size_t)n);
            at += n;
        }
    };
    if (sizeof(float) * (size_t)count < kThreadedCopyFrom) part(0, count);
    else on_threads<kCopyThreads>([&](int i) { part(count / kCopyThreads * i, i + 1 < kCopyThreads ? count / kCopyThreads * (i + 1) : count); });
    for (int64_t row = 0; row < pc->n_irs; ++row)
        for (int64_t k = taps; k < stride; ++k) to[row * stride + k] = 0.f;
}

static void free_kernel_buffers(ma_pconv* pc) {
    free_coarse(pc);
    pc->h_taps.reset();
    if (pc->d_h) (void)cudaFree(pc->d_h);
    if (pc->d_ch2ir) (void)cudaFree(pc->d_ch2ir);
    if (pc->d_ring) (void)cudaFree(pc->d_ring);
    if (pc->d_tail) (void)cudaFree(pc->d_tail);
    if (pc->d_partial) (void)cudaFree(pc->d_partial);
    pc->d_h = nullptr;
    pc->d_ch2ir = nullptr;
    pc->d_ring = nullptr;
    pc->d_tail = nullptr;
    pc->d_partial = nullptr;
    free_signal_buffers(pc);
    (void)cudaGetLastError();
}

}  // namespace ma

using namespace ma;

extern "C" {

ma_status ma_pconv_create(ma_context* ctx, int32_t block_size, int32_t n_channels, ma_pconv** out) {
    if (out == nullptr) return MA_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    MA_TRY(enter(ctx, MA_FAULT_ALLOC));
    if (block_size <= 0 || n_channels <= 0) return MA_ERR_INVALID_ARGUMENT;
    if ((block_size & (block_size - 1)) != 0) return MA_ERR_SIZE_NOT_POW2;
    if (2 * (int64_t)block_size > kMaxSmallN) return MA_ERR_UNSUPPORTED;
    ma_pconv* pc = new (std::nothrow) ma_pconv();
    if (pc == nullptr) return MA_ERR_ALLOC;
    pc->ctx = ctx;
    pc->block = block_size;
    pc->channels = n_channels;
    ma_status st = ma_fft_plan_create(ctx, 2 * block_size, nullptr, block_size, &pc->plan);
    if (st != MA_OK) {
        delete pc;
        return st;
    }
    *out = pc;
    return MA_OK;
}

ma_status ma_pconv_destroy(ma_pconv* pc) {
    if (pc == nullptr) return MA_OK;
    if (pc->ctx) {
        (void)cudaSetDevice(pc->ctx->device);
        (void)cudaStreamSynchronize(pc->ctx->stream);
    }
    free_kernel_buffers(pc);
    ma_fft_plan_destroy(pc->plan);
    delete pc;
    return MA_OK;
}

ma_status ma_pconv_set_kernels(ma_pconv* pc, const float* irs, int64_t taps, int32_t n_irs,
                               const int32_t* channel_to_ir) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    ma_context* ctx = pc->ctx;
    MA_TRY(enter(ctx, MA_FAULT_ALLOC));
    if (irs == nullptr || n_irs <= 0) return MA_ERR_INVALID_ARGUMENT;
    if (taps <= 0) return MA_ERR_EMPTY_KERNEL;
    const int B = pc->block, C = pc->channels;
    const int64_t P64 = (taps + B - 1) / B;
    if (P64 > (1 << 24)) return MA_ERR_OUTPUT_OVERFLOW;
    const int P = (int)P64;
    std::vector<int32_t> map((size_t)C, 0);
    if (channel_to_ir != nullptr) {
        for (int c = 0; c < C; ++c) {
            if (channel_to_ir[c] < 0 || channel_to_ir[c] >= n_irs) return MA_ERR_INVALID_ARGUMENT;
            map[(size_t)c] = channel_to_ir[c];
        }
    }
    // Largest aligned channel group (4, 2, 1) whose members all use one IR.
    int share = 1;
    for (int cand : {4, 2}) {
        if (C % cand != 0) continue;
        bool ok = true;
        for (int c = 0; c < C && ok; ++c) ok = map[(size_t)c] == map[(size_t)(c - c % cand)];
        if (ok) {
            share = cand;
            break;
        }
    }
    MA_CUDA(cudaStreamSynchronize(ctx->stream));
    free_kernel_buffers(pc);
    pc->taps = taps;
    pc->partitions = P;
    pc->n_irs = n_irs;
    pc->share = share;
    pc->write_index = 0;
    pc->step_captured = false;
    // Partition splits of the streaming step: about 5.25 CTAs per SM in all (the multiply-accumulate
    // kernel fits 7 of its 128-thread CTAs on an SM; measured for 512 / 256 / 128 channels of block 256
    // with 512 partitions: 768 CTAs 92 / 53 / 35 us per step, 640 CTAs 99 / 58 / 36 us, 1024 CTAs
    // 97 / 58 / 36 us - a wave that nearly fills the device, with room left for the step's other
    // kernels), each split still covering at least eight partitions per thread row.
    {
        const int vec = B >= 2 ? 2 : 1;
        const int bp = B / vec;
        const int bpt = bp < kMacThreads ? bp : kMacThreads;
        const int rows = kMacThreads / bpt;
        const int64_t tiles = (int64_t)(C / share) * (bp / bpt);
        int64_t want = ((int64_t)ctx->sm_count * 21 / 4 + tiles / 2) / tiles;
        int64_t max_splits = P / (8 * rows);
        if (max_splits < 1) max_splits = 1;
        if (want > max_splits) want = max_splits;
        if (want < 1) want = 1;
        if (want > 64) want = 64;
        if (want >= 16) want = (want + 4) / 8 * 8;  // whole clusters of eight splits (see step_cluster)
        if (want > max_splits) want = max_splits;
        pc->splits = (int)want;
    }
    const size_t spec_bytes = (size_t)P * B * sizeof(float2);
    ma_status st = MA_OK;
    cudaError_t e = cudaMalloc((void**)&pc->d_h, spec_bytes * (size_t)n_irs);
    if (e == cudaSuccess) e = cudaMalloc((void**)&pc->d_ch2ir, sizeof(int32_t) * (size_t)C);
    if (e == cudaSuccess) e = cudaMalloc((void**)&pc->d_ring, spec_bytes * (size_t)C);
    if (e == cudaSuccess) e = cudaMalloc((void**)&pc->d_tail, sizeof(float) * (size_t)C * B);
    if (e == cudaSuccess)
        e = cudaMalloc((void**)&pc->d_partial, sizeof(float2) * (size_t)pc->splits * (size_t)C * B);
    if (e != cudaSuccess) st = cuda_fail(e);
    if (st == MA_OK) st = copy_h2d(ctx, pc->d_ch2ir, map.data(), sizeof(int32_t) * (size_t)C);
    float* d_taps = nullptr;
    if (st == MA_OK && whole_block(B, taps) != B) keep_taps(pc, irs);
    if (st == MA_OK) st = temp_alloc(ctx, sizeof(float) * (size_t)(taps_stride(taps) * n_irs), (void**)&d_taps);
    if (st == MA_OK) st = upload_taps(pc, irs, d_taps);
    if (st == MA_OK) st = partition_spectra(pc, pc->plan, d_taps, B, P, pc->d_h);
    temp_free(ctx, d_taps);
    if (st == MA_OK) st = ma_pconv_reset(pc);
    if (st == MA_OK) {
        cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
        if (e2 != cudaSuccess) st = cuda_fail(e2);
    }
    if (st != MA_OK) free_kernel_buffers(pc);
    return st;
}

ma_status ma_pconv_partition_count(ma_pconv* pc, int32_t* partitions) {
    if (pc == nullptr || partitions == nullptr) return MA_ERR_INVALID_ARGUMENT;
    *partitions = pc->partitions;
    return MA_OK;
}

ma_status ma_pconv_step_splits(ma_pconv* pc, int32_t set_to, int32_t* splits) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    if (pc->d_h == nullptr) return MA_ERR_KERNEL_NOT_CONFIGURED;
    if (set_to > 0) {
        ma_context* ctx = pc->ctx;
        MA_TRY(enter(ctx, MA_FAULT_ALLOC));
        if (set_to > pc->partitions || set_to > 64) return MA_ERR_INVALID_ARGUMENT;
        if (set_to != pc->splits) {
            // the partial spectra of earlier steps may still be in use: wait, then resize
            MA_CUDA(cudaStreamSynchronize(ctx->stream));
            float2* fresh = nullptr;
            MA_CUDA(cudaMalloc((void**)&fresh, sizeof(float2) * (size_t)set_to * (size_t)pc->channels * pc->block));
            if (pc->d_partial) (void)cudaFree(pc->d_partial);
            pc->d_partial = fresh;
            pc->splits = set_to;
        }
    }
    if (splits != nullptr) *splits = pc->splits;
    return MA_OK;
}

ma_status ma_pconv_reset(ma_pconv* pc) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    MA_TRY(enter(pc->ctx, MA_FAULT_LAUNCH));
    if (pc->d_ring == nullptr) return MA_OK;  // nothing configured yet
    const size_t ring_bytes = (size_t)pc->channels * pc->partitions * pc->block * sizeof(float2);
    MA_CUDA(cudaMemsetAsync(pc->d_ring, 0, ring_bytes, pc->ctx->stream));
    MA_CUDA(cudaMemsetAsync(pc->d_tail, 0, sizeof(float) * (size_t)pc->channels * pc->block, pc->ctx->stream));
    pc->write_index = 0;
    pc->clear = true;
    return MA_OK;
}

ma_status ma_pconv_reserve(ma_pconv* pc, int64_t max_len) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    ma_context* ctx = pc->ctx;
    MA_TRY(enter(ctx, MA_FAULT_ALLOC));
    if (pc->d_h == nullptr) return MA_ERR_KERNEL_NOT_CONFIGURED;
    if (max_len <= 0) return MA_ERR_INVALID_ARGUMENT;
    if (max_len <= pc->reserved_len) return MA_OK;
    int64_t full;
    if (__builtin_add_overflow(max_len, pc->taps - 1, &full)) return MA_ERR_OUTPUT_OVERFLOW;
    MA_CUDA(cudaStreamSynchronize(ctx->stream));
    free_signal_buffers(pc);
    ma_status st = pc->w_plan == nullptr ? build_coarse(pc) : MA_OK;
    if (st == MA_OK) st = alloc_signal_buffers(pc, full);
    if (st == MA_ERR_ALLOC && pc->w_plan != pc->plan) {
        // what the coarse partition takes may be what these buffers lack
        use_own_block(pc);
        st = alloc_signal_buffers(pc, full);
    }
    if (st != MA_OK) {
        free_coarse(pc);  // the next call lays the taps out afresh
        return st;
    }
    pc->h_taps.reset();
    pc->reserved_len = max_len;
    return MA_OK;
}

}  // extern "C"

static bool capturing(const ma_context* ctx) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(ctx->stream, &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
}

// Whether a whole-signal call may take the coarse partition, which assumes a delay line of zeros.
static bool runs_coarse(const ma_pconv* pc) { return pc->clear && !pc->step_captured; }

// Once per whole-signal call, before its channel ranges.
static void open_whole(ma_pconv* pc) {
    if (++pc->mark <= 0) pc->mark = 1;
}

// Once per whole-signal call, after its channel ranges (`done`: all of them are queued).  A call pushes
// ceil((len + taps - 1)/B) >= ceil(len/B) + P - 1 blocks, so the only spectrum of its input that can still be in the
// delay line is in the slot the next block overwrites.  A recorded call has not run yet: it leaves `clear` alone.
static ma_status close_whole(ma_pconv* pc, bool done) {
    if (!runs_coarse(pc)) MA_TRY(clear_prefix(pc));
    if (done) {
        pc->write_index = 0;
        if (!capturing(pc->ctx)) pc->clear = true;
    }
    return MA_OK;
}

// Whole-signal convolution of channels [c0, c0 + nc) (nc a multiple of the IR-sharing group): `in`
// and `out` point at channel c0's rows.  Every buffer of the object is per channel, so a range runs
// on its own slices; open_whole comes before the first range, close_whole after the last.
static ma_status process_range(ma_pconv* pc, int c0, int nc, const float* in, int64_t len, int64_t in_stride,
                               float* out, int64_t out_stride, int64_t full) {
    ma_context* ctx = pc->ctx;
    const bool coarse = runs_coarse(pc);
    const bool rescue = coarse && pc->w_plan != pc->plan;
    ma_fft_plan* plan = coarse ? pc->w_plan : pc->plan;
    const int B = coarse ? pc->w_block : pc->block, P = coarse ? pc->w_partitions : pc->partitions;
    const int64_t T = (full + B - 1) / B;
    const int64_t tl_len = (int64_t)P - 1 + T;
    const int64_t tl_stride = coarse ? pc->w_stride : tl_len * B;
    float2* ring = pc->d_ring + (int64_t)c0 * pc->partitions * pc->block;
    float2* timeline = pc->d_timeline + (int64_t)c0 * tl_stride;
    float2* y = pc->d_y + (int64_t)c0 * T * B;

    // 1. history -> timeline prefix (a clear delay line: zeros, see clear_prefix)
    if (P > 1 && !coarse) {
        const int64_t total = (int64_t)nc * (P - 1) * B;
        int grid = (int)((total + 255) / 256 < (int64_t)ctx->sm_count * 8 ? (total + 255) / 256 : (int64_t)ctx->sm_count * 8);
        pconv_history_kernel<<<grid, 256, 0, ctx->stream>>>(ring, timeline, tl_stride, P, B, pc->write_index, 0, 1, nc);
        MA_TRY(after_launch(ctx));
    }
    // 2. all input blocks -> spectra
    {
        R2CParams p{};
        p.in = in;
        p.signal_stride = in_stride;
        p.frames_per_signal = T;
        p.total_frames = T * nc;
        p.signal_len = len;
        p.hop = B;
        p.frame_valid = B;
        p.out_a = reinterpret_cast<float*>(timeline + (int64_t)(P - 1) * B);
        p.out_signal_stride = tl_stride;
        p.out_frame_stride = B;
        p.layout = LAYOUT_HALF_PACKED;
        p.mag_kind = MAG_NONE;
        p.marks = rescue ? pc->d_marks + c0 : nullptr;
        p.mark = pc->mark;
        MA_TRY(launch_r2c_small(plan, p));
    }
    // 3. delay-line multiply-accumulate for every (channel, block)
    {
        MacParams q{};
        q.x = timeline;
        q.x_chan_stride = tl_stride;
        q.h = coarse ? pc->d_hw : pc->d_h;
        q.ch2ir = pc->d_ch2ir + c0;
        q.out = y;
        q.out_split_stride = 0;
        q.out_chan_stride = T * B;
        q.out_t_stride = B;
        q.block = B;
        q.partitions = P;
        q.w0 = P - 1;
        q.wrap = 0;
        q.splits = 1;
        q.p_per_split = P;
        // One or two partitions: nothing is reused over time, and the fused products of the streaming kernel
        // round less than component-wise sums.
        if (B >= 32 && P > 2 && T < (int64_t)1 << 30) MA_TRY(launch_mac_tiled(pc, q, nc, T, tl_len));
        else MA_TRY(launch_mac(pc, q, nc, false, T));
    }
    // A call in place overwrites samples that pconv_rescue_kernel may want: their copy goes where the spectra were.
    const float* samples = in;
    int64_t samples_stride = in_stride;
    const int64_t in_span = (nc - 1) * in_stride + len, out_span = (nc - 1) * out_stride + full;
    if (rescue && in < out + out_span && out < in + in_span) {
        float* copy = reinterpret_cast<float*>(timeline + (int64_t)(P - 1) * B);
        MA_CUDA(cudaMemcpy2DAsync(copy, sizeof(float2) * (size_t)tl_stride, in, sizeof(float) * (size_t)(nc > 1 ? in_stride : len),
                                  sizeof(float) * (size_t)len, (size_t)nc, cudaMemcpyDeviceToDevice, ctx->stream));
        samples = copy;
        samples_stride = 2 * tl_stride;
    }
    // 4. inverse transform + block overlap-add, truncated at len + taps - 1
    {
        C2RParams p{};
        p.in_a = reinterpret_cast<const float*>(y);
        p.in_signal_stride = T * B;
        p.in_frame_stride = B;
        p.frames_per_signal = T;
        p.n_signals = nc;
        p.layout = LAYOUT_HALF_PACKED;
        p.hop = B;
        p.window = nullptr;
        p.out = out;
        p.out_signal_stride = out_stride;
        p.out_len = full;
        p.floor = -1.0f;
        MA_TRY(launch_istft_small(plan, p));
    }
    if (rescue) {
        RescueParams p{};
        p.in = samples;
        p.len = len;
        p.in_stride = samples_stride;
        p.taps = pc->d_taps;
        p.n_taps = pc->taps;
        p.taps_stride = taps_stride(pc->taps);
        p.ch2ir = pc->d_ch2ir + c0;
        p.out = out;
        p.out_stride = out_stride;
        p.full = full;
        p.marks = pc->d_marks + c0;
        p.mark = pc->mark;
        p.channels = nc;
        p.block = pc->block;
        p.coarse = B;
        p.reach = (int64_t)pc->partitions * pc->block;
        p.coarse_reach = (int64_t)P * B;
        const int64_t chunks = (full + kRescueOutputs - 1) / kRescueOutputs, most = 4 * (int64_t)ctx->sm_count;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(chunks < most ? chunks : most));
        cfg.blockDim = dim3(kRescueThreads);
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, pconv_rescue_kernel, p);  // an error is picked up by after_launch
        MA_TRY(after_launch(ctx));
    }
    // 5. the last P block spectra become the delay line (clear before the call: it stays clear, see close_whole)
    if (!coarse) {
        const int64_t total = (int64_t)nc * P * B;
        int grid = (int)((total + 255) / 256 < (int64_t)ctx->sm_count * 8 ? (total + 255) / 256 : (int64_t)ctx->sm_count * 8);
        pconv_history_kernel<<<grid, 256, 0, ctx->stream>>>(ring, timeline, tl_stride, P, B, 0, T - 1, 0, nc);
        MA_TRY(after_launch(ctx));
        MA_CUDA(cudaMemsetAsync(pc->d_tail + (int64_t)c0 * B, 0, sizeof(float) * (size_t)nc * B, ctx->stream));
    }
    return MA_OK;
}

extern "C" {

ma_status ma_pconv_process_dev(ma_pconv* pc, const float* in, int64_t len, int64_t in_stride, float* out,
                               int64_t out_stride) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    ma_context* ctx = pc->ctx;
    MA_TRY(enter(ctx, MA_FAULT_LAUNCH));
    if (pc->d_h == nullptr) return MA_ERR_KERNEL_NOT_CONFIGURED;
    if (len == 0) return MA_OK;  // empty input -> empty output (Convolution.swift:339-342)
    if (len < 0 || in == nullptr || out == nullptr) return MA_ERR_INVALID_ARGUMENT;
    if (pc->write_index < 0 || pc->write_index >= pc->partitions) return MA_ERR_INVALID_PARTITION_STATE;
    int64_t full;
    if (__builtin_add_overflow(len, pc->taps - 1, &full)) return MA_ERR_OUTPUT_OVERFLOW;
    if (len > pc->reserved_len) return MA_ERR_INVALID_ARGUMENT;
    if (pc->channels > 1 && (in_stride < len || out_stride < full)) return MA_ERR_INVALID_ARGUMENT;
    open_whole(pc);
    const ma_status st = process_range(pc, 0, pc->channels, in, len, in_stride, out, out_stride, full);
    const ma_status closed = close_whole(pc, st == MA_OK);
    return st != MA_OK ? st : closed;
}

// Host form: groups of channels go through the context's three-stage pipeline (copy in, convolve,
// copy out on three streams, two workspace lanes deep) when both host arrays are pinned, so the
// transfers of neighbouring groups run under the convolution of the current one; pageable arrays
// take the same groups one after the other through the staging buffer.
ma_status ma_pconv_process_host(ma_pconv* pc, const float* in, int64_t len, int64_t in_stride, float* out,
                                int64_t out_stride) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    ma_context* ctx = pc->ctx;
    MA_TRY(enter(ctx, MA_FAULT_LAUNCH));
    if (pc->d_h == nullptr) return MA_ERR_KERNEL_NOT_CONFIGURED;
    if (len == 0) return MA_OK;
    if (len < 0 || in == nullptr || out == nullptr) return MA_ERR_INVALID_ARGUMENT;
    if (pc->write_index < 0 || pc->write_index >= pc->partitions) return MA_ERR_INVALID_PARTITION_STATE;
    int64_t full;
    if (__builtin_add_overflow(len, pc->taps - 1, &full)) return MA_ERR_OUTPUT_OVERFLOW;
    const int C = pc->channels;
    if (C > 1 && (in_stride < len || out_stride < full)) return MA_ERR_INVALID_ARGUMENT;
    MA_TRY(ma_pconv_reserve(pc, len));
    const int group = pc->share;  // channels that must stay together (they share one impulse response)
    const size_t in_row = round256(sizeof(float) * (size_t)len), out_row = round256(sizeof(float) * (size_t)full);
    const bool pinned = is_pinned(in) && is_pinned(out);
    open_whole(pc);
    Pipe pp;
    MA_TRY(pipe_open(pp, ctx, pinned, C / group, (in_row + out_row) * (size_t)group, 0));
    const int64_t step = pp.chunk * group;
    int64_t i = 0;
    for (int64_t c0 = 0; c0 < C && pp.st == MA_OK; c0 += step, ++i) {
        const int nc = (int)(C - c0 < step ? C - c0 : step);
        char* lane = pp.lane[i & 1];
        float* d_in = reinterpret_cast<float*>(lane);
        float* d_out = reinterpret_cast<float*>(lane + in_row * (size_t)nc);
        pp.before_copy_in(i);
        pp.in2d(d_in, in_row, in + c0 * in_stride, sizeof(float) * (size_t)in_stride, sizeof(float) * (size_t)len, (size_t)nc);
        pp.before_kernels(i);
        if (pp.st == MA_OK)
            pp.st = process_range(pc, (int)c0, nc, d_in, len, (int64_t)(in_row / sizeof(float)), d_out,
                                  (int64_t)(out_row / sizeof(float)), full);
        pp.before_copy_out(i);
        pp.out2d(out + c0 * out_stride, sizeof(float) * (size_t)out_stride, d_out, out_row, sizeof(float) * (size_t)full, (size_t)nc);
        pp.after_copy_out(i);
    }
    const ma_status st = pp.finish();
    const ma_status closed = close_whole(pc, st == MA_OK);
    return st != MA_OK ? st : closed;
}

ma_status ma_pconv_step_dev(ma_pconv* pc, const float* in_block, int64_t in_stride, float* out_block,
                            int64_t out_stride) {
    if (pc == nullptr) return MA_ERR_INVALID_ARGUMENT;
    ma_context* ctx = pc->ctx;
    MA_TRY(enter(ctx, MA_FAULT_LAUNCH));
    if (pc->d_h == nullptr) return MA_ERR_KERNEL_NOT_CONFIGURED;
    if (in_block == nullptr || out_block == nullptr) return MA_ERR_INVALID_ARGUMENT;
    const int B = pc->block, P = pc->partitions, C = pc->channels;
    if (C > 1 && (in_stride < B || out_stride < B)) return MA_ERR_INVALID_ARGUMENT;
    if (pc->write_index < 0 || pc->write_index >= P) return MA_ERR_INVALID_PARTITION_STATE;
    const int w = pc->write_index;
    pc->clear = false;
    if (!pc->step_captured && capturing(ctx)) pc->step_captured = true;
    // The three kernels are chained by programmatic dependent launch: this step's r2c may run
    // beside the previous step's c2r (see fft_small.cu).  That is only sound when the kernel right
    // before this r2c on the stream is that c2r and the two share no data: r2c reads its input
    // before it waits for the earlier kernel.  So r2c is launched plainly when the caller feeds the
    // previous step's output block straight back in, and whenever the library queued anything else
    // on this context since the last step (whose output might be this step's input).
    const float* in_end = in_block + (int64_t)(C - 1) * in_stride + B;
    const bool feeds_back = ctx->step_out != nullptr && in_block < ctx->step_out_end && ctx->step_out < in_end;
    const bool follows_step = ctx->launch_seq == ctx->step_end_seq;
    // 1. this block's spectrum into ring slot w
    {
        R2CParams p{};
        p.dependent_launch = (follows_step && !feeds_back) ? 1 : 0;
        p.in = in_block;
        p.signal_stride = in_stride;
        p.frames_per_signal = 1;
        p.total_frames = C;
        p.signal_len = B;
        p.hop = B;
        p.frame_valid = B;
        p.out_a = reinterpret_cast<float*>(pc->d_ring + (int64_t)w * B);
        p.out_signal_stride = (int64_t)P * B;
        p.out_frame_stride = 0;
        p.layout = LAYOUT_HALF_PACKED;
        p.mag_kind = MAG_NONE;
        MA_TRY(launch_r2c_small(pc->plan, p));
    }
    // 2. stream the whole delay line once: partial sums per partition split
    {
        MacParams q{};
        q.x = pc->d_ring;
        q.x_chan_stride = (int64_t)P * B;
        q.h = pc->d_h;
        q.ch2ir = pc->d_ch2ir;
        q.out = pc->d_partial;
        q.out_split_stride = (int64_t)C * B;
        q.out_chan_stride = B;
        q.out_t_stride = 0;
        q.block = B;
        q.partitions = P;
        q.w0 = w;
        q.wrap = P;
        q.splits = pc->splits;
        q.p_per_split = (P + pc->splits - 1) / pc->splits;
        q.dependent_launch = 1;
        q.cluster = step_cluster(pc->splits);
        MA_TRY(launch_mac(pc, q, pc->channels, true, 1));
    }
    // 3. sum the partials, inverse transform, add the kept tail, keep the new one
    const int partials = pc->splits / step_cluster(pc->splits);  // partial spectra the multiply-accumulate left
    const bool own_sum = partials >= kSumKernelFromSplits && ((int64_t)C * B) % 2 == 0;
    if (own_sum) {
        const int64_t n4 = (int64_t)C * B / 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((n4 + 255) / 256));
        cfg.blockDim = dim3(256);
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, pconv_sum_partials_kernel, reinterpret_cast<float4*>(pc->d_partial), n4, n4,
                                 partials);  // an error is picked up by after_launch
        MA_TRY(after_launch(ctx));
    }
    {
        C2RParams p{};
        p.in_a = reinterpret_cast<const float*>(pc->d_partial);
        p.in_signal_stride = B;
        p.in_frame_stride = 0;
        p.frames_per_signal = 1;
        p.n_signals = C;
        p.layout = LAYOUT_HALF_PACKED;
        p.n_partials = own_sum ? 1 : partials;
        p.partial_stride = (int64_t)C * B;
        p.out = out_block;
        p.out_signal_stride = out_stride;
        p.tail = pc->d_tail;
        p.dependent_launch = 1;
        MA_TRY(launch_c2r_small(pc->plan, p));
    }
    ctx->step_end_seq = ctx->launch_seq;
    ctx->step_out = out_block;
    ctx->step_out_end = out_block + (int64_t)(C - 1) * out_stride + B;
    pc->write_index = (w + 1) % P;
    return MA_OK;
}

}  // extern "C"
