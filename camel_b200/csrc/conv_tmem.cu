// conv2d for layers with few channels on both sides (at most 32 in, at most 64 out, a small
// filter; the 32 -> 64 channel 3x3 layer of a small CNN).  Two forms: conv_pairs_kernel, on float16 pairs, computes
// almost every image and has its own comment further down; the tf32 form that this comment is about computes, behind it, the
// images whose values float16 pairs cannot hold.  In it the filters live in tensor memory.
//
// Why another kernel.  With 64 output channels the tensor core cannot be given a wide tile:
// measured on B200 (ct_measure_mma_rate), tcgen05.mma kind::tf32 of 128 x N x 8 takes ~138 clocks
// at N = 256, ~73 at N = 128, ~54 at N = 64 and never less than ~49, and M = 64 takes as long as
// M = 128.  The pixels-on-rows kernel (conv_swap_stream_kernel) issues 128 x 64 x 8 MMAs and
// re-fetches, per filter tap, a shifted copy of the same pixels and the tap's filter rows; its
// operands cross shared memory twice (TMA in, MMA out), about 10 KB per MMA, and that traffic,
// not the tensor pipe, sets its pace (~80 clocks per MMA).  Here
//   * the filters are the A operand and stay in TENSOR MEMORY for the whole launch: rows 0..63
//     hold the tf32 "hi" part of the 64 filters, rows 64..127 the "lo" part, 8 columns per k-step
//     (tap, group of 8 input channels) - written once per CTA with tcgen05.st, never re-read from
//     shared memory;
//   * the pixels are the B operand, N = 128 per tile: th output rows of PW = w + 2 pad positions
//     (the two halo columns of every row are computed and dropped).  A tile's input - th + kh - 1
//     rows of PW positions, halo included, zeros outside the image - is fetched ONCE by one 4-D
//     TMA box per plane; because a position's row index in the box is y * PW + x, the pixels a
//     tap (r, s) needs are the same rows shifted by r * PW + s, i.e. the same shared memory
//     through a descriptor whose start address is moved by that many 128-byte rows;
//   * per k-step two MMAs, [W_hi; W_lo] x X_hi and [W_hi; W_lo] x X_lo, accumulate into one
//     128 x 128 accumulator: lane c holds W_hi . (X_hi + X_lo), lane 64 + c holds W_lo . (X_hi +
//     X_lo); the epilogue adds the two lanes (all four terms of the split product).
// Shared-memory traffic per k-step drops to ~9 KB for 146 clocks of tensor work, so the tensor
// pipe is the bound again: ~0.7 of the 3xTF32 ceiling for this shape instead of ~0.3.
//
// Roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer (and TMEM owner), warps 2-9
// epilogue: each drains a 32-lane x 64-column block of the accumulator into a shared-memory block
// [lane][position] (128-bit stores), which frees the accumulator for the next tile's MMAs; then
// warp e writes out channels e, e + 8, ...: hi lane + lo lane, bias, relu, optional 2x2 max-pool,
// its lanes over consecutive positions, so a store instruction covers consecutive pixels of one
// NCHW channel plane.  The epilogue of tile i runs while the MMAs of tile i + 1 are issued; it has
// to stay shorter than those (~2.7 us), which is why a position's pixel offset is computed once per
// kernel, not per value.  One CTA per SM walks the tiles.  Every wait is bounded.
#include "common.cuh"
#include "tc_ptx.cuh"
#include "half_split.cuh"
#include "split.cuh"
#include "tmap.cuh"

#include <algorithm>

// Optional per-CTA clock accounting for tuning; compiled in only with -DCT_CONV_TRACE.
#ifdef CT_CONV_TRACE
__device__ unsigned long long g_conv_trace[256 * 16];
#define CV_CLOCK() clock64()
#define CV_ACCUM(slot, cycles)                                                          \
    do {                                                                                \
        if (blockIdx.x < 256)                                                           \
            g_conv_trace[blockIdx.x * 16 + (slot)] += (unsigned long long)(cycles);     \
    } while (0)
extern "C" int ct_debug_conv_trace(unsigned long long *host, int count, int clear) {
    int rc = (int)cudaMemcpyFromSymbol(host, g_conv_trace, sizeof(unsigned long long) * (size_t)count);
    if (clear) {
        static unsigned long long zeros[256 * 16];
        cudaMemcpyToSymbol(g_conv_trace, zeros, sizeof(zeros));
    }
    return rc;
}
#else
#define CV_CLOCK() 0ll
#define CV_ACCUM(slot, cycles) do { } while (0)
#endif

namespace ct {
namespace {

using namespace ptx;

constexpr int kTA_EpiWarps  = 8;
constexpr int kTA_Threads   = 64 + 32 * kTA_EpiWarps;
constexpr int kTA_CvtWarps  = 4;                  // raw mode: warps that turn float32 boxes into hi/lo planes
constexpr int kTA_ThreadsRaw = kTA_Threads + 32 * kTA_CvtWarps;
constexpr int kTA_RawStages = 2;
constexpr int kTA_MaxKSteps = 48;                 // 8 TMEM columns each: 384 of the 512 columns
constexpr int kTA_DCol      = kTA_MaxKSteps * 8;  // the accumulator's first column
constexpr int kTA_N         = 128;                // positions per tile (MMA N)
constexpr int kTA_StageRowF = kTA_N + 4;          // epilogue staging: [128 lanes][132] floats: rows 16-byte aligned,
                                                  // 128-bit stores of 8 consecutive lanes fall into distinct banks
constexpr int kTA_StagingBytes = 128 * kTA_StageRowF * 4;

struct ConvTmemParams {
    const float *w;   // filters [ko][c][kh][kw], float32
    const float *bias;
    float *out;       // [batch][ko][ho][wo], or [batch][ko][ho/2][wo/2] with pool
    uint32_t *flags;
    int ko, c, kh, kw, pad;
    int ho, wo, pw;   // pw = input width + 2 pad: positions per tile row
    int th;           // output rows per tile
    int tiles_y;      // ceil(ho / th)
    int ksteps;       // kh * kw * 4
    int box_bytes;    // bytes of one plane's TMA box
    int plane_bytes;  // shared-memory bytes reserved per plane (box plus the rows shifted reads run into)
    int stages;
    int act, pool;
    const float *image_scale; // planes: [batch] inverse scales, 0 for an image that needs tf32 terms
    uint2 *tile_range;        // raw: [range_tiles to an image] range of the values of each of conv_pairs_kernel's tiles, and
                              // behind them one entry whose .x says that the filters need tf32 terms
    int range_tiles, range_total;
    // raw mode (the input is read as it is, NCHW float32, and split into planes inside the kernel)
    int box_w;        // floats per row of the raw box (a multiple of four)
    int off_x;        // the tile's first position (x = -pad) sits this many floats into a raw row
    int box_rows;     // th + kh - 1
    int raw_bytes;    // bytes of one raw box: 32 channels x box_rows x box_w floats
    int raw_stride;   // shared-memory bytes reserved per raw stage
};

// Whether image `img` is left to the tf32 form: its values, over all its tiles (every pixel is in one of them), or the
// filters do not fit float16 pairs.  A property of the image alone, so that its bits do not depend on how the launch
// was cut into tiles (the fused pool takes rows by twos), on what else is in the batch, or on how it was read.
template <bool RAW> __device__ __forceinline__ bool image_needs_tf32(const ConvTmemParams &p, int img) {
    if (!RAW)
        return __ldg(p.image_scale + img) == 0.0f;
    const uint32_t filters = p.tile_range[p.range_total].x;
    const uint2 *src       = p.tile_range + (int64_t)img * p.range_tiles;
    uint2 range            = make_uint2(0u, kNoneSmallest);
    for (int t = 0; t < p.range_tiles; t += 8) {
        uint2 r[8]; // eight loads in flight: one after the other they cost an idle launch 4 us
#pragma unroll
        for (int j = 0; j < 8; ++j)
            r[j] = src[min(t + j, p.range_tiles - 1)];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            range = range_join(range, r[j]);
    }
    float scale, inverse;
    return filters != 0u || !half_range_fits(range, scale, inverse);
}

// Tiles of a block of the tf32 form, a bit each: at most kTA_MaxOwn to a block (the grid grows beyond that).
constexpr int kTA_MaxOwn = 4096;
__device__ __forceinline__ int next_own(const uint32_t *mask, int q, int own) {
    while (q < own) {
        const uint32_t bits = mask[q >> 5] >> (q & 31);
        if (bits)
            return q + __ffs(bits) - 1;
        q = (q | 31) + 1;
    }
    return own;
}

// The filters [ko][row] in shared memory, rows an odd number of floats apart so that lanes that own filters read distinct
// banks; a warp per filter, which it hands to `seen` as it goes (every lane has its share).  Read from global
// memory by the lanes that write them to tensor memory - 128 threads, a sector for every value - the set-up took
// 35 of the 41 us of a layer on four images.
template <typename Seen>
__device__ __forceinline__ void stage_filters(const float *w, int ko, int row, float *rows, int warp, int warps, int lane, Seen seen) {
    const int stride = row | 1;
    // four of the warp's filters at a time, so that their loads are in flight together
    for (int f0 = warp; f0 < ko; f0 += 4 * warps) {
        uint2 range[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            range[q] = make_uint2(0u, kNoneSmallest);
#pragma unroll 2
        for (int e = lane; e < row; e += 32) {
            float v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                v[q] = f0 + q * warps < ko ? w[(int64_t)(f0 + q * warps) * row + e] : 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (f0 + q * warps < ko)
                    range_take(range[q], v[q]), rows[(f0 + q * warps) * stride + e] = v[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (f0 + q * warps < ko)
                seen(f0 + q * warps, range[q]);
    }
}
// ... and of a region that the asynchronous proxy writes next.
__device__ __forceinline__ void filters_taken() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_st_32x32_x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_tf32_a_tmem(
    uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// RAW = false: map_x_hi / map_x_lo cover NHWC hi / lo planes written by a pre-pass.
// RAW = true:  map_x_hi covers the input itself, [batch][c][h][w] float32 (map_x_lo is not used);
//              the producer fetches a tile's box of it - 32 channels x box_rows x box_w floats, zeros
//              outside the image and past the last channel - and four more warps rewrite it as the
//              two planes the MMAs read: position (y, x) becomes row y * pw + x, its 32 channels the
//              128 bytes of the row (swizzled as TMA would have), each value split into tf32 parts.
//              The pre-pass and its 12 bytes of traffic per input element are gone.
template <bool RAW>
__global__ void __launch_bounds__(kTA_ThreadsRaw, 1) conv_tmem_filters_kernel(
    const __grid_constant__ CUtensorMap map_x_hi, const __grid_constant__ CUtensorMap map_x_lo,
    const ConvTmemParams p, const int total_tiles) {
    griddep_wait(); // no early successor: it could take the tensor memory that an image of wide range will need here
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[4];
    __shared__ uint64_t bar_empty[4];
    __shared__ uint64_t bar_raw_full[kTA_RawStages];
    __shared__ uint64_t bar_raw_empty[kTA_RawStages];
    __shared__ uint64_t bar_tmem_full;
    __shared__ uint64_t bar_tmem_empty;
    __shared__ uint64_t bar_done;
    __shared__ uint64_t bar_epi; // the four epilogue warps meet here (bounded, unlike bar.sync)
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s;
    __shared__ uint32_t own_mask[kTA_MaxOwn / 32];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // this block's tiles, blockIdx.x + q gridDim.x, whose images the float16 form leaves to this one
    const int own = (total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
    int any       = 0;
    for (int q0 = warp * 32; q0 < own; q0 += (int)blockDim.x) {
        const int q         = q0 + lane;
        const bool mine     = q < own && image_needs_tf32<RAW>(p, ((int)blockIdx.x + q * (int)gridDim.x) / p.tiles_y);
        const uint32_t bits = __ballot_sync(0xffffffffu, mine);
        any |= bits != 0u;
        if (lane == 0)
            own_mask[q0 >> 5] = bits;
    }
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
    if (!__syncthreads_or(any) || abort_flag_s)
        return; // conv_pairs_kernel has computed them all

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = 2u * (uint32_t)p.plane_bytes;
    // planes | raw boxes (raw mode) | epilogue staging
    const uint32_t raw_base = smem_base + (uint32_t)p.stages * stage_bytes;
    const uint32_t raw_all  = RAW ? (uint32_t)kTA_RawStages * (uint32_t)p.raw_stride : 0u;
    float *staging = reinterpret_cast<float *>(smem_raw + (raw_base - smem_u32(smem_raw)) + raw_all);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), RAW ? kTA_CvtWarps : 1); // raw mode: the converting warps fill a stage
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int s = 0; s < kTA_RawStages; ++s) {
            mbar_init(smem_u32(&bar_raw_full[s]), 1);
            mbar_init(smem_u32(&bar_raw_empty[s]), kTA_CvtWarps);
        }
        mbar_init(smem_u32(&bar_tmem_full), 1);
        mbar_init(smem_u32(&bar_tmem_empty), kTA_EpiWarps);
        mbar_init(smem_u32(&bar_done), 1);
        mbar_init(smem_u32(&bar_epi), kTA_EpiWarps);
        mbar_fence_init();
        prefetch_tensormap(&map_x_hi);
        prefetch_tensormap(&map_x_lo);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    float *filters = reinterpret_cast<float *>(smem_raw + (smem_base - smem_u32(smem_raw))); // where the stages will be
    stage_filters(p.w, p.ko, p.c * p.kh * p.kw, filters, warp, (int)blockDim.x / 32, lane, [](int, uint2) {});
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;

    // ---- the filters go to tensor memory, once: warps 2..5 own the four lane quarters ----------
    if (warp >= 2 && warp < 6) {
        const int quarter = warp & 3;
        const int m       = quarter * 32 + lane;      // TMEM lane = row of the A operand
        const int ch      = m & 63;                   // filter
        const bool lo_row = m >= 64;                  // rows 64..127: the low parts
        const int taps    = p.kh * p.kw;
        const float *src  = filters + ch * ((p.c * taps) | 1);
#pragma unroll 2
        for (int ks = 0; ks < p.ksteps; ++ks) {
            const int tap = ks >> 2, c0 = (ks & 3) * 8;
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float x = (ch < p.ko && c0 + j < p.c) ? src[(c0 + j) * taps + tap] : 0.0f;
                float hi, lo;
                split_tf32_flat(x, hi, lo);
                v[j] = __float_as_uint(lo_row ? lo : hi);
            }
            tmem_st_32x32_x8(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ks * 8), v);
        }
        tmem_st_wait();
        filters_taken();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    if (warp == 0) {
        // ===== TMA producer: one halo box per plane and tile (raw mode: one box of the input) =====
        if (elect_one()) {
            int i = 0;
            bool ok = true;
            const int nstages = RAW ? kTA_RawStages : p.stages;
            for (int q = next_own(own_mask, 0, own); q < own && ok; q = next_own(own_mask, q + 1, own), ++i) {
                const int tile = (int)blockIdx.x + q * (int)gridDim.x;
                const int img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
                const int s       = i % nstages;
                const uint32_t ph = (uint32_t)(i / nstages) & 1u;
                if (!mbar_wait_patient(smem_u32(RAW ? &bar_raw_empty[s] : &bar_empty[s]), ph ^ 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                const int32_t h0 = ty * p.th - p.pad;
                if (RAW) {
                    const uint32_t full = smem_u32(&bar_raw_full[s]);
                    mbar_expect_tx(full, (uint32_t)p.raw_bytes);
                    // the box starts off_x floats left of x = -pad so that its first byte is 16-byte aligned
                    tma_load_4d(raw_base + (uint32_t)s * (uint32_t)p.raw_stride, &map_x_hi, full, -p.pad - p.off_x, h0, 0, img);
                } else {
                    const uint32_t full = smem_u32(&bar_full[s]);
                    const uint32_t dst  = smem_base + (uint32_t)s * stage_bytes;
                    mbar_expect_tx(full, 2u * (uint32_t)p.box_bytes);
                    const int32_t w0 = -p.pad;
                    tma_load_4d(dst, &map_x_hi, full, 0, w0, h0, img);
                    tma_load_4d(dst + (uint32_t)p.plane_bytes, &map_x_lo, full, 0, w0, h0, img);
                }
            }
            if (*abort_flag) {
                // unwind: let the copies still in flight land before the CTA goes away
                const int first = i - nstages < 0 ? 0 : i - nstages;
                for (int k2 = first; k2 < i; ++k2) {
                    const uint32_t bar = smem_u32(RAW ? &bar_raw_full[k2 % nstages] : &bar_full[k2 % nstages]);
                    const uint32_t ph  = (uint32_t)(k2 / nstages) & 1u;
                    const uint64_t t0  = globaltimer_ns();
                    while (!mbar_try_wait(bar, ph) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        if (elect_one()) {
            const uint32_t idesc  = make_idesc(2u, 128, (uint32_t)kTA_N);
            const uint32_t d_tmem = tmem_base + (uint32_t)kTA_DCol;
            int i = 0;
            bool ok = true;
            const long long t_start = CV_CLOCK();
            for (int q = next_own(own_mask, 0, own); q < own && ok; q = next_own(own_mask, q + 1, own), ++i) {
                const int s       = i % p.stages;
                const uint32_t ph = (uint32_t)(i / p.stages) & 1u;
                // the accumulator of the previous tile has been drained
                const long long t0 = CV_CLOCK();
                if (!mbar_wait(smem_u32(&bar_tmem_empty), ((uint32_t)i & 1u) ^ 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                const long long t1 = CV_CLOCK();
                if (!mbar_wait(smem_u32(&bar_full[s]), ph, abort_flag)) {
                    ok = false;
                    break;
                }
                CV_ACCUM(0, t1 - t0);          // waiting for the accumulator
                CV_ACCUM(1, CV_CLOCK() - t1);  // waiting for the halo
                tc_fence_after_sync();
                const uint32_t x_hi = smem_base + (uint32_t)s * stage_bytes;
                const uint32_t x_lo = x_hi + (uint32_t)p.plane_bytes;
                int ks = 0;
                for (int r = 0; r < p.kh; ++r) {
                    for (int sx = 0; sx < p.kw; ++sx) {
                        // the tap's pixels: the same box, (r * pw + sx) rows of 128 bytes further on
                        const uint32_t shift = (uint32_t)(r * p.pw + sx) * 128u;
                        const uint64_t db_hi = smem_desc_k<128>(x_hi + shift), db_lo = smem_desc_k<128>(x_lo + shift);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk, ++ks) {
                            const uint64_t adv    = (uint64_t)(kk * 32 >> 4);
                            const uint32_t a_tmem = tmem_base + (uint32_t)(ks * 8);
                            mma_tf32_a_tmem(d_tmem, a_tmem, db_lo + adv, idesc, ks == 0 ? 0u : 1u);
                            mma_tf32_a_tmem(d_tmem, a_tmem, db_hi + adv, idesc, 1u);
                        }
                    }
                }
                tc_commit(smem_u32(&bar_empty[s]));   // the stage is free once these MMAs have retired
                tc_commit(smem_u32(&bar_tmem_full));  // and the accumulator is complete
            }
            CV_ACCUM(2, CV_CLOCK() - t_start); // the MMA thread's whole loop
            CV_ACCUM(3, i);
            if (!ok || *abort_flag) {
                tc_commit(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else if (RAW && warp < 2 + kTA_CvtWarps) {
        // ===== raw mode: float32 box -> hi / lo planes =====
        // A thread takes a position (y, x) of the box: its 32 channel values lie box_rows * box_w floats
        // apart in the raw box (consecutive lanes read consecutive x: no bank conflicts) and become the
        // 128-byte row y * pw + x of both planes, 16-byte chunk j at chunk j ^ (row & 7) - the 128-byte
        // swizzle the MMA's descriptors expect.
        // (these warps come before the epilogue warps: the schedulers favour older warps, and eight
        // epilogue warps polling their barrier kept younger converting warps from issuing - a tile's
        // conversion took 9900 clocks behind them)
        const int ct   = threadIdx.x - 64;
        const int npos = p.box_rows * p.pw;
        const int cstride = p.box_rows * p.box_w; // floats between two channels of one position
        int i = 0;
        for (int q = next_own(own_mask, 0, own); q < own; q = next_own(own_mask, q + 1, own), ++i) {
            const int rs       = i % kTA_RawStages;
            const uint32_t rph = (uint32_t)(i / kTA_RawStages) & 1u;
            const int s        = i % p.stages;
            const uint32_t ph  = (uint32_t)(i / p.stages) & 1u;
            const long long v0 = CV_CLOCK();
            bool got = mbar_wait_patient(smem_u32(&bar_raw_full[rs]), rph, abort_flag);
            const long long v1 = CV_CLOCK();
            got      = got && mbar_wait_patient(smem_u32(&bar_empty[s]), ph ^ 1u, abort_flag); // the planes' stage is free
            if (!__all_sync(0xffffffffu, got))
                break;
            const long long v2 = CV_CLOCK();
            const float *raw = reinterpret_cast<const float *>(smem_raw + (raw_base - smem_u32(smem_raw)) + (uint32_t)rs * (uint32_t)p.raw_stride);
            uint8_t *x_hi    = smem_raw + (smem_base - smem_u32(smem_raw)) + (uint32_t)s * stage_bytes;
            uint8_t *x_lo    = x_hi + p.plane_bytes;
            for (int pos = ct; pos < npos; pos += 32 * kTA_CvtWarps) {
                const int y = pos / p.pw, x = pos - y * p.pw;
                const float *src = raw + y * p.box_w + x + p.off_x;
                const uint32_t row_off = (uint32_t)pos * 128u;
                const uint32_t sw      = (uint32_t)pos & 7u;
                // sixteen channels at a time: all their loads first (a store to shared memory in between
                // would hold back the loads behind it), then the splits and the eight stores
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float v[16];
#pragma unroll
                    for (int t = 0; t < 16; ++t)
                        v[t] = src[(16 * half + t) * cstride];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float hi[4], lo[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            split_tf32_flat(v[4 * j + t], hi[t], lo[t]);
                        const uint32_t at = row_off + (((uint32_t)(4 * half + j) ^ sw) << 4);
                        *reinterpret_cast<float4 *>(x_hi + at) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                        *reinterpret_cast<float4 *>(x_lo + at) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                    }
                }
            }
            // the planes were written through the generic proxy and are read by the tensor core's
            // asynchronous proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&bar_full[s]));
                mbar_arrive(smem_u32(&bar_raw_empty[rs]));
            }
            if (ct == 0) {
                CV_ACCUM(9, v1 - v0);            // converter: waiting for the raw box
                CV_ACCUM(10, v2 - v1);           // waiting for a free plane stage
                CV_ACCUM(11, CV_CLOCK() - v2);   // converting
            }
        }
    } else {
        // ===== epilogue =====
        const int quarter = warp & 3;        // TMEM lanes this warp may read: 32 * quarter ..
        const int ew      = warp - (RAW ? 2 + kTA_CvtWarps : 2); // 0..7: which channels this warp writes out
        const int half    = ew >> 2;         // which 64 columns of the accumulator it drains
        uint32_t epi_phase = 0;
        auto epi_sync = [&]() -> bool {
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&bar_epi));
            bool ok = mbar_wait_patient(smem_u32(&bar_epi), epi_phase, abort_flag);
            epi_phase ^= 1u;
            return __all_sync(0xffffffffu, ok);
        };
        // Where this lane's positions land, once for the whole kernel: position pos = lane + 32 g
        // of a tile is pixel (y, x) = (pos / pw, pos % pw) of the tile's rows; -1 for the halo columns
        // and past the tile.  With the pool: lane q = pooled pixel (py, px) of the tile.
        int off[4], yy[4];
        const int npos = p.th * p.pw;
        const int pw2 = p.wo >> 1, ph2 = p.ho >> 1;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int pos = lane + 32 * g;
            off[g] = -1, yy[g] = 0;
            if (p.pool == 0) {
                const int y = pos / p.pw, x = pos - y * p.pw;
                if (pos < npos && x < p.wo)
                    off[g] = y * p.wo + x, yy[g] = y;
            } else {
                const int py = pos / pw2, px = pos - py * pw2;
                if (py < (p.th >> 1))
                    off[g] = (2 * py) * p.pw + 2 * px, yy[g] = py; // here: the window's first position
            }
        }
        // this warp's channels are the same for every tile: their bias values are read once (a load
        // per channel inside the tile loop costs a trip to L2 that the add then waits for)
        float bias_r[64 / kTA_EpiWarps];
#pragma unroll
        for (int j = 0; j < 64 / kTA_EpiWarps; ++j) {
            const int ch = ew + kTA_EpiWarps * j;
            bias_r[j]    = (p.bias && ch < p.ko) ? p.bias[ch] : 0.0f;
        }
        int i = 0;
        for (int q = next_own(own_mask, 0, own); q < own; q = next_own(own_mask, q + 1, own), ++i) {
            const int tile = (int)blockIdx.x + q * (int)gridDim.x;
            const int img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
            const long long e0 = CV_CLOCK();
            bool got = mbar_wait_patient(smem_u32(&bar_tmem_full), (uint32_t)i & 1u, abort_flag);
            if (!__all_sync(0xffffffffu, got))
                break;
            const long long e1 = CV_CLOCK();
            const int y0 = ty * p.th;
            tc_fence_after_sync();
            // lane m of the accumulator -> row m of the staging block
            float4 *mine = reinterpret_cast<float4 *>(staging + (quarter * 32 + lane) * kTA_StageRowF + half * 64);
            const uint32_t taddr =
                tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(kTA_DCol + half * 64);
            // both halves of this warp's 64 columns are requested before the one wait, and the
            // accumulator is handed back as soon as the values are in registers: the next tile's
            // MMAs then start while these threads are still writing the staging block
            uint32_t r0[32], r1[32];
            tmem_ld_32x32(taddr, r0);
            tmem_ld_32x32(taddr + 32, r1);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&bar_tmem_empty)); // the next tile's MMAs may start
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                mine[j]     = make_float4(__uint_as_float(r0[4 * j]), __uint_as_float(r0[4 * j + 1]),
                                          __uint_as_float(r0[4 * j + 2]), __uint_as_float(r0[4 * j + 3]));
                mine[8 + j] = make_float4(__uint_as_float(r1[4 * j]), __uint_as_float(r1[4 * j + 1]),
                                          __uint_as_float(r1[4 * j + 2]), __uint_as_float(r1[4 * j + 3]));
            }
            const long long e2 = CV_CLOCK();
            if (!epi_sync())
                break;
            const long long e3 = CV_CLOCK();
            // which of this lane's four positions are stored for this tile (rows past the image's
            // last row of a partial tile are not)
            unsigned okmask = 0;
#pragma unroll
            for (int g = 0; g < 4; ++g)
                if (off[g] >= 0 && (p.pool ? (y0 >> 1) + yy[g] < ph2 : y0 + yy[g] < p.ho))
                    okmask |= 1u << g;
            // Two channels at a time, every load of the pair before the first dependent instruction, no
            // branch inside: a channel past the last filter or a position that is not stored is masked
            // at the store (its loads read rows of the staging block that hold nothing of interest).
            if (p.pool == 0) {
#pragma unroll
                for (int jj = 0; jj < 64 / kTA_EpiWarps; jj += 2) {
                    float h[2][4], l[2][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int ch    = ew + kTA_EpiWarps * (jj + u);
                        const float *hi = staging + ch * kTA_StageRowF + lane, *lo = hi + 64 * kTA_StageRowF;
#pragma unroll
                        for (int g = 0; g < 4; ++g)
                            h[u][g] = hi[32 * g], l[u][g] = lo[32 * g];
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int ch = ew + kTA_EpiWarps * (jj + u);
                        const float b = bias_r[jj + u];
                        float *plane  = p.out + (((int64_t)img * p.ko + ch) * p.ho + y0) * p.wo;
                        const unsigned mask = ch < p.ko ? okmask : 0u;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            float v = __fadd_rn(h[u][g], l[u][g]);
                            if (p.bias)
                                v = __fadd_rn(v, b);
                            if (p.act == CT_ACT_RELU)
                                v = __fmul_rn(v, v > 0.0f ? 1.0f : 0.0f);
                            if (mask & (1u << g))
                                plane[off[g]] = v;
                        }
                    }
                }
            } else {
                // 2x2 max-pool of the activated values; window order and strict '>' as in
                // maxpool2d (the first element seeds, a NaN never wins)
                const int pooled = (p.th >> 1) * pw2;           // pooled pixels of a tile
                const int groups = (pooled + 31) >> 5;          // the same for every lane: no divergence
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (g >= groups)
                        break;
                    const bool live = (okmask >> g) & 1u;
                    const int pos   = live ? off[g] : 0;
#pragma unroll
                    for (int jj = 0; jj < 64 / kTA_EpiWarps; jj += 2) {
                        float h[2][4], l[2][4];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int ch    = ew + kTA_EpiWarps * (jj + u);
                            const float *hi = staging + ch * kTA_StageRowF + pos, *lo = hi + 64 * kTA_StageRowF;
                            h[u][0] = hi[0], h[u][1] = hi[1], h[u][2] = hi[p.pw], h[u][3] = hi[p.pw + 1];
                            l[u][0] = lo[0], l[u][1] = lo[1], l[u][2] = lo[p.pw], l[u][3] = lo[p.pw + 1];
                        }
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int ch  = ew + kTA_EpiWarps * (jj + u);
                            const float b = bias_r[jj + u];
                            float v[4];
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                v[t] = __fadd_rn(h[u][t], l[u][t]);
                                if (p.bias)
                                    v[t] = __fadd_rn(v[t], b);
                                if (p.act == CT_ACT_RELU)
                                    v[t] = __fmul_rn(v[t], v[t] > 0.0f ? 1.0f : 0.0f);
                            }
                            float best = v[0];
                            if (v[1] > best)
                                best = v[1];
                            if (v[2] > best)
                                best = v[2];
                            if (v[3] > best)
                                best = v[3];
                            if (live && ch < p.ko) {
                                float *plane = p.out + (((int64_t)img * p.ko + ch) * ph2 + (y0 >> 1)) * pw2;
                                plane[lane + 32 * g] = best; // pooled pixels of a tile are consecutive: py * pw2 + px
                            }
                        }
                    }
                }
            }
            const long long e4 = CV_CLOCK();
            if (!epi_sync()) // the staging block is rewritten by the next tile
                break;
            if (ew == 0 && lane == 0) {
                CV_ACCUM(4, e1 - e0);           // epilogue: waiting for the accumulator to be complete
                CV_ACCUM(5, e2 - e1);           // drain
                CV_ACCUM(6, e3 - e2);           // first meeting of the epilogue warps
                CV_ACCUM(7, e4 - e3);           // add, activate, store
                CV_ACCUM(8, CV_CLOCK() - e4);   // second meeting
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && *abort_flag)
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

// ---- split float16 --------------------------------------------------------------------------
//
// Two 11-bit terms in float16 instead of tf32 (half_split.cuh), pixels on the accumulator rows.  A tile is 2 jp output
// rows of an image: its even rows are the 128 rows of one accumulator, its odd rows those of another, positions j * pw + x
// each.  A CTA has a tile, or two tiles belong to a pair of CTAs whose MMAs (cta_group::2) are issued by the leader.  The input rows of a
// tile lie in shared memory as two regions, even and odd rows of the box, so that filter tap
// (r, s) is, for the even (odd) output rows, region r & 1 ((r + 1) & 1) through a descriptor moved by
// (r >> 1) * pw + s (((r + 1) >> 1) * pw + s) rows.  The filters are the B operand and stay in shared memory for the
// whole launch: hi and lo terms in a CTA by itself; in a pair the leader has the hi and its peer the lo terms, and each half of the hi
// terms once more.  Per 16 channels and tap two MMAs an accumulator:
//     [main | cross] += X_hi x [W_hi; W_lo]     N = 2 kop
//             cross  += X_lo x W_hi             N = kop
// with the low terms stored 2^11 times larger and the cross products in columns of their own, as in gemm_half.cu.  The product of
// two low terms (2^-24 of a product) is left out: it would be half as much work again (256 x 32 x 28 x 28 -> 64 44 us, with it 54).
// What errs most are the additions, which truncate.  So the leading product of the last k-step does not join the others': when all
// cross products are in, this MMA moves their columns down by 2^11, by the scale of its D, and adds to them, and the chain
// is a step shorter (256 x 32 x 28 x 28 -> 64 44.2 -> 44.9 us).  That makes up for the product of the low terms: against 64 bits
// 3.66e-7 -> 3.39e-7, with them 3.64e-7; 16 channels 2.19e-7 -> 1.93e-7.
//
// Why so.  With the filters on the rows and in tensor memory (hi and lo terms on rows 0 - 63 and 64 - 127, the layout of the
// tf32 form above) the two halves of an output met in shared memory, 128 KB a tile of 128 positions, and that epilogue
// took 5200 clocks where the MMAs took 2628.  Here a lane holds a pixel and its registers channels: the two accumulators'
// rows are vertical neighbours, horizontal ones are lanes, so the sum, the activation, the 2x2 maximum and the store
// need no shared memory at all, and a store covers consecutive pixels of a channel.
//
// Shared memory is what bounds it (128 bytes per clock): at 32 channels and 64 filters a CTA by itself reads 14 KB for the two MMAs of a k-step,
// 5900 clocks a tile with what the conversion reads and writes; each CTA of a pair reads 11 KB, 3600 clocks of a tile's 6500, and
// what is left is the epilogue (5000), which waits for the same memory.  With one k-step to a tap or fewer filters the pair's
// larger start and padding cost more than that (conv_pair_form has both sides).  Sixteen epilogue warps instead of eight are no faster (889
// us: 72 registers a thread).
//
// Scales: per filter, and per tile (raw: the converting warps see the whole box before they split it) or, from planes, per
// image.  The converting warps also leave the range of every tile in the call's own scratch; conv_tmem_filters_kernel,
// launched behind this one, computes the images that float16 pairs cannot hold.  A tile that shows that by itself is
// neither converted nor stored here; what its stage happens to hold is multiplied, and nobody reads the sums.
// Converting warps: with ten the boxes of up to 320 positions are held in registers (30 x 10 of a 28 x 28 image), larger ones are read
// twice.  Against the kernel before, 256 images, 3 x 3: 32 -> 64 channels at 12 x 12 36 -> 23 us, 28 x 28 65 -> 44, 32 x 32 90 -> 61,
// 40 x 40 146 -> 114, 60 x 60 298 -> 238; 16 -> 32 at 56 x 56 233 -> 151.
// Two float32 operations in one instruction, each rounded as by itself.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
constexpr int kCP_CvtWarps  = 10;
constexpr int kCP_EpiWarps  = 8;
constexpr int kCP_Threads   = 64 + 32 * (kCP_CvtWarps + kCP_EpiWarps);
constexpr int kCP_RowB      = 64; // a position's 32 channels
constexpr int kCP_MaxStages = 4;
constexpr int kCP_Smem      = 226 * 1024;

struct ConvPairParams {
    const float *w;    // filters [ko][c][kh][kw], float32
    const float *bias;
    float *out;        // [batch][ko][ho][wo], or [batch][ko][ho/2][wo/2] with pool
    uint32_t *flags;
    int ko, kop, c, kh, kw, pad; // kop: ko rounded up to 16, for a pair to 32, the columns of an MMA
    int ho, wo, pw;    // pw = input width + 2 pad
    int jp, tiles_y;   // pairs of output rows per tile, tiles per image
    int region_rows;   // input rows of a region
    int region_bytes;  // shared memory of a region of one plane
    int filter_bytes;
    int stages;
    int act, pool;
    const float *image_scale; // planes: [batch] inverse scales, 0 for an image that needs tf32 terms
    uint2 *tile_range;        // as in ConvTmemParams
    // raw mode, as in ConvTmemParams
    int box_w, off_x, box_rows, raw_bytes, raw_stride;
};

template <bool RAW, int CG>
__global__ void __launch_bounds__(kCP_Threads, 1) conv_pairs_kernel(
    const __grid_constant__ CUtensorMap map_x_hi, const __grid_constant__ CUtensorMap map_x_lo,
    const __grid_constant__ ConvPairParams p, const int total_tiles) {
    griddep_launch_dependents(); // the tf32 form, which allocates no tensor memory before this kernel ends
    griddep_wait();
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[kCP_MaxStages], bar_empty[kCP_MaxStages];
    __shared__ uint64_t bar_raw_full, bar_raw_empty;
    __shared__ uint64_t bar_scale_full[kCP_MaxStages], bar_scale_empty[kCP_MaxStages]; // the tile's scale is there, has been read by the epilogue
    __shared__ uint64_t bar_acc_full[2], bar_acc_empty[2]; // tiles alternate between two sets of 256 columns
    __shared__ uint64_t bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s, filters_wide_s, cvt_word[2], epi_word[2];
    __shared__ uint2 cvt_range[2][kCP_CvtWarps];
    __shared__ float tile_scale[kCP_MaxStages]; // inverse scale of the tile in each plane stage; 0: left to the tf32 form
    __shared__ __align__(16) float filter_inv[64], bias_s[64];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31; // known to be the same for the warp
    const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0; // in the cluster of two
    const int first = (int)blockIdx.x / CG, stride = (int)gridDim.x / CG, passes = (total_tiles + CG - 1) / CG;
    if (threadIdx.x == 0) {
        abort_flag_s   = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
        filters_wide_s = 0;
    }
    if (threadIdx.x < 64) {
        filter_inv[threadIdx.x] = 1.0f;
        bias_s[threadIdx.x]     = p.bias && (int)threadIdx.x < p.ko ? p.bias[threadIdx.x] : -0.0f; // which no sum notices
    }

    const uint32_t smem_base   = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *const smem_ptr    = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t region      = (uint32_t)p.region_bytes;
    const uint32_t stage_bytes = 4u * region; // hi even, hi odd, lo even, lo odd
    const uint32_t stage_base  = smem_base + (uint32_t)p.filter_bytes;
    const uint32_t raw_base    = stage_base + (uint32_t)p.stages * stage_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), RAW ? CG * kCP_CvtWarps : 1); // of both CTAs
            mbar_init(smem_u32(&bar_empty[s]), 1);
            mbar_init(smem_u32(&bar_scale_full[s]), 1);
            mbar_init(smem_u32(&bar_scale_empty[s]), kCP_EpiWarps);
        }
        mbar_init(smem_u32(&bar_raw_full), 1);
        mbar_init(smem_u32(&bar_raw_empty), kCP_CvtWarps);
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), CG * kCP_EpiWarps);
        }
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        prefetch_tensormap(&map_x_hi);
        prefetch_tensormap(&map_x_lo);
    }
    __syncthreads(); // the defaults of filter_inv
    float *filters = reinterpret_cast<float *>(smem_ptr + p.filter_bytes); // where the stages will be
    const int taps = p.kh * p.kw, filter_stride = (p.c * taps) | 1;
    stage_filters(p.w, p.ko, p.c * taps, filters, warp, kCP_Threads / 32, lane, [&](int f, uint2 range) {
        float scale, inverse;
        const bool fits = half_range_fits(range_warp(range), scale, inverse);
        if (lane == 0) {
            filter_inv[f] = inverse;
            if (!fits)
                filters_wide_s = 1;
        }
    });
    if (warp == 1) {
        if (CG == 2) {
            tmem_alloc_pair(smem_u32(&tmem_base_slot), 512);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(&tmem_base_slot), 512);
            tmem_relinquish();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    const bool failed        = abort_flag_s != 0;   // an earlier launch failed: no work
    const bool filters_wide  = filters_wide_s != 0; // every tile is left to the tf32 form
    if (RAW && blockIdx.x == 0 && threadIdx.x == 0)
        p.tile_range[total_tiles] = make_uint2(filters_wide ? 1u : 0u, 0u);

    // ---- the filters' planes, once, 64-byte rows, swizzled.  One CTA: per tap kop rows of hi, then of lo terms.  A pair: per tap kop rows of
    // the leader's hi or its peer's lo terms; behind those of all taps, per tap half of the hi terms; then half of the last tap's lo
    // terms ----
    const int half_rows = p.kop >> 1, q_at = CG == 2 ? taps * p.kop : 0, r_at = CG == 2 ? q_at + taps * half_rows : (2 * taps - 1) * p.kop;
    const int shift = p.kop == 64 ? 6 : 5; // a pair's is 32 or 64
    if (!filters_wide)
        for (int i = threadIdx.x; i < taps * p.kop * 4; i += kCP_Threads) {
            const int chunk = i & 3, row = i >> 2, tap = CG == 2 ? row >> shift : row / p.kop, f = row - tap * p.kop, c0 = chunk * 8;
            const float *src  = filters + f * filter_stride;
            const float scale = 1.0f / filter_inv[f]; // both are powers of two
            __half2 hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int ic  = c0 + 2 * j;
                const float a = (f < p.ko && ic < p.c) ? src[ic * taps + tap] : 0.0f;
                const float b = (f < p.ko && ic + 1 < p.c) ? src[(ic + 1) * taps + tap] : 0.0f;
                split_half_pair(a * scale, b * scale, hi[j], lo[j]);
            }
            auto put = [&](int to, const __half2 (&v)[4]) {
                *reinterpret_cast<uint4 *>(smem_ptr + (size_t)to * kCP_RowB + ((chunk ^ ((to >> 1) & 3)) << 4)) = *reinterpret_cast<const uint4 *>(v);
            };
            if (CG == 1) {
                put(row + tap * p.kop, hi);
                put(row + tap * p.kop + p.kop, lo);
                continue;
            }
            if (rank)
                put(row, lo);
            else
                put(row, hi);
            const int mine = f - rank * half_rows;
            if (mine >= 0 && mine < half_rows) {
                put(q_at + tap * half_rows + mine, hi);
                if (tap == taps - 1)
                    put(r_at + mine, lo);
            }
        }
    filters_taken();
    __syncthreads();
    if (CG == 2)
        cluster_sync(); // the MMAs read both CTAs' filters, and nothing is signalled on the partner's barriers before they exist

    // this CTA's tile of pass u (the last may have one for a pair: then both compute it, and the leader stores it), and, from planes, whether
    // either image of the pass is left to this kernel
    auto tile_of = [&](int u) { return CG == 2 ? min(2 * u + rank, total_tiles - 1) : u; };
    auto wanted  = [&](int u) {
        return RAW || __any_sync(0xffffffffu, p.image_scale[CG * u / p.tiles_y] != 0.0f ||
                                                  (CG == 2 && p.image_scale[min(2 * u + 1, total_tiles - 1) / p.tiles_y] != 0.0f));
    };

    if (filters_wide || failed) {
    } else if (warp == 0) {
        // ===== TMA producer: one box per plane and region (raw mode: one box of the input) =====
        int i = 0;
        const int nstages = RAW ? 1 : p.stages;
        for (int u = first; u < passes; u += stride) {
            if (!wanted(u))
                continue;
            const int tile = tile_of(u), img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
            const int s       = i % nstages;
            const uint32_t ph = (uint32_t)(i / nstages) & 1u;
            if (!mbar_wait_patient_warp(smem_u32(RAW ? &bar_raw_empty : &bar_empty[s]), ph ^ 1u, abort_flag))
                break;
            const int32_t h0 = ty * 2 * p.jp - p.pad;
            if (elect_one()) {
                if (RAW) {
                    const uint32_t full = smem_u32(&bar_raw_full);
                    mbar_expect_tx(full, (uint32_t)p.raw_bytes);
                    // the box starts off_x floats left of x = -pad so that its first byte is 16-byte aligned
                    tma_load_4d(raw_base, &map_x_hi, full, -p.pad - p.off_x, h0, 0, img);
                } else {
                    const uint32_t full = smem_u32(&bar_full[s]), dst = stage_base + (uint32_t)s * stage_bytes;
                    if (rank == 0) // both CTAs' bytes are counted on the leader's barrier
                        mbar_expect_tx(full, (uint32_t)CG * 4u * (uint32_t)(p.region_rows * p.pw * kCP_RowB));
                    for (int g = 0; g < 2; ++g) { // region g: rows h0 + g + 2 i, which lie in one of the two sub-images
                        const int32_t row = (h0 + g) >> 1, sub = (h0 + g) & 1;
                        if (CG == 2) {
                            tma_load_5d_pair(dst + (uint32_t)g * region, &map_x_hi, leader_addr(full), 0, -p.pad, row, sub, img);
                            tma_load_5d_pair(dst + (uint32_t)(2 + g) * region, &map_x_lo, leader_addr(full), 0, -p.pad, row, sub, img);
                        } else {
                            tma_load_5d(dst + (uint32_t)g * region, &map_x_hi, full, 0, -p.pad, row, sub, img);
                            tma_load_5d(dst + (uint32_t)(2 + g) * region, &map_x_lo, full, 0, -p.pad, row, sub, img);
                        }
                    }
                }
            }
            __syncwarp();
            ++i;
        }
        if (*abort_flag && (RAW || rank == 0)) {
            // unwind: let the copies still in flight land before the CTA goes away (from planes the leader's barriers count the
            // partner's copies too, and neither CTA leaves before the other)
            for (int k2 = i - nstages < 0 ? 0 : i - nstages; k2 < i; ++k2) {
                const uint32_t bar = smem_u32(RAW ? &bar_raw_full : &bar_full[k2 % nstages]);
                const uint64_t t0  = globaltimer_ns();
                while (!mbar_try_wait(bar, (uint32_t)(k2 / nstages) & 1u) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        // (the leader's, for a pair; a whole warp with uniform control flow, so that descriptors stay in uniform registers)
        if (rank == 0) {
            const uint32_t idesc2 = make_idesc(0u, 128 * CG, (uint32_t)(2 * p.kop)), idesc1 = make_idesc(0u, 128 * CG, (uint32_t)p.kop);
            const bool two = p.c > 16; // k-steps that hold channels
            // descriptors are moved by adding to their address field (16-byte units; shared memory is far below its range)
            const uint32_t unit = kCP_RowB >> 4, lo_terms = 2 * region >> 4, kop = (uint32_t)p.kop;
            const uint32_t p_step = (CG == 2 ? kop : 2 * kop) * unit, q_step = (CG == 2 ? kop >> 1 : 2 * kop) * unit;
            const uint32_t p_0 = (uint32_t)smem_desc_k<kCP_RowB>(smem_base), q_0 = p_0 + (uint32_t)q_at * unit, last_lo = p_0 + (uint32_t)r_at * unit;
            auto desc = [](uint32_t low) { return smem_desc_k<kCP_RowB>(0) & 0xffffffff00000000ull | low; };
            int i   = 0, s = 0;
            uint32_t full_phase = 0;
            bool ok = true;
            for (int u = first; u < passes; u += stride) {
                if (!wanted(u))
                    continue;
                const int set = i & 1;
                // the accumulators have been read, the planes are complete
                ok = mbar_wait_warp<CG == 2 ? kClusterRead : kCta>(smem_u32(&bar_acc_empty[set]), ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag) &&
                     mbar_wait_warp<RAW && CG == 2 ? kClusterWritten : kCta>(smem_u32(&bar_full[s]), full_phase, abort_flag);
                if (!ok)
                    break;
                tc_fence_after_sync();
                const uint32_t hi0 = stage_base + (uint32_t)s * stage_bytes;
                const uint32_t d_even = tmem_base + (uint32_t)(set * 256), d_odd = d_even + 128u;
                uint32_t w_p = p_0, w_q = q_0, accumulate = 0u;
                auto step = [&](uint32_t even, uint32_t odd, uint32_t k, uint32_t acc) {
                    mma_f16_warp<CG>(d_even, desc(even + k), desc(w_p + k), idesc2, acc);
                    mma_f16_warp<CG>(d_odd, desc(odd + k), desc(w_p + k), idesc2, acc);
                    mma_f16_warp<CG>(d_even + kop, desc(even + lo_terms + k), desc(w_q + k), idesc1, 1u);
                    mma_f16_warp<CG>(d_odd + kop, desc(odd + lo_terms + k), desc(w_q + k), idesc1, 1u);
                };
                for (int r = 0; r < p.kh; ++r) {
                    // the tap's pixels for the even and the odd output rows
                    uint32_t even = (uint32_t)smem_desc_k<kCP_RowB>(hi0 + (uint32_t)(r & 1) * region + (uint32_t)((r >> 1) * p.pw * kCP_RowB));
                    uint32_t odd  = (uint32_t)smem_desc_k<kCP_RowB>(hi0 + (uint32_t)((r + 1) & 1) * region + (uint32_t)(((r + 1) >> 1) * p.pw * kCP_RowB));
                    const int whole = r + 1 < p.kh ? p.kw : p.kw - 1; // all but the last tap
                    for (int sx = 0; sx < whole; ++sx, even += unit, odd += unit, w_p += p_step, w_q += q_step) {
                        step(even, odd, 0, accumulate);
                        accumulate = 1u;
                        if (two)
                            step(even, odd, 2, 1u);
                    }
                    if (r + 1 == p.kh) {
                        uint32_t k = 0;
                        if (two)
                            step(even, odd, 0, 1u), k = 2;
                        mma_f16_warp<CG>(d_even + kop, desc(even + lo_terms + k), desc(w_q + k), idesc1, 1u);
                        mma_f16_warp<CG>(d_odd + kop, desc(odd + lo_terms + k), desc(w_q + k), idesc1, 1u);
                        mma_f16_warp<CG>(d_even + kop, desc(even + k), desc(last_lo + k), idesc1, 1u);
                        mma_f16_warp<CG>(d_odd + kop, desc(odd + k), desc(last_lo + k), idesc1, 1u);
                        mma_f16_shifted_warp<kHalfLoBits, CG>(d_even + kop, desc(even + k), desc(w_q + k), idesc1);
                        mma_f16_shifted_warp<kHalfLoBits, CG>(d_odd + kop, desc(odd + k), desc(w_q + k), idesc1);
                    }
                }
                tc_commit_warp<CG>(smem_u32(&bar_empty[s]));      // the stage is free once these MMAs have retired
                tc_commit_warp<CG>(smem_u32(&bar_acc_full[set])); // and the accumulators are complete
                ++i;
                if (++s == p.stages)
                    s = 0, full_phase ^= 1u;
            }
            if (!ok || *abort_flag) {
                __syncwarp();
                tc_commit_warp<CG>(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else if (warp < 2 + kCP_CvtWarps) {
        // ===== raw mode: float32 box -> float16 planes (warps before the epilogue's: the schedulers favour older warps) =====
        if (RAW) {
            const int ct      = threadIdx.x - 64;
            const int npos    = p.box_rows * p.pw;
            const int cstride = p.box_rows * p.box_w; // floats between two channels of one position
            const float *raw  = reinterpret_cast<const float *>(smem_ptr + (raw_base - smem_base));
            const bool one    = npos <= 32 * kCP_CvtWarps;
            const int first_raw = ct / p.pw * p.box_w + ct % p.pw + p.off_x;
            int i = 0, s = 0;
            uint32_t stage_phase = 1u;
            for (int u = first; u < passes; u += stride, ++i) {
                const int tile = tile_of(u);
                if (!group_wait(
                        warp == 2, [&] { return mbar_wait(smem_u32(&bar_raw_full), (uint32_t)i & 1u, abort_flag); }, cvt_word, 0, 1, 32 * kCP_CvtWarps))
                    break;
                // The tile's range.  Where every thread has at most one position its channels stay in registers between the range
                // and the split, and the box is free for the next tile's before this one's planes are.
                uint2 range = make_uint2(0u, kNoneSmallest);
                float v[32];
                if (one) {
                    const float *src = raw + (ct < npos ? first_raw : 0);
#pragma unroll
                    for (int t = 0; t < 32; ++t)
                        v[t] = ct < npos ? src[t * cstride] : 0.0f;
#pragma unroll
                    for (int t = 0; t < 32; ++t)
                        range_take(range, v[t]);
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(smem_u32(&bar_raw_empty));
                } else { // the whole box, alignment columns included: they are pixels or zero
                    const float4 *r4 = reinterpret_cast<const float4 *>(raw);
#pragma unroll 4
                    for (int e = ct; e < p.raw_bytes / 16; e += 32 * kCP_CvtWarps) {
                        const float4 q = r4[e];
                        range_take(range, q.x), range_take(range, q.y), range_take(range, q.z), range_take(range, q.w);
                    }
                }
                range = range_warp(range);
                if (lane == 0)
                    cvt_range[i & 1][warp - 2] = range;
                // all ranges are there, the stage is free, and so is its scale
                if (!group_wait(
                        warp == 2,
                        [&] {
                            return mbar_wait(smem_u32(&bar_empty[s]), stage_phase, abort_flag) &&
                                   mbar_wait(smem_u32(&bar_scale_empty[s]), stage_phase, abort_flag);
                        },
                        cvt_word, 1, 1, 32 * kCP_CvtWarps))
                    break;
#pragma unroll
                for (int u = 0; u < kCP_CvtWarps; ++u)
                    range = range_join(range, cvt_range[i & 1][u]);
                float scale, inverse;
                const bool fits = half_tile_fits(range, scale, inverse);
                if (ct == 0) {
                    tile_scale[s] = fits ? inverse : 0.0f;
                    mbar_arrive(smem_u32(&bar_scale_full[s])); // the planes' barrier is the leader's
                }
                uint8_t *planes = smem_ptr + p.filter_bytes + (uint32_t)s * stage_bytes;
                // a position's (y, x) 32 channels become row (y >> 1) * pw + x of region y & 1 in both planes, 16-byte chunk j
                // at j ^ ((row >> 1) & 3), the 64-byte swizzle
                auto put = [&](int pos) {
                    const int y = pos / p.pw, x = pos - y * p.pw, row = (y >> 1) * p.pw + x;
                    uint8_t *dst     = planes + (uint32_t)(y & 1) * region + (uint32_t)row * kCP_RowB;
                    const uint32_t sw = ((uint32_t)row >> 1) & 3u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        __half2 hi[4], lo[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            split_half_pair(__fmul_rn(v[8 * j + 2 * t], scale), __fmul_rn(v[8 * j + 2 * t + 1], scale), hi[t], lo[t]);
                        const uint32_t at = ((uint32_t)j ^ sw) << 4;
                        *reinterpret_cast<uint4 *>(dst + at)              = *reinterpret_cast<uint4 *>(hi);
                        *reinterpret_cast<uint4 *>(dst + 2 * region + at) = *reinterpret_cast<uint4 *>(lo);
                    }
                };
                if (one) {
                    if (fits && ct < npos)
                        put(ct);
                } else {
                    for (int pos = fits ? ct : npos; pos < npos; pos += 32 * kCP_CvtWarps) {
                        const int y = pos / p.pw;
                        const float *src = raw + y * p.box_w + pos - y * p.pw + p.off_x;
#pragma unroll
                        for (int t = 0; t < 32; ++t)
                            v[t] = src[t * cstride];
                        put(pos);
                    }
                }
                // written through the generic proxy, read by the tensor core's asynchronous proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2)
                        mbar_arrive_peer_written(leader_addr(smem_u32(&bar_full[s])));
                    else
                        mbar_arrive(smem_u32(&bar_full[s]));
                    if (!one)
                        mbar_arrive(smem_u32(&bar_raw_empty));
                }
                if (ct == 0)
                    p.tile_range[tile] = range;
                if (++s == p.stages)
                    s = 0, stage_phase ^= 1u;
            }
        }
    } else {
        // ===== epilogue: a lane has a position, groups of sixteen channels in turn =====
        const int quarter = warp & 3;                       // TMEM lanes this warp may read
        const int half    = (warp - 2 - kCP_CvtWarps) >> 2; // which groups of channels are its
        const int m = quarter * 32 + lane, j = m / p.pw, x = m - j * p.pw;
        const int groups = p.kop >> 4;
        const int64_t plane = p.pool ? (int64_t)(p.ho >> 1) * (p.wo >> 1) : (int64_t)p.ho * p.wo;
        const bool inside = j < p.jp && x < p.wo && !(p.pool && (x & 1));
        const bool relu = p.act == CT_ACT_RELU;
        int i = 0, s = 0;
        uint32_t scale_phase = 0;
        for (int u = first; u < passes; u += stride) {
            if (!wanted(u))
                continue;
            const int tile = tile_of(u), img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
            const bool mine = CG * u + rank < total_tiles;
            const int set = i & 1;
            if (!group_wait(
                    warp == 2 + kCP_CvtWarps,
                    [&] {
                        return mbar_wait(smem_u32(&bar_acc_full[set]), (uint32_t)(i >> 1) & 1u, abort_flag) &&
                               (!RAW || mbar_wait(smem_u32(&bar_scale_full[s]), scale_phase, abort_flag));
                    },
                    epi_word, i, 2, 32 * kCP_EpiWarps))
                break;
            const float is = RAW ? *const_cast<volatile float *>(&tile_scale[s]) : p.image_scale[img];
            tc_fence_after_sync();
            const int y = (ty * p.jp + j) * 2; // the even row; the odd one may be past the image
            const bool live_even = inside && y < p.ho, live_low = inside && !p.pool && y + 1 < p.ho; // pooled rows are even and odd
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * 256);
            float *dst = p.out + ((int64_t)img * p.ko + half * 16) * plane + (p.pool ? (int64_t)(y >> 1) * (p.wo >> 1) + (x >> 1) : (int64_t)y * p.wo + x);
            const uint64_t is2 = pack2(is, is);
            // Values of sixteen channels, then their neighbours, then the stores, without a branch among them: channel after
            // channel, with the activation behind a branch, a group took 4300 clocks.
            for (int g = half; g < groups && is != 0.0f && mine; g += 2, dst += 32 * plane) {
                float even[16], odd[16];
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    uint32_t a[8], b[8], c[8], d[8];
                    tmem_ld_32x8(taddr + (uint32_t)(16 * g + h), a);
                    tmem_ld_32x8(taddr + (uint32_t)(p.kop + 16 * g + h), b);
                    tmem_ld_32x8(taddr + (uint32_t)(128 + 16 * g + h), c);
                    tmem_ld_32x8(taddr + (uint32_t)(128 + p.kop + 16 * g + h), d);
                    tmem_ld_wait();
#pragma unroll
                    for (int u = 0; u < 8; u += 4) {
                        const float4 f4 = *reinterpret_cast<const float4 *>(filter_inv + 16 * g + h + u);
                        const float4 b4 = *reinterpret_cast<const float4 *>(bias_s + 16 * g + h + u);
                        const uint64_t fs[2] = {mul2(pack2(f4.x, f4.y), is2), mul2(pack2(f4.z, f4.w), is2)}, bs[2] = {pack2(b4.x, b4.y), pack2(b4.z, b4.w)};
#pragma unroll
                        for (int q = 0; q < 4; q += 2) {
                            auto value = [&](const uint32_t (&main)[8], const uint32_t (&cross)[8], float *to) { // the products with powers of two are exact
                                const uint64_t v = add2(mul2(add2(pack2(main[u + q], main[u + q + 1]), pack2(cross[u + q], cross[u + q + 1])), fs[q / 2]), bs[q / 2]);
                                float x, y, x0, y0;
                                unpack2(v, x, y);
                                unpack2(mul2(v, 0ull), x0, y0);
                                to[0] = !relu || x > 0.0f ? x : x0;
                                to[1] = !relu || y > 0.0f ? y : y0;
                            };
                            value(a, b, even + h + u + q), value(c, d, odd + h + u + q);
                        }
                    }
                }
                const int filters = p.ko - 16 * g < 16 ? p.ko - 16 * g : 16;
                if (p.pool) {
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        // window order and strict '>' as in maxpool2d, one after the other: the maximum of the lower row by itself
                        // would lose its second element where the first is NaN
                        const float even1 = __shfl_down_sync(0xffffffffu, even[u], 1), odd1 = __shfl_down_sync(0xffffffffu, odd[u], 1);
                        even[u] = even1 > even[u] ? even1 : even[u];
                        even[u] = odd[u] > even[u] ? odd[u] : even[u];
                        even[u] = odd1 > even[u] ? odd1 : even[u];
                    }
                }
                float *at = dst;
#pragma unroll
                for (int u = 0; u < 16; ++u, at += plane) {
                    if (u < filters) {
                        if (live_even)
                            at[0] = even[u];
                        if (live_low)
                            at[p.wo] = odd[u];
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if (CG == 2)
                    mbar_arrive_peer_read(leader_addr(smem_u32(&bar_acc_empty[set])));
                else
                    mbar_arrive(smem_u32(&bar_acc_empty[set]));
                if (RAW)
                    mbar_arrive(smem_u32(&bar_scale_empty[s]));
            }
            ++i;
            if (++s == p.stages)
                s = 0, scale_phase ^= 1u;
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (CG == 2)
        cluster_sync(); // neither CTA goes while the other's MMAs, copies or arrivals may still reach it
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        if (CG == 2)
            tmem_dealloc_pair(tmem_base, 512);
        else
            tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && !failed && *abort_flag)
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

} // namespace

// Shared-memory plan of a launch: tile rows, bytes per plane and per raw box, pipeline stages.
static bool conv_tmem_plan(
    ConvTmemParams &p, int64_t h, int64_t wd, int64_t kh, int64_t kw, int64_t pad, int pool, bool raw, int row_bytes = 128) {
    p.pad = (int)pad, p.kh = (int)kh, p.kw = (int)kw;
    p.pw  = (int)(wd + 2 * pad);
    p.wo  = p.pw - (int)kw + 1;
    p.ho  = (int)(h + 2 * pad - kh + 1);
    p.th  = kTA_N / p.pw < p.ho ? kTA_N / p.pw : p.ho;
    if (pool)
        p.th &= ~1;
    if (p.th < 1)
        return false;
    p.tiles_y  = (p.ho + p.th - 1) / p.th;
    p.ksteps   = (int)(kh * kw * 4);
    p.box_rows = p.th + (int)kh - 1;
    p.box_bytes = p.box_rows * p.pw * row_bytes;
    // a tap's shifted window of kTA_N rows may run past the box: reserve those rows too
    int rows_needed = ((int)kh - 1) * p.pw + ((int)kw - 1) + kTA_N;
    if (rows_needed < p.box_rows * p.pw)
        rows_needed = p.box_rows * p.pw;
    p.plane_bytes = (rows_needed * row_bytes + 1023) & ~1023;
    // raw mode: the box starts at the 16-byte boundary at or left of x = -pad and is a whole number
    // of 16-byte units wide
    const int pad_up = ((int)pad + 3) & ~3;
    p.off_x      = pad_up - (int)pad;
    p.box_w      = (p.off_x + p.pw + 3) & ~3;
    p.raw_bytes  = 32 * p.box_rows * p.box_w * 4;
    p.raw_stride = (p.raw_bytes + 127) & ~127;
    if (raw && (p.box_w > 256 || p.box_rows > 256))
        return false;
    const int budget = 226 * 1024 - 1024 - kTA_StagingBytes - (raw ? kTA_RawStages * p.raw_stride : 0);
    // (stages, boxes and the staging block also hold the filters for a moment at the start: at least 42 KB to spare over all
    // shapes that conv_tmem_applicable accepts)
    p.stages         = budget / (2 * p.plane_bytes);
    if (p.stages > 4)
        p.stages = 4;
    return p.stages >= 2;
}

static bool conv_pair_plan(
    ConvPairParams &p, int64_t c, int64_t h, int64_t wd, int64_t ko, int64_t kh, int64_t kw, int64_t pad, bool raw, int cg, size_t *smem) {
    p.ko = (int)ko, p.kop = (int)((ko + 16 * cg - 1) / (16 * cg) * (16 * cg)), p.c = (int)c;
    p.kh = (int)kh, p.kw = (int)kw, p.pad = (int)pad;
    p.pw  = (int)(wd + 2 * pad);
    p.wo  = p.pw - (int)kw + 1;
    p.ho  = (int)(h + 2 * pad - kh + 1);
    if (p.pw > 128 || p.wo < 1 || p.ho < 1 || kh * kw < 2) // one tap would leave the leading columns empty
        return false;
    p.jp          = std::min(128 / p.pw, (p.ho + 1) / 2);
    p.tiles_y     = ((p.ho + 1) / 2 + p.jp - 1) / p.jp;
    p.box_rows    = 2 * p.jp + (int)kh - 1;
    p.region_rows = (p.box_rows + 1) / 2;
    // a tap's window of 128 rows may run past the region: reserve those rows too
    const int rows = std::max(p.region_rows * p.pw, (int)(kh / 2) * p.pw + (int)kw - 1 + 128);
    p.region_bytes = (rows * kCP_RowB + 1023) & ~1023;
    p.filter_bytes = (int)(((cg == 2 ? kh * kw * 3 + 1 : kh * kw * 4) * (p.kop / 2) * kCP_RowB + 1023) & ~1023);
    // raw mode: the box starts at the 16-byte boundary at or left of x = -pad and is a whole number of 16-byte units wide
    p.off_x      = (((int)pad + 3) & ~3) - (int)pad;
    p.box_w      = (p.off_x + p.pw + 3) & ~3;
    p.raw_bytes  = 32 * p.box_rows * p.box_w * 4;
    p.raw_stride = raw ? (p.raw_bytes + 127) & ~127 : 0;
    if (p.box_w > 256 || p.box_rows > 256)
        return false;
    p.stages = std::min(kCP_MaxStages, (kCP_Smem - 1024 - p.filter_bytes - p.raw_stride) / (4 * p.region_bytes));
    // the float32 filters lie for a moment where the stages will be
    const int filters = (int)(ko * ((c * kh * kw) | 1) * 4), planes = p.stages * 4 * p.region_bytes + p.raw_stride;
    *smem = 1024 + (size_t)p.filter_bytes + (size_t)std::max(filters, planes);
    return p.stages >= 2 && *smem <= (size_t)kCP_Smem;
}

// Whether the filters-in-tensor-memory kernel takes this layer.  The answer does not depend on
// whether a max-pool is fused, so that conv2d and conv2d + pool of one layer run the same arithmetic;
// *pool_ok says whether the fused 2x2 pool is possible (even output extents, two rows per tile).
bool conv_tmem_applicable(int64_t c, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride,
                          int64_t pad, bool *pool_ok) {
    if (pool_ok)
        *pool_ok = false;
    if (stride != 1 || c < 1 || c > 32 || ko < 1 || ko > 64 || kh * kw * 4 > kTA_MaxKSteps)
        return false;
    const int64_t pw = w + 2 * pad, wo = pw - kw + 1, ho = h + 2 * pad - kh + 1;
    if (wo < 1 || ho < 1 || pw > kTA_N || pw > 256)
        return false;
    int64_t th = kTA_N / pw;
    if (th > ho)
        th = ho;
    if (th < 1 || th + kh - 1 > 256)
        return false;
    // worth it only where the tile is reasonably full (else the pixels-on-rows kernel)
    if (!(th * pw >= 96 || th == ho))
        return false;
    if (pool_ok)
        *pool_ok = (wo & 1) == 0 && (ho & 1) == 0 && (pw & 1) == 0 && th >= 2; // horizontal neighbours in one warp
    ConvPairParams pairs;
    ConvTmemParams wide;
    size_t smem;
    return (conv_pair_plan(pairs, c, h, w, ko, kh, kw, pad, false, 2, &smem) || conv_pair_plan(pairs, c, h, w, ko, kh, kw, pad, false, 1, &smem)) &&
           conv_tmem_plan(wide, h, w, kh, kw, pad, 0, false);
}

// The form in which the layer runs: the input read as it is (NCHW float32) where a tensor map covers it, which needs row strides of
// whole 16-byte units and an aligned base, and where the raw boxes fit into shared memory beside two stages of planes; else from
// pre-split NHWC planes.  Pairs of CTAs, which read a fifth less shared memory for an MMA, where that decides: two k-steps to a tap, more
// than four taps, many tiles, and no padding of the filters to 32 unless the boxes are read twice or come as planes (8192 x 32 x
// 28 x 28 -> 64 with the pool 932 us by single CTAs, 887 by pairs, 2000 x 24 x 30 x 29 -> 32 269 and 252, 256 x 60 x 60 -> 16 128 and 125).  Elsewhere
// single CTAs, which start without a cluster and pad filters to 16 (4 x 16 x 28 x 28 -> 64 16.9 us and 18.5, 1024 x 16 x 28 x 28 -> 32 75
// and 89, 2048 x 48 129 and 165, 512 x 24 x 56 x 56 -> 16, 2 x 2, 118 and 156, 640 tiles of 32 -> 64 33.0 and 33.6).
static bool conv_pair_form(
    ConvPairParams &p, ConvTmemParams &wide, const float *x, int64_t batch, int64_t c, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw,
    int64_t pad, int pool, int64_t sms, bool *raw, int *cg, size_t *smem) {
    const bool mapped = (w & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    for (const bool as_is : {true, false}) {
        if ((as_is && !mapped) || !conv_tmem_plan(wide, h, w, kh, kw, pad, pool, as_is))
            continue;
        *raw = as_is;
        const bool padded = (ko - 1) % 32 < 16;
        if (c > 16 && kh * kw > 4 && conv_pair_plan(p, c, h, w, ko, kh, kw, pad, as_is, 2, smem) && p.tiles_y * batch >= 6 * sms &&
            !(padded && as_is && p.box_rows * p.pw <= 32 * kCP_CvtWarps)) {
            *cg = 2;
            return true;
        }
        for (*cg = 1; *cg <= 2; ++*cg)
            if (conv_pair_plan(p, c, h, w, ko, kh, kw, pad, as_is, *cg, smem))
                return true;
    }
    return false;
}

// x NCHW float32.  The layer in split float16, and behind it the tf32 form for the images that need it.  Where the
// rows allow a tensor map over it the input is read as it is, with the tiles' ranges in scratch of this call's own (such
// a layer shares no memory with calls on other streams); else from planes in the workspace:
// [filter scale][image scale][image ranges][image slots].
ct_status conv_tmem_filters(
    DeviceState *st, const float *x, const float *w, const float *bias, int64_t batch, int64_t c, int64_t h, int64_t wd,
    int64_t ko, int64_t kh, int64_t kw, int64_t pad, int act, int pool, float *out) {
    bool raw;
    int cg;
    ConvPairParams pp;
    ConvTmemParams pt; // the tf32 form
    size_t pair_smem;
    if (!conv_pair_form(pp, pt, x, batch, c, h, wd, ko, kh, kw, pad, pool, st->sm_count, &raw, &cg, &pair_smem))
        return fail(CT_ERR_INVALID, "conv2d: internal tile shape not usable");
    pp.w = pt.w = w, pp.bias = pt.bias = bias, pp.out = pt.out = out, pp.flags = pt.flags = st->flags_dev;
    pt.ko = (int)ko, pt.c = (int)c;
    pp.act = pt.act = act, pp.pool = pt.pool = pool;
    pp.image_scale = pt.image_scale = nullptr, pp.tile_range = pt.tile_range = nullptr;
    const int64_t tiles = (int64_t)pt.tiles_y * batch, pair_tiles = (int64_t)pp.tiles_y * batch;
    if (tiles > 0x7fffffffll || pair_tiles > 0x7fffffffll)
        return fail(CT_ERR_TOO_LARGE, "conv2d: too many tiles");
    pt.range_tiles = pp.tiles_y, pt.range_total = (int)pair_tiles;
    static bool attr_set_dev[16] = {}; // the attribute belongs to a device's context
    if (!attr_set_dev[st->device & 15]) {
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_filters_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_filters_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        for (auto kernel : {conv_pairs_kernel<false, 1>, conv_pairs_kernel<false, 2>, conv_pairs_kernel<true, 1>, conv_pairs_kernel<true, 2>})
            CT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCP_Smem));
        attr_set_dev[st->device & 15] = true;
    }
    const size_t smem32 = (size_t)pt.stages * 2 * pt.plane_bytes + (raw ? (size_t)kTA_RawStages * pt.raw_stride : 0) + kTA_StagingBytes + 1024;
    const unsigned grid   = (unsigned)cg * (unsigned)std::min<int64_t>((pair_tiles + cg - 1) / cg, st->sm_count / cg);
    const unsigned grid32 = (unsigned)std::max<int64_t>(std::min<int64_t>(tiles, st->sm_count), (tiles + kTA_MaxOwn - 1) / kTA_MaxOwn);
    if (raw) {
        // the input [batch][c][h][w]; box = box_w floats x box_rows rows x 32 channels of one image, not
        // swizzled; outside the image and past the last channel it reads as zero: padding for free
        CUtensorMap map, map32;
        const uint64_t dims[4]    = {(uint64_t)wd, (uint64_t)h, (uint64_t)c, (uint64_t)batch};
        const uint64_t strides[3] = {4ull * (uint64_t)wd, 4ull * (uint64_t)wd * (uint64_t)h,
                                     4ull * (uint64_t)wd * (uint64_t)h * (uint64_t)c};
        const uint32_t box[4]     = {(uint32_t)pp.box_w, (uint32_t)pp.box_rows, 32, 1};
        const uint32_t box32[4]   = {(uint32_t)pt.box_w, (uint32_t)pt.box_rows, 32, 1};
        CT_TRY(encode_tiled_map_f32(&map, x, 4, dims, strides, box, /*swizzle_bytes=*/0));
        CT_TRY(encode_tiled_map_f32(&map32, x, 4, dims, strides, box32, /*swizzle_bytes=*/0));
        void *ranges = nullptr;
        CT_TRY(ct_alloc(&ranges, (size_t)(pair_tiles + 1) * sizeof(uint2)));
        pp.tile_range = pt.tile_range = static_cast<uint2 *>(ranges);
        cudaError_t launched;
        {
            ProfScope prof("gemm_tc");
            (void)launch_dependent_cluster(cg == 2 ? conv_pairs_kernel<true, 2> : conv_pairs_kernel<true, 1>, cg, dim3(grid), dim3(kCP_Threads), pair_smem, stream(), map, map, pp, (int)pair_tiles);
            (void)launch_dependent(conv_tmem_filters_kernel<true>, dim3(grid32), dim3(kTA_ThreadsRaw), smem32, stream(), map32, map32, pt, (int)tiles);
            launched = cudaGetLastError();
        }
        CT_TRY(ct_free(ranges)); // in stream order, behind both
        if (launched != cudaSuccess)
            return cuda_fail(launched, "conv_tmem");
        count_launch(2);
        return CT_OK;
    }
    auto align_up       = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    const int64_t hs     = (h + 1) / 2; // rows of a sub-image: even and odd rows lie apart (float16 only)
    const size_t f_words = align_up((size_t)ko * 4), words = align_up((size_t)batch * 4), slot = (size_t)hs * 2 * wd * 32 * 8;
    const size_t ranges  = align_up((size_t)batch * conv_range_slices(batch, c * h * wd) * 8);
    CT_TRY(ensure_ws(&st->gemm_ws, &st->gemm_ws_bytes, f_words + words + ranges + (size_t)batch * slot));
    uint8_t *ws = static_cast<uint8_t *>(st->gemm_ws), *planes = ws + f_words + words + ranges;
    float *image_scale = reinterpret_cast<float *>(ws + f_words);
    CT_TRY(conv_prepass(x, w, batch, c, h, wd, 32, ko, kh * kw, nullptr, nullptr, 0, 0, nullptr, reinterpret_cast<float *>(ws), nullptr, nullptr,
                        ws + f_words + words, image_scale, planes, ConvSubImages{2, 1, 3u, true, (int)hs, (int)wd}));
    pp.image_scale = pt.image_scale = image_scale;
    // float16 planes [batch][row & 1][row >> 1][w][32 channels], box = 32 channels x pw positions x region_rows rows of one
    // sub-image; tf32 planes [batch][h][w][32 channels]; swizzled over a row; outside the image they read as zero: the padding
    auto encode16 = [&](CUtensorMap *map, const void *base) {
        const uint64_t dims[5] = {32, (uint64_t)wd, (uint64_t)hs, 2, (uint64_t)batch};
        const uint64_t strides[4] = {64, 64ull * (uint64_t)wd, 64ull * (uint64_t)(wd * hs), slot};
        const uint32_t box[5] = {32, (uint32_t)pp.pw, (uint32_t)pp.region_rows, 1, 1};
        return encode_tiled_map_f16(map, base, 5, dims, strides, box, kCP_RowB);
    };
    auto encode32 = [&](CUtensorMap *map, const void *base) {
        const uint64_t dims[4] = {32, (uint64_t)wd, (uint64_t)h, (uint64_t)batch};
        const uint64_t strides[3] = {128, 128ull * (uint64_t)wd, slot};
        const uint32_t box[4] = {32, (uint32_t)pt.pw, (uint32_t)pt.box_rows, 1};
        return encode_tiled_map_f32(map, base, 4, dims, strides, box, 128);
    };
    CUtensorMap m16_hi, m16_lo, m32_hi, m32_lo;
    CT_TRY(encode16(&m16_hi, planes));
    CT_TRY(encode16(&m16_lo, planes + slot / 4));
    CT_TRY(encode32(&m32_hi, planes));
    CT_TRY(encode32(&m32_lo, planes + slot / 2));
    ProfScope prof("gemm_tc");
    (void)launch_dependent_cluster(cg == 2 ? conv_pairs_kernel<false, 2> : conv_pairs_kernel<false, 1>, cg, dim3(grid), dim3(kCP_Threads), pair_smem, stream(), m16_hi, m16_lo, pp, (int)pair_tiles);
    CT_LAUNCH_CHECK("conv_pairs");
    (void)launch_dependent(conv_tmem_filters_kernel<false>, dim3(grid32), dim3(kTA_Threads), smem32, stream(), m32_hi, m32_lo, pt, (int)tiles);
    CT_LAUNCH_CHECK("conv_tmem_filters");
    return CT_OK;
}

} // namespace ct
