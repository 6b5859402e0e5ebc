// conv2d for layers with few channels on both sides (at most 32 in, at most 64 out, a small
// filter; the 32 -> 64 channel 3x3 layer of a small CNN): the filters live in tensor memory.
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
    uint2 *tile_range;        // raw: [total tiles] range of the values of each tile, and one entry whose .x says that
                              // the filters need tf32 terms
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
template <bool RAW> __device__ __forceinline__ bool image_needs_tf32(const ConvTmemParams &p, int img, int total_tiles) {
    if (!RAW)
        return __ldg(p.image_scale + img) == 0.0f;
    const uint32_t filters = p.tile_range[total_tiles].x;
    const uint2 *src       = p.tile_range + (int64_t)img * p.tiles_y;
    uint2 range            = make_uint2(0u, kNoneSmallest);
    for (int t = 0; t < p.tiles_y; t += 8) {
        uint2 r[8]; // eight loads in flight: one after the other they cost an idle launch 4 us
#pragma unroll
        for (int j = 0; j < 8; ++j)
            r[j] = src[min(t + j, p.tiles_y - 1)];
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
__device__ __forceinline__ int filter_stride(const ConvTmemParams &p) { return (p.c * p.kh * p.kw) | 1; }
template <typename Seen>
__device__ __forceinline__ void stage_filters(const ConvTmemParams &p, float *rows, int warp, int warps, int lane, Seen seen) {
    const int row = p.c * p.kh * p.kw, stride = filter_stride(p);
    for (int f = warp; f < p.ko; f += warps) {
        uint2 range = make_uint2(0u, kNoneSmallest);
#pragma unroll 4
        for (int e = lane; e < row; e += 32) {
            const float v = p.w[(int64_t)f * row + e];
            range_take(range, v);
            rows[f * stride + e] = v;
        }
        seen(f, range);
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
        const bool mine     = q < own && image_needs_tf32<RAW>(p, ((int)blockIdx.x + q * (int)gridDim.x) / p.tiles_y, total_tiles);
        const uint32_t bits = __ballot_sync(0xffffffffu, mine);
        any |= bits != 0u;
        if (lane == 0)
            own_mask[q0 >> 5] = bits;
    }
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
    if (!__syncthreads_or(any) || abort_flag_s)
        return; // conv_tmem_half_kernel has computed them all

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
    stage_filters(p, filters, warp, (int)blockDim.x / 32, lane, [](int, uint2) {});
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
        const float *src  = filters + ch * filter_stride(p);
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
        if (lane == 0) {
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
        if (lane == 0) {
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

// ---- the same in split float16 ------------------------------------------------------------
//
// Two 11-bit terms in float16 instead of tf32 (half_split.cuh): 16 channels per MMA instead of 8, so half the
// MMAs, half the filter columns in tensor memory and half the plane bytes.  The filters are scaled per
// filter, the pixels per tile (the converting warps see the whole box before they split it) or, from planes,
// per image.  The low terms are stored 2^11 times larger, so hi and lo products have accumulators of their own:
//     D1 = [W_hi; W_lo] x X_hi,  D2 = [W_hi; W_lo] x X_lo   (128 x 128 each, next to at most 192 filter columns)
// and a thread that drains row m forms D1 + 2^-11 D2 before anything is parked, which leaves the rest of the
// epilogue as it is above (hi row + lo row).  Eight warps convert (four needed 4250 clocks per tile where the
// MMAs now take 2628) and what sets the pace is the epilogue.  The converting warps also leave the range of every
// tile in the call's own scratch; conv_tmem_filters_kernel, launched behind this one, computes the images that
// float16 pairs cannot hold.  A tile that shows that by itself is not converted, multiplied or stored here.
constexpr int kTH_CvtWarps = 8;
constexpr int kTH_Threads  = 64 + 32 * kTH_CvtWarps + 32 * kTA_EpiWarps;
constexpr int kTH_D1 = 192, kTH_D2 = 320; // accumulator columns behind 24 k-steps of 8 filter columns
constexpr int kTH_RowB = 64;              // a position's 32 channels

__device__ __forceinline__ void mma_f16_a_tmem(
    uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <bool RAW>
__global__ void __launch_bounds__(kTH_Threads, 1) conv_tmem_half_kernel(
    const __grid_constant__ CUtensorMap map_x_hi, const __grid_constant__ CUtensorMap map_x_lo,
    const __grid_constant__ ConvTmemParams p, const int total_tiles) {
    constexpr int kMaxStages = 4;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[kMaxStages], bar_empty[kMaxStages];
    __shared__ uint64_t bar_raw_full[kTA_RawStages], bar_raw_empty[kTA_RawStages];
    __shared__ uint64_t bar_scale_empty[kMaxStages]; // the tile's scale has been read by the epilogue
    __shared__ uint64_t bar_tmem_full, bar_tmem_empty, bar_done, bar_epi, bar_cvt;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s, filters_wide_s;
    __shared__ uint2 cvt_range[2][kTH_CvtWarps];
    __shared__ float tile_scale[kMaxStages]; // inverse scale of the tile in each plane stage; 0: left to the tf32 form
    __shared__ float filter_inv[64];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag_s   = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
        filters_wide_s = 0;
    }
    if (threadIdx.x < 64)
        filter_inv[threadIdx.x] = 1.0f; // rows without a filter are zero
    __syncthreads();
    if (abort_flag_s)
        return;

    const uint32_t smem_base   = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = 2u * (uint32_t)p.plane_bytes;
    const uint32_t raw_base    = smem_base + (uint32_t)p.stages * stage_bytes;
    const uint32_t raw_all     = RAW ? (uint32_t)kTA_RawStages * (uint32_t)p.raw_stride : 0u;
    float *staging = reinterpret_cast<float *>(smem_raw + (raw_base - smem_u32(smem_raw)) + raw_all);

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), RAW ? kTH_CvtWarps : 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
            mbar_init(smem_u32(&bar_scale_empty[s]), kTA_EpiWarps);
        }
        for (int s = 0; s < kTA_RawStages; ++s) {
            mbar_init(smem_u32(&bar_raw_full[s]), 1);
            mbar_init(smem_u32(&bar_raw_empty[s]), kTH_CvtWarps);
        }
        mbar_init(smem_u32(&bar_tmem_full), 1);
        mbar_init(smem_u32(&bar_tmem_empty), kTA_EpiWarps);
        mbar_init(smem_u32(&bar_done), 1);
        mbar_init(smem_u32(&bar_epi), kTA_EpiWarps);
        mbar_init(smem_u32(&bar_cvt), kTH_CvtWarps);
        mbar_fence_init();
        prefetch_tensormap(&map_x_hi);
        prefetch_tensormap(&map_x_lo);
    }
    float *filters = reinterpret_cast<float *>(smem_raw + (smem_base - smem_u32(smem_raw))); // where the stages will be
    stage_filters(p, filters, warp, kTH_Threads / 32, lane, [&](int f, uint2 range) {
        float scale, inverse;
        const bool fits = half_range_fits(range_warp(range), scale, inverse);
        if (lane == 0) {
            filter_inv[f] = inverse;
            if (!fits)
                filters_wide_s = 1;
        }
    });
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    const bool filters_wide  = filters_wide_s != 0; // every tile is left to the tf32 form
    if (RAW && blockIdx.x == 0 && threadIdx.x == 0)
        p.tile_range[total_tiles] = make_uint2(filters_wide ? 1u : 0u, 0u);

    // ---- the filters go to tensor memory, once: warps 2..5 own the four lane quarters ----------
    if (warp >= 2 && warp < 6 && !filters_wide) {
        const int quarter = warp & 3;
        const int m = quarter * 32 + lane, ch = m & 63; // TMEM lane = row of the A operand; filter
        const bool lo_row = m >= 64;
        const int taps    = p.kh * p.kw;
        const float *src  = filters + ch * filter_stride(p);
        const float scale = 1.0f / filter_inv[ch]; // both are powers of two
#pragma unroll 2
        for (int ks = 0; ks < 2 * taps; ++ks) {
            const int tap = ks >> 1, c0 = (ks & 1) * 16;
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int ic  = c0 + 2 * j;
                const float a = (ch < p.ko && ic < p.c) ? src[ic * taps + tap] : 0.0f;
                const float b = (ch < p.ko && ic + 1 < p.c) ? src[(ic + 1) * taps + tap] : 0.0f;
                __half2 hi, lo;
                split_half_pair(a * scale, b * scale, hi, lo);
                v[j] = lo_row ? *reinterpret_cast<uint32_t *>(&lo) : *reinterpret_cast<uint32_t *>(&hi);
            }
            tmem_st_32x32_x8(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ks * 8), v);
        }
        tmem_st_wait();
        filters_taken();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    if (filters_wide) {
    } else if (warp == 0) {
        // ===== TMA producer: one halo box per plane and tile (raw mode: one box of the input) =====
        if (lane == 0) {
            int i = 0;
            const int nstages = RAW ? kTA_RawStages : p.stages;
            for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
                const int img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
                if (!RAW && image_needs_tf32<RAW>(p, img, total_tiles))
                    continue;
                const int s       = i % nstages;
                const uint32_t ph = (uint32_t)(i / nstages) & 1u;
                if (!mbar_wait_patient(smem_u32(RAW ? &bar_raw_empty[s] : &bar_empty[s]), ph ^ 1u, abort_flag))
                    break;
                const int32_t h0 = ty * p.th - p.pad;
                if (RAW) {
                    const uint32_t full = smem_u32(&bar_raw_full[s]);
                    mbar_expect_tx(full, (uint32_t)p.raw_bytes);
                    // the box starts off_x floats left of x = -pad so that its first byte is 16-byte aligned
                    tma_load_4d(raw_base + (uint32_t)s * (uint32_t)p.raw_stride, &map_x_hi, full, -p.pad - p.off_x, h0, 0, img);
                } else {
                    const uint32_t full = smem_u32(&bar_full[s]), dst = smem_base + (uint32_t)s * stage_bytes;
                    mbar_expect_tx(full, 2u * (uint32_t)p.box_bytes);
                    tma_load_4d(dst, &map_x_hi, full, 0, -p.pad, h0, img);
                    tma_load_4d(dst + (uint32_t)p.plane_bytes, &map_x_lo, full, 0, -p.pad, h0, img);
                }
                ++i;
            }
            if (*abort_flag) {
                // unwind: let the copies still in flight land before the CTA goes away
                for (int k2 = i - nstages < 0 ? 0 : i - nstages; k2 < i; ++k2) {
                    const uint32_t bar = smem_u32(RAW ? &bar_raw_full[k2 % nstages] : &bar_full[k2 % nstages]);
                    const uint64_t t0  = globaltimer_ns();
                    while (!mbar_try_wait(bar, (uint32_t)(k2 / nstages) & 1u) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        if (lane == 0) {
            const uint32_t idesc = make_idesc(0u, 128, (uint32_t)kTA_N);
            const uint32_t d1 = tmem_base + (uint32_t)kTH_D1, d2 = tmem_base + (uint32_t)kTH_D2;
            int i   = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
                if (!RAW && image_needs_tf32<RAW>(p, tile / p.tiles_y, total_tiles))
                    continue;
                const int s = i % p.stages;
                // the accumulators of the previous tile have been read, the planes are complete
                ok = mbar_wait(smem_u32(&bar_tmem_empty), ((uint32_t)i & 1u) ^ 1u, abort_flag) &&
                     mbar_wait(smem_u32(&bar_full[s]), (uint32_t)(i / p.stages) & 1u, abort_flag);
                if (!ok)
                    break;
                tc_fence_after_sync();
                const uint32_t x_hi = smem_base + (uint32_t)s * stage_bytes, x_lo = x_hi + (uint32_t)p.plane_bytes;
                int ks = 0;
                const int rows = RAW && *const_cast<volatile float *>(&tile_scale[s]) == 0.0f ? 0 : p.kh;
                for (int r = 0; r < rows; ++r) {
                    for (int sx = 0; sx < p.kw; ++sx) {
                        // the tap's pixels: the same box, (r * pw + sx) rows further on
                        const uint32_t shift = (uint32_t)(r * p.pw + sx) * (uint32_t)kTH_RowB;
                        const uint64_t db_hi = smem_desc_k<kTH_RowB>(x_hi + shift), db_lo = smem_desc_k<kTH_RowB>(x_lo + shift);
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk, ++ks) {
                            const uint32_t a_tmem = tmem_base + (uint32_t)(ks * 8);
                            mma_f16_a_tmem(d1, a_tmem, db_hi + 2 * kk, idesc, ks == 0 ? 0u : 1u);
                            mma_f16_a_tmem(d2, a_tmem, db_lo + 2 * kk, idesc, ks == 0 ? 0u : 1u);
                        }
                    }
                }
                tc_commit(smem_u32(&bar_empty[s]));  // the stage is free once these MMAs have retired
                tc_commit(smem_u32(&bar_tmem_full)); // and the accumulators are complete
                ++i;
            }
            if (!ok || *abort_flag) {
                tc_commit(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else if (warp < 2 + kTH_CvtWarps) {
        // ===== raw mode: float32 box -> float16 planes (warps before the epilogue's: see above) =====
        if (RAW) {
            const int ct      = threadIdx.x - 64;
            const int npos    = p.box_rows * p.pw;
            const int cstride = p.box_rows * p.box_w; // floats between two channels of one position
            int i = 0;
            for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++i) {
                const int rs = i % kTA_RawStages, s = i % p.stages;
                bool got = mbar_wait_patient(smem_u32(&bar_raw_full[rs]), (uint32_t)(i / kTA_RawStages) & 1u, abort_flag);
                if (!__all_sync(0xffffffffu, got))
                    break;
                const float *raw = reinterpret_cast<const float *>(smem_raw + (raw_base - smem_u32(smem_raw)) + (uint32_t)rs * (uint32_t)p.raw_stride);
                // the tile's range (the whole box, alignment columns included: they are pixels or zero)
                uint2 range       = make_uint2(0u, kNoneSmallest);
                const float4 *r4  = reinterpret_cast<const float4 *>(raw);
#pragma unroll 4
                for (int e = ct; e < p.raw_bytes / 16; e += 32 * kTH_CvtWarps) {
                    const float4 q = r4[e];
                    range_take(range, q.x), range_take(range, q.y), range_take(range, q.z), range_take(range, q.w);
                }
                range = range_warp(range);
                if (lane == 0) {
                    cvt_range[i & 1][warp - 2] = range;
                    mbar_arrive(smem_u32(&bar_cvt));
                }
                got = mbar_wait(smem_u32(&bar_cvt), (uint32_t)i & 1u, abort_flag) && // all eight ranges
                      mbar_wait_patient(smem_u32(&bar_empty[s]), ((uint32_t)(i / p.stages) & 1u) ^ 1u, abort_flag) &&
                      mbar_wait_patient(smem_u32(&bar_scale_empty[s]), ((uint32_t)(i / p.stages) & 1u) ^ 1u, abort_flag);
                if (!__all_sync(0xffffffffu, got))
                    break;
#pragma unroll
                for (int u = 0; u < kTH_CvtWarps; ++u)
                    range = range_join(range, cvt_range[i & 1][u]);
                float scale, inverse;
                const bool fits = half_range_fits(range, scale, inverse);
                if (ct == 0) {
                    tile_scale[s]      = fits ? inverse : 0.0f;
                    p.tile_range[tile] = range;
                }
                uint8_t *x_hi = smem_raw + (smem_base - smem_u32(smem_raw)) + (uint32_t)s * stage_bytes;
                uint8_t *x_lo = x_hi + p.plane_bytes;
                // a thread takes a position: 32 channels become the 64-byte row y * pw + x of both planes, 16-byte
                // chunk j at j ^ ((row >> 1) & 3), the 64-byte swizzle
                for (int pos = fits ? ct : npos; pos < npos; pos += 32 * kTH_CvtWarps) {
                    const int y = pos / p.pw, x = pos - y * p.pw;
                    const float *src = raw + y * p.box_w + x + p.off_x;
                    const uint32_t row_off = (uint32_t)pos * (uint32_t)kTH_RowB, sw = ((uint32_t)pos >> 1) & 3u;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        float v[16];
#pragma unroll
                        for (int t = 0; t < 16; ++t)
                            v[t] = src[(16 * half + t) * cstride];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            __half2 hi[4], lo[4];
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                split_half_pair(__fmul_rn(v[8 * j + 2 * t], scale), __fmul_rn(v[8 * j + 2 * t + 1], scale), hi[t], lo[t]);
                            }
                            const uint32_t at = row_off + (((uint32_t)(2 * half + j) ^ sw) << 4);
                            *reinterpret_cast<uint4 *>(x_hi + at) = *reinterpret_cast<uint4 *>(hi);
                            *reinterpret_cast<uint4 *>(x_lo + at) = *reinterpret_cast<uint4 *>(lo);
                        }
                    }
                }
                // written through the generic proxy, read by the tensor core's asynchronous proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(smem_u32(&bar_full[s]));
                    mbar_arrive(smem_u32(&bar_raw_empty[rs]));
                }
            }
        }
    } else {
        // ===== epilogue =====
        const int quarter = warp & 3;                // TMEM lanes this warp may read
        const int ew      = warp - 2 - kTH_CvtWarps; // 0..7: which channels this warp writes out
        const int half    = ew >> 2;                 // which 64 columns of the accumulators it drains
        uint32_t epi_phase = 0;
        auto epi_sync = [&]() -> bool {
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&bar_epi));
            bool ok = mbar_wait_patient(smem_u32(&bar_epi), epi_phase, abort_flag);
            epi_phase ^= 1u;
            return __all_sync(0xffffffffu, ok);
        };
        // where this lane's positions land, once for the whole kernel (see conv_tmem_filters_kernel)
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
        float bias_r[64 / kTA_EpiWarps];
#pragma unroll
        for (int j = 0; j < 64 / kTA_EpiWarps; ++j) {
            const int ch = ew + kTA_EpiWarps * j;
            bias_r[j]    = (p.bias && ch < p.ko) ? p.bias[ch] : 0.0f;
        }
        const int m       = quarter * 32 + lane;
        const float row_f = m < 64 ? filter_inv[m] : filter_inv[m - 64] * kHalfLoInv;
        int i = 0;
        for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++i) {
            const int img = tile / p.tiles_y, ty = tile - img * p.tiles_y;
            if (!RAW && image_needs_tf32<RAW>(p, img, total_tiles)) {
                --i;
                continue;
            }
            bool got = mbar_wait_patient(smem_u32(&bar_tmem_full), (uint32_t)i & 1u, abort_flag);
            if (!__all_sync(0xffffffffu, got))
                break;
            const float is = RAW ? *const_cast<volatile float *>(&tile_scale[i % p.stages]) : p.image_scale[img];
            const int y0   = ty * p.th;
            tc_fence_after_sync();
            if (RAW && is == 0.0f) {
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(smem_u32(&bar_tmem_empty));
                    mbar_arrive(smem_u32(&bar_scale_empty[i % p.stages]));
                }
                continue;
            }
            float4 *mine         = reinterpret_cast<float4 *>(staging + m * kTA_StageRowF + half * 64);
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 64);
            // D1 + 2^-11 D2, sixteen columns of each at a time; the accumulators are handed back before anything
            // is parked
            float t[64];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t a[16], b[16];
                tmem_ld_32x16(taddr + kTH_D1 + 16 * g, a);
                tmem_ld_32x16(taddr + kTH_D2 + 16 * g, b);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    t[16 * g + j] = __fadd_rn(__uint_as_float(a[j]), __fmul_rn(__uint_as_float(b[j]), kHalfLoInv));
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&bar_tmem_empty)); // the next tile's MMAs may start
                mbar_arrive(smem_u32(&bar_scale_empty[i % p.stages]));
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
                mine[j] = make_float4(__fmul_rn(t[4 * j], row_f), __fmul_rn(t[4 * j + 1], row_f),
                                      __fmul_rn(t[4 * j + 2], row_f), __fmul_rn(t[4 * j + 3], row_f));
            if (!epi_sync())
                break;
            unsigned okmask = 0;
#pragma unroll
            for (int g = 0; g < 4; ++g)
                if (off[g] >= 0 && (p.pool ? (y0 >> 1) + yy[g] < ph2 : y0 + yy[g] < p.ho))
                    okmask |= 1u << g;
            // two channels at a time, every load of the pair before the first dependent instruction, masked stores
            if (p.pool == 0) {
#pragma unroll
                for (int jj = 0; jj < 64 / kTA_EpiWarps; jj += 2) {
                    float h[2][4], l[2][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float *hi = staging + (ew + kTA_EpiWarps * (jj + u)) * kTA_StageRowF + lane, *lo = hi + 64 * kTA_StageRowF;
#pragma unroll
                        for (int g = 0; g < 4; ++g)
                            h[u][g] = hi[32 * g], l[u][g] = lo[32 * g];
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int ch = ew + kTA_EpiWarps * (jj + u);
                        float *plane = p.out + (((int64_t)img * p.ko + ch) * p.ho + y0) * p.wo;
                        const unsigned mask = ch < p.ko ? okmask : 0u;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            float v = __fmul_rn(__fadd_rn(h[u][g], l[u][g]), is);
                            if (p.bias)
                                v = __fadd_rn(v, bias_r[jj + u]);
                            if (p.act == CT_ACT_RELU)
                                v = __fmul_rn(v, v > 0.0f ? 1.0f : 0.0f);
                            if (mask & (1u << g))
                                plane[off[g]] = v;
                        }
                    }
                }
            } else {
                // 2x2 max-pool of the activated values; window order and strict '>' as in maxpool2d.  Four channels
                // at a time with all their loads first, a window row as one 8-byte read where rows are even: with
                // scalar reads for two channels this phase took 3500 clocks per tile, the longest of all.
                const int groups = ((p.th >> 1) * pw2 + 31) >> 5;
                const bool even  = (p.pw & 1) == 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (g >= groups)
                        break;
                    const bool live = (okmask >> g) & 1u;
                    const int pos   = live ? off[g] : 0;
#pragma unroll
                    for (int jj = 0; jj < 64 / kTA_EpiWarps; jj += 4) {
                        float2 h[4][2], l[4][2];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float *hi = staging + (ew + kTA_EpiWarps * (jj + u)) * kTA_StageRowF + pos, *lo = hi + 64 * kTA_StageRowF;
                            if (even) {
                                h[u][0] = *reinterpret_cast<const float2 *>(hi), h[u][1] = *reinterpret_cast<const float2 *>(hi + p.pw);
                                l[u][0] = *reinterpret_cast<const float2 *>(lo), l[u][1] = *reinterpret_cast<const float2 *>(lo + p.pw);
                            } else {
                                h[u][0] = make_float2(hi[0], hi[1]), h[u][1] = make_float2(hi[p.pw], hi[p.pw + 1]);
                                l[u][0] = make_float2(lo[0], lo[1]), l[u][1] = make_float2(lo[p.pw], lo[p.pw + 1]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int ch = ew + kTA_EpiWarps * (jj + u);
                            const float hv[4] = {h[u][0].x, h[u][0].y, h[u][1].x, h[u][1].y};
                            const float lv[4] = {l[u][0].x, l[u][0].y, l[u][1].x, l[u][1].y};
                            float v[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                v[q] = __fmul_rn(__fadd_rn(hv[q], lv[q]), is);
                                if (p.bias)
                                    v[q] = __fadd_rn(v[q], bias_r[jj + u]);
                                if (p.act == CT_ACT_RELU)
                                    v[q] = __fmul_rn(v[q], v[q] > 0.0f ? 1.0f : 0.0f);
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
                                plane[lane + 32 * g] = best; // pooled pixels of a tile are consecutive
                            }
                        }
                    }
                }
            }
            if (!epi_sync()) // the staging block is rewritten by the next tile
                break;
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

} // namespace

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
        *pool_ok = (wo & 1) == 0 && (ho & 1) == 0 && th >= 2;
    return true;
}

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

// Whether the kernel can read this input as it is (NCHW float32) instead of pre-split NHWC planes:
// the tensor map over it needs row strides of whole 16-byte units and an aligned base, and the raw
// boxes have to fit into shared memory beside two stages of planes.
static bool conv_tmem_reads_input_directly(const float *x, int64_t h, int64_t w, int64_t kh, int64_t kw, int64_t pad, int pool) {
    if ((w & 3) != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) != 0)
        return false;
    ConvTmemParams p;
    return conv_tmem_plan(p, h, w, kh, kw, pad, pool, true);
}

// x NCHW float32.  The layer in split float16, and behind it the tf32 form for the images that need it.  Where the
// rows allow a tensor map over it the input is read as it is, with the tiles' ranges in scratch of this call's own (such
// a layer shares no memory with calls on other streams); else from planes in the workspace:
// [filter scale][image scale][image ranges][image slots].
ct_status conv_tmem_filters(
    DeviceState *st, const float *x, const float *w, const float *bias, int64_t batch, int64_t c, int64_t h, int64_t wd,
    int64_t ko, int64_t kh, int64_t kw, int64_t pad, int act, int pool, float *out) {
    const bool raw = conv_tmem_reads_input_directly(x, h, wd, kh, kw, pad, pool);
    ConvTmemParams p[2]; // float16, tf32
    for (int f = 0; f < 2; ++f) {
        p[f].w = w, p[f].bias = bias, p[f].out = out, p[f].flags = st->flags_dev;
        p[f].ko = (int)ko, p[f].c = (int)c;
        p[f].act = act, p[f].pool = pool;
        p[f].image_scale = nullptr, p[f].tile_range = nullptr;
        if (!conv_tmem_plan(p[f], h, wd, kh, kw, pad, pool, raw, f == 0 ? kTH_RowB : 128))
            return fail(CT_ERR_INVALID, "conv2d: internal tile shape %d x %d not usable", p[f].th, p[f].pw);
    }
    const int64_t tiles = (int64_t)p[0].tiles_y * batch;
    if (tiles > 0x7fffffffll)
        return fail(CT_ERR_TOO_LARGE, "conv2d: too many tiles");
    static bool attr_set_dev[16] = {}; // the attribute belongs to a device's context
    if (!attr_set_dev[st->device & 15]) {
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_filters_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_filters_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_half_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        CT_CUDA(cudaFuncSetAttribute(conv_tmem_half_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        attr_set_dev[st->device & 15] = true;
    }
    auto smem_of = [&](const ConvTmemParams &q) {
        return (size_t)q.stages * 2 * q.plane_bytes + (raw ? (size_t)kTA_RawStages * q.raw_stride : 0) + kTA_StagingBytes + 1024;
    };
    const unsigned grid   = (unsigned)(tiles < st->sm_count ? tiles : st->sm_count);
    const unsigned grid32 = (unsigned)std::max<int64_t>(grid, (tiles + kTA_MaxOwn - 1) / kTA_MaxOwn);
    if (raw) {
        // the input [batch][c][h][w]; box = box_w floats x box_rows rows x 32 channels of one image, not
        // swizzled; outside the image and past the last channel it reads as zero: padding for free
        CUtensorMap map;
        const uint64_t dims[4]    = {(uint64_t)wd, (uint64_t)h, (uint64_t)c, (uint64_t)batch};
        const uint64_t strides[3] = {4ull * (uint64_t)wd, 4ull * (uint64_t)wd * (uint64_t)h,
                                     4ull * (uint64_t)wd * (uint64_t)h * (uint64_t)c};
        const uint32_t box[4]     = {(uint32_t)p[0].box_w, (uint32_t)p[0].box_rows, 32, 1};
        CT_TRY(encode_tiled_map_f32(&map, x, 4, dims, strides, box, /*swizzle_bytes=*/0));
        void *ranges = nullptr;
        CT_TRY(ct_alloc(&ranges, (size_t)(tiles + 1) * sizeof(uint2)));
        p[0].tile_range = p[1].tile_range = static_cast<uint2 *>(ranges);
        cudaError_t launched;
        {
            ProfScope prof("gemm_tc");
            conv_tmem_half_kernel<true><<<grid, kTH_Threads, smem_of(p[0]), stream()>>>(map, map, p[0], (int)tiles);
            conv_tmem_filters_kernel<true><<<grid32, kTA_ThreadsRaw, smem_of(p[1]), stream()>>>(map, map, p[1], (int)tiles);
            launched = cudaGetLastError();
        }
        CT_TRY(ct_free(ranges)); // in stream order, behind both
        if (launched != cudaSuccess)
            return cuda_fail(launched, "conv_tmem");
        count_launch(2);
        return CT_OK;
    }
    auto align_up       = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    const size_t f_words = align_up((size_t)ko * 4), words = align_up((size_t)batch * 4), slot = (size_t)h * wd * 32 * 8;
    const size_t ranges  = align_up((size_t)batch * conv_range_slices(batch, c * h * wd) * 8);
    CT_TRY(ensure_ws(&st->gemm_ws, &st->gemm_ws_bytes, f_words + words + ranges + (size_t)batch * slot));
    uint8_t *ws = static_cast<uint8_t *>(st->gemm_ws), *planes = ws + f_words + words + ranges;
    float *image_scale = reinterpret_cast<float *>(ws + f_words);
    CT_TRY(conv_prepass(st, x, w, batch, c, h, wd, 32, ko, kh * kw, nullptr, nullptr, 0, 0, reinterpret_cast<float *>(ws),
                        ws + f_words + words, image_scale, planes, ConvSubImages{}));
    p[0].image_scale = p[1].image_scale = image_scale;
    // planes [batch][h][w][32 channels]; box = 32 channels x pw positions x (th + kh - 1) rows of one image,
    // swizzled over a row; positions outside the image read as zero: the padding
    auto encode = [&](CUtensorMap *map, const void *base, int elem) {
        const uint64_t row = 32ull * (uint64_t)elem;
        const uint64_t dims[4] = {32, (uint64_t)wd, (uint64_t)h, (uint64_t)batch};
        const uint64_t strides[3] = {row, row * (uint64_t)wd, slot};
        const uint32_t box[4] = {32, (uint32_t)p[0].pw, (uint32_t)p[0].box_rows, 1};
        return elem == 4 ? encode_tiled_map_f32(map, base, 4, dims, strides, box, 128)
                         : encode_tiled_map_f16(map, base, 4, dims, strides, box, kTH_RowB);
    };
    CUtensorMap m16_hi, m16_lo, m32_hi, m32_lo;
    CT_TRY(encode(&m16_hi, planes, 2));
    CT_TRY(encode(&m16_lo, planes + slot / 4, 2));
    CT_TRY(encode(&m32_hi, planes, 4));
    CT_TRY(encode(&m32_lo, planes + slot / 2, 4));
    ProfScope prof("gemm_tc");
    conv_tmem_half_kernel<false><<<grid, kTH_Threads, smem_of(p[0]), stream()>>>(m16_hi, m16_lo, p[0], (int)tiles);
    CT_LAUNCH_CHECK("conv_tmem_half");
    conv_tmem_filters_kernel<false><<<grid32, kTA_Threads, smem_of(p[1]), stream()>>>(m32_hi, m32_lo, p[1], (int)tiles);
    CT_LAUNCH_CHECK("conv_tmem_filters");
    return CT_OK;
}

} // namespace ct
