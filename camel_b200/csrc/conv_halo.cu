// Implicit-GEMM conv2d (stride 1 to 3): the input halo of a tile is fetched once per channel block and serves all
// filter taps.
//
// The streaming implicit GEMM of gemm_tc.cu fetches, for every (tap, channel block), the tile's
// pixels again - the same values shifted by the tap.  Shared memory then carries, per k-block of 16
// channels, 28 KB of pixel planes and 16 KB of filter planes in (TMA) plus 66 KB out (six MMAs read
// their operands), and that traffic, not the tensor pipe, sets the kernel's pace (0.65 of the
// measured 3xTF32 ceiling on 64 -> 128 channels, 56 x 56).  Here a tile is th output rows of
// PW = w + 2 pad positions (the two halo columns of every row are computed and dropped), its
// input for one block of 16 channels - th + kh - 1 rows of PW positions, zeros outside the image -
// is ONE 4-D TMA box per plane, and tap (r, s) reads the same shared memory through a descriptor
// moved by r * PW + s rows of 64 bytes (a position's row in the box is y * PW + x).  Pixel planes
// enter shared memory once per nine taps; per k-block 19 KB in instead of 44.
//
// Arithmetic: split float16 (half_split.cuh), scaled per filter and per image - a scale has to be constant
// along k, and an output's patch crosses the whole halo - with the cross products in an accumulator of their
// own, as in gemm_half.cu.  A 64-byte row then holds 32 channels, so the layer takes half the MMAs, half the
// filter stages and half the plane traffic of the tf32 form.  An image that spans too many powers of two - or
// every image, where a filter does - has tf32 planes in the same place, and this kernel runs the same loop over
// those for its tiles (16 channels per row); the other images of the batch are not touched by it.
//
// Strides: the rows and columns of the input that are alike modulo the stride are sub-images of the planes, and a tap is a
// shift inside one of them, so a strided layer is the same loop with a halo per sub-image; its patches are never written
// (64 x 48 x 57 x 57 -> 96 at stride 2: 121 us through a patch matrix, 70 so).  Longer k than 1024: the leading
// accumulator is drained every 1024 values, as in gemm_half.cu.  Additions into an accumulator truncate, and those of k-steps that
// are mostly padding cost least while the sums are small, so where channels do not fill the k-steps the last block is taken first
// (45 x 33 x 64 x 64 -> 35 6.0e-7 -> 4.0e-7 against 64 bits, 49 channels 7.5e-7 -> 6.2e-7, the same time).
//
// One CTA per SM walks the tiles.  Both accumulators (512 columns) belong to one tile; the epilogue reads the
// cross products first, which the next tile starts with, so the tensor pipe waits for about the drain of
// the leading accumulator (a few hundred of ~14,000 clocks per tile of 64 channels) and the store runs under
// the next tile's MMAs.  Two rings of stages: filter k-blocks (one per tap and channel block) and halos (one
// per channel block).  Rows = 128 output channels, columns = positions.  Every wait is bounded.
#include "common.cuh"
#include "half_split.cuh"
#include "split.cuh"
#include "tc_ptx.cuh"
#include "tmap.cuh"

#include <algorithm>

// Optional per-CTA clock accounting for tuning; compiled in only with -DCT_CONV_TRACE.
#ifdef CT_CONV_TRACE
__device__ unsigned long long g_halo_trace[256 * 16];
#define CH_CLOCK() clock64()
#define CH_ACCUM(slot, cycles)                                                          \
    do {                                                                                \
        if (blockIdx.x < 256)                                                           \
            g_halo_trace[blockIdx.x * 16 + (slot)] += (unsigned long long)(cycles);     \
    } while (0)
extern "C" int ct_debug_halo_trace(unsigned long long *host, int count, int clear) {
    int rc = (int)cudaMemcpyFromSymbol(host, g_halo_trace, sizeof(unsigned long long) * (size_t)count);
    if (clear) {
        static unsigned long long zeros[256 * 16];
        cudaMemcpyToSymbol(g_halo_trace, zeros, sizeof(zeros));
    }
    return rc;
}
#else
#define CH_CLOCK() 0ll
#define CH_ACCUM(slot, cycles) do { } while (0)
#endif

namespace ct {
namespace {

using namespace ptx;

constexpr int kH_RowB       = 64;                     // bytes of k per operand row and k-block: 32 float16 / 16 tf32
constexpr int kH_AStages    = 4;
constexpr int kH_HaloStages = 4;                      // at most; as many as shared memory holds
constexpr int kH_ABytes     = 128 * kH_RowB;          // one filter plane of a k-block
constexpr int kH_AStageBytes = 2 * kH_ABytes;         // hi + lo
constexpr int kH_EpiWarps   = 8;
constexpr int kH_Threads    = 64 + 32 * kH_EpiWarps;
constexpr int kH_EpiRowBytes  = 32 * 4 + 16;          // 32 columns staged at a time, rows padded
constexpr int kH_EpiWarpBytes = 32 * kH_EpiRowBytes;
constexpr int kH_EpiBytes     = kH_EpiWarps * kH_EpiWarpBytes;
constexpr int kH_MinFilters = 17;
constexpr int kH_MaxTaps    = 32;
constexpr int kH_MaxStride  = 3;
constexpr int kH_MaxHalos   = kH_MaxStride * kH_MaxStride;
constexpr int kH_MaxK       = 1024; // values of k per drain of the leading accumulator
constexpr int kH_BiasSlots    = 256;                  // output channels whose bias is kept in shared memory

struct ConvHaloParams {
    const float *bias;
    float *out;       // [batch][ko][ho][wo]
    uint32_t *flags;
    int ko, tiles_m;
    int ho, wo, pw;   // pw: positions of a tile row
    int th, tiles_y;
    // The filter taps in the order of the halos that they read (one halo for stride 1; the rows and columns of the input
    // that are alike modulo the stride are a sub-image each).
    int halos;                          // per channel block
    uint8_t halo_image[kH_MaxHalos];    // its sub-image
    uint8_t halo_taps[kH_MaxHalos + 1]; // its first tap in the list; the last entry is the number of taps
    uint8_t tap[kH_MaxTaps];            // r * kw + s
    uint16_t tap_shift[kH_MaxTaps];     // position of the tap's first pixel in the box
    int box_x0, box_y0;                 // of tile row 0 in the sub-images
    int chunk_blocks;                   // blocks of 32 channels per drain of the leading accumulator
    int chunk_wide;                     // tf32 images: blocks of 16
    int c;                              // channels of the layer
    int last_first;                     // the channel blocks in descending order
    const float *filter_scale; // [ko] inverse scales
    const float *image_scale;  // [batch]; 0: this image's planes are tf32
    int c_pad;        // channels of the planes (k offset of a tap in the filter planes: tap * c_pad)
    int n_mma;        // th * pw rounded up to 16
    int box_bytes;    // one plane's halo box
    int halo_plane_bytes, halo_stages;
    int act;
};

struct ConvHaloMaps {
    CUtensorMap w16_hi, w16_lo, x16_hi, x16_lo;
    CUtensorMap w32_hi, w32_lo, x32_hi, x32_lo;
};

__global__ void __launch_bounds__(kH_Threads, 1) conv_halo_stream_kernel(
    const __grid_constant__ ConvHaloMaps maps, const __grid_constant__ ConvHaloParams p, const int all_tiles) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_a_full[kH_AStages], bar_a_empty[kH_AStages];
    __shared__ uint64_t bar_h_full[kH_HaloStages], bar_h_empty[kH_HaloStages];
    __shared__ uint64_t bar_tmem_full[2], bar_tmem_empty[2]; // 0: leading accumulator, 1: cross products
    __shared__ uint64_t bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s;
    // the layer's bias, read once: a load per stored row would put a trip to L2 in front of the add
    __shared__ float bias_s[kH_BiasSlots];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    griddep_launch_dependents();
    const uint32_t smem_base  = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t halo_base  = smem_base + kH_AStages * kH_AStageBytes;
    const uint32_t halo_stage = 2u * (uint32_t)p.halo_plane_bytes;
    uint8_t *epi_base = smem_raw + (smem_base - smem_u32(smem_raw)) + kH_AStages * kH_AStageBytes + (uint32_t)p.halo_stages * halo_stage;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kH_AStages; ++s) {
            mbar_init(smem_u32(&bar_a_full[s]), 1);
            mbar_init(smem_u32(&bar_a_empty[s]), 1);
        }
        for (int s = 0; s < kH_HaloStages; ++s) {
            mbar_init(smem_u32(&bar_h_full[s]), 1);
            mbar_init(smem_u32(&bar_h_empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_tmem_full[b]), 1);
            mbar_init(smem_u32(&bar_tmem_empty[b]), kH_EpiWarps);
        }
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        prefetch_tensormap(&maps.w16_hi);
        prefetch_tensormap(&maps.w16_lo);
        prefetch_tensormap(&maps.x16_hi);
        prefetch_tensormap(&maps.x16_lo);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    griddep_wait(); // the planes, the scales and what the caller's earlier kernels wrote
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
    for (int c = threadIdx.x; c < kH_BiasSlots; c += kH_Threads)
        bias_s[c] = (p.bias && c < p.ko) ? p.bias[c] : 0.0f;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    const bool failed        = abort_flag_s != 0; // an earlier launch failed: no work
    const int total_tiles    = failed ? 0 : all_tiles;
    __syncthreads(); // every thread has read abort_flag_s before a role may raise it

    // tile -> (row tile of output channels, tile row, image): neighbouring CTAs take the row tiles
    // of one pixel tile, so they read the same halo out of L2
    auto coords = [&](int tile, int &tm, int &ty, int &img) {
        tm       = tile % p.tiles_m;
        int rest = tile / p.tiles_m;
        img      = rest / p.tiles_y;
        ty       = rest - img * p.tiles_y;
    };

    if (warp == 0) {
        // ===== TMA producer =====
        if (elect_one()) {
            int ka = 0, kh2 = 0; // filter k-blocks and halos issued so far
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                int tm, ty, img;
                coords(tile, tm, ty, img);
                const bool wide          = p.image_scale[img] == 0.0f;
                const CUtensorMap *mw_hi = wide ? &maps.w32_hi : &maps.w16_hi, *mw_lo = wide ? &maps.w32_lo : &maps.w16_lo;
                const CUtensorMap *mx_hi = wide ? &maps.x32_hi : &maps.x16_hi, *mx_lo = wide ? &maps.x32_lo : &maps.x16_lo;
                const int block_k = wide ? 16 : 32, cblocks = p.c_pad / block_k; // channels per k-block
                for (int b = 0; b < cblocks && ok; ++b) {
                    const int cb = p.last_first ? cblocks - 1 - b : b;
                    for (int h = 0; h < p.halos && ok; ++h, ++kh2) {
                        const int hs = kh2 % p.halo_stages;
                        if (!mbar_wait(smem_u32(&bar_h_empty[hs]), ((uint32_t)(kh2 / p.halo_stages) & 1u) ^ 1u, abort_flag)) {
                            ok = false;
                            break;
                        }
                        const uint32_t hfull = smem_u32(&bar_h_full[hs]);
                        const uint32_t hdst  = halo_base + (uint32_t)hs * halo_stage;
                        const int y0 = ty * p.th + p.box_y0, sub = p.halo_image[h];
                        mbar_expect_tx(hfull, 2u * (uint32_t)p.box_bytes);
                        tma_load_5d(hdst, mx_hi, hfull, cb * block_k, p.box_x0, y0, sub, img);
                        tma_load_5d(hdst + (uint32_t)p.halo_plane_bytes, mx_lo, hfull, cb * block_k, p.box_x0, y0, sub, img);
                        for (int t = p.halo_taps[h]; t < p.halo_taps[h + 1]; ++t, ++ka) {
                            const int s = ka % kH_AStages;
                            if (!mbar_wait(smem_u32(&bar_a_empty[s]), ((uint32_t)(ka / kH_AStages) & 1u) ^ 1u, abort_flag)) {
                                ok = false;
                                break;
                            }
                            const uint32_t full = smem_u32(&bar_a_full[s]);
                            const uint32_t dst  = smem_base + (uint32_t)s * kH_AStageBytes;
                            mbar_expect_tx(full, (uint32_t)kH_AStageBytes);
                            const int32_t kc = p.tap[t] * p.c_pad + cb * block_k;
                            tma_load_2d(dst, mw_hi, full, kc, tm * 128);
                            tma_load_2d(dst + kH_ABytes, mw_lo, full, kc, tm * 128);
                        }
                    }
                }
            }
            if (*abort_flag) {
                // unwind: let the copies still in flight land before the CTA goes away
                for (int k2 = ka - kH_AStages < 0 ? 0 : ka - kH_AStages; k2 < ka; ++k2) {
                    const uint64_t t0 = globaltimer_ns();
                    while (!mbar_try_wait(smem_u32(&bar_a_full[k2 % kH_AStages]), (uint32_t)(k2 / kH_AStages) & 1u) &&
                           globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
                for (int k2 = kh2 - p.halo_stages < 0 ? 0 : kh2 - p.halo_stages; k2 < kh2; ++k2) {
                    const uint64_t t0 = globaltimer_ns();
                    while (!mbar_try_wait(smem_u32(&bar_h_full[k2 % p.halo_stages]), (uint32_t)(k2 / p.halo_stages) & 1u) &&
                           globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        if (elect_one()) {
            int ka = 0, kh2 = 0, i = 0, crosses = 0, mains = 0; // accumulations begun so far
            bool ok = true;
            const long long t_start = CH_CLOCK();
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++i) {
                int tm, ty, img;
                coords(tile, tm, ty, img);
                const bool wide      = p.image_scale[img] == 0.0f; // looked up while the MMAs of the last tile run
                const uint32_t idesc = make_idesc(wide ? 2u : 0u, 128, (uint32_t)p.n_mma);
                const int cblocks = p.c_pad / (wide ? 16 : 32), chunk = wide ? p.chunk_wide : p.chunk_blocks;
                // what the accumulator held before has been read
                auto wait_empty = [&](int acc) {
                    const bool got = mbar_wait(smem_u32(&bar_tmem_empty[acc]), ((uint32_t)(acc ? crosses++ : mains++) & 1u) ^ 1u, abort_flag);
                    tc_fence_after_sync();
                    return got;
                };
                const uint32_t d_main = tmem_base, d_cross = tmem_base + 256u;
                bool first_cross = true, first_main = true;
                for (int b = 0; b < cblocks && ok; ++b) {
                    const int cb   = p.last_first ? cblocks - 1 - b : b;
                    const bool two = p.c - cb * 32 > 16; // k-steps of this block that hold channels
                    for (int h = 0; h < p.halos && ok; ++h, ++kh2) {
                        const int hs = kh2 % p.halo_stages;
                        const long long t1 = CH_CLOCK();
                        if (!mbar_wait(smem_u32(&bar_h_full[hs]), (uint32_t)(kh2 / p.halo_stages) & 1u, abort_flag)) {
                            ok = false;
                            break;
                        }
                        CH_ACCUM(1, CH_CLOCK() - t1); // waiting for a halo
                        const uint32_t x_hi = halo_base + (uint32_t)hs * halo_stage;
                        const uint32_t x_lo = x_hi + (uint32_t)p.halo_plane_bytes;
                        for (int t = p.halo_taps[h]; t < p.halo_taps[h + 1]; ++t, ++ka) {
                            const int s = ka % kH_AStages;
                            const long long t2 = CH_CLOCK();
                            if (!mbar_wait(smem_u32(&bar_a_full[s]), (uint32_t)(ka / kH_AStages) & 1u, abort_flag)) {
                                ok = false;
                                break;
                            }
                            CH_ACCUM(2, CH_CLOCK() - t2); // waiting for filter planes
                            tc_fence_after_sync();
                            const uint32_t a_hi = smem_base + (uint32_t)s * kH_AStageBytes, a_lo = a_hi + kH_ABytes;
                            // the tap's pixels: the halo, so many rows of 64 bytes further on
                            const uint32_t shift = (uint32_t)p.tap_shift[t] * (uint32_t)kH_RowB;
                            const uint64_t da_hi = smem_desc_k<kH_RowB>(a_hi), da_lo = smem_desc_k<kH_RowB>(a_lo);
                            const uint64_t db_hi = smem_desc_k<kH_RowB>(x_hi + shift), db_lo = smem_desc_k<kH_RowB>(x_lo + shift);
                            if (first_cross && !wait_empty(1)) {
                                ok = false;
                                break;
                            }
                            if (!wide) {
                                mma_f16(d_cross, da_lo, db_hi, idesc, first_cross ? 0u : 1u);
                                mma_f16(d_cross, da_hi, db_lo, idesc, 1u);
                                if (two) {
                                    mma_f16(d_cross, da_lo + 2, db_hi + 2, idesc, 1u);
                                    mma_f16(d_cross, da_hi + 2, db_lo + 2, idesc, 1u);
                                }
                            } else {
#pragma unroll
                                for (int kk = 0; kk < kH_RowB / 32; ++kk) {
                                    mma_tf32(d_cross, da_lo + 2 * kk, db_hi + 2 * kk, idesc, first_cross && kk == 0 ? 0u : 1u);
                                    mma_tf32(d_cross, da_hi + 2 * kk, db_lo + 2 * kk, idesc, 1u);
                                }
                            }
                            if (first_main && !wait_empty(0)) {
                                ok = false;
                                break;
                            }
                            if (!wide) {
                                mma_f16(d_main, da_hi, db_hi, idesc, first_main ? 0u : 1u);
                                if (two)
                                    mma_f16(d_main, da_hi + 2, db_hi + 2, idesc, 1u);
                            } else {
#pragma unroll
                                for (int kk = 0; kk < kH_RowB / 32; ++kk)
                                    mma_tf32(d_main, da_hi + 2 * kk, db_hi + 2 * kk, idesc, first_main && kk == 0 ? 0u : 1u);
                            }
                            first_cross = false;
                            first_main = false;
                            tc_commit(smem_u32(&bar_a_empty[s]));
                        }
                        if (ok)
                            tc_commit(smem_u32(&bar_h_empty[hs])); // the halo is free once its taps' MMAs have retired
                    }
                    if (ok && b + 1 < cblocks && (b + 1) % chunk == 0) {
                        tc_commit(smem_u32(&bar_tmem_full[0]));
                        first_main = true;
                    }
                }
                if (ok) {
                    tc_commit(smem_u32(&bar_tmem_full[1]));
                    tc_commit(smem_u32(&bar_tmem_full[0]));
                }
            }
            CH_ACCUM(3, CH_CLOCK() - t_start); // the MMA thread's whole loop
            CH_ACCUM(4, i);
            if (!ok || *abort_flag) {
                tc_commit(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else {
        // ===== epilogue: drain tile i to registers, release the accumulator, then store =====
        const int ew      = warp - 2;
        const int quarter = warp & 3;
        const int half    = ew >> 2;
        uint8_t *stg      = epi_base + (uint32_t)ew * kH_EpiWarpBytes;
        // where this lane's columns land: column col = half * 128 + 32 j + lane is position
        // (y, x) = (col / pw, col % pw); -1 for the halo columns and past the tile
        int off[4];
        const int npos = p.th * p.pw;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = half * 128 + 32 * j + lane;
            const int y = col / p.pw, x = col - y * p.pw;
            off[j] = (col < npos && x < p.wo) ? y * p.wo + x : -1;
        }
        const bool relu = p.act == CT_ACT_RELU;
        int mains = 0, crosses = 0;
        for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
            int tm, ty, img;
            coords(tile, tm, ty, img);
            const int row0     = tm * 128 + quarter * 32; // first output channel of this warp's block
            const float inv    = p.image_scale[img];
            const bool wide    = inv == 0.0f;
            const float rs     = (!wide && row0 + lane < p.ko) ? p.filter_scale[row0 + lane] : 1.0f;
            // powers of two; a missing bias is -0, which no sum notices
            const float scale  = wide ? 1.0f : __fmul_rn(rs, inv);
            const int ch       = row0 + lane;
            const float bias   = !p.bias || ch >= p.ko ? -0.0f : (ch < kH_BiasSlots ? bias_s[ch] : p.bias[ch]);
            const long long e0 = CH_CLOCK();
            float acc[128];
            const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 128);
            auto await = [&](int which) {
                const bool got = mbar_wait(smem_u32(&bar_tmem_full[which]), (uint32_t)(which ? crosses++ : mains++) & 1u, abort_flag);
                tc_fence_after_sync();
                return __all_sync(0xffffffffu, got) != 0;
            };
            auto hand_back = [&](int which) {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(smem_u32(&bar_tmem_empty[which]));
            };
            // The leading accumulator of every chunk but the last, the cross products, the last chunk.
            // The first of them straight into the sums, with one wait for all columns.
            const int cblocks = p.c_pad / (wide ? 16 : 32), chunk = wide ? p.chunk_wide : p.chunk_blocks, chunks = (cblocks + chunk - 1) / chunk;
            const int events  = chunks + 1;
            const float cross = wide ? 1.0f : kHalfLoInv;
            auto which_of     = [&](int e) { return e == chunks - 1 ? 1 : 0; };
            const int first_acc = which_of(0);
            if (!await(first_acc))
                break;
            {
                uint32_t r[4][32];
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    tmem_ld_32x32(lane_base + (uint32_t)(first_acc * 256 + g * 32), r[g]);
                tmem_ld_wait();
                hand_back(first_acc);
                const float weight = first_acc ? cross : 1.0f;
#pragma unroll
                for (int j = 0; j < 128; ++j)
                    acc[j] = __fmul_rn(__uint_as_float(r[j / 32][j % 32]), weight);
            }
            bool ok = true;
#pragma unroll 1
            for (int e = 1; e < events; ++e) {
                const int which    = which_of(e);
                const float weight = which ? cross : 1.0f;
                ok                 = await(which);
                if (!ok)
                    break;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    uint32_t r[16];
                    tmem_ld_32x16(lane_base + (uint32_t)(which * 256 + g * 16), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[g * 16 + j] = __fadd_rn(acc[g * 16 + j], __fmul_rn(__uint_as_float(r[j]), weight));
                }
                hand_back(which);
            }
            if (!ok)
                break;
            const long long e1 = CH_CLOCK();

            const int y0   = ty * p.th;
            // positions of rows past the image's last row (a partial last tile) are dropped:
            // position col lies in row col / pw, so the valid ones are col < rows_left * pw
            const int col_limit = (p.ho - y0 < p.th ? p.ho - y0 : p.th) * p.pw;
            // Scales, bias and activation where a lane has a channel, with its constants in registers; what remains for the
            // stores is a read, an address and the store.  (With them behind the exchange, a value took 35 instructions and
            // a tile the epilogue 18,000 clocks, four thousand more than its MMAs.)
            const int64_t plane = (int64_t)p.ho * p.wo;
            float *out_img = p.out + ((int64_t)img * p.ko + row0) * plane + (int64_t)y0 * p.wo;
            const int rows = p.ko - row0 < 32 ? p.ko - row0 : 32;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (half * 128 + g * 32 >= npos || rows <= 0)
                    break;
                float4 *mine = reinterpret_cast<float4 *>(stg + lane * kH_EpiRowBytes);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float y[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        y[q] = __fadd_rn(__fmul_rn(acc[g * 32 + 4 * j + q], scale), bias);
                        y[q] = !relu || y[q] > 0.0f ? y[q] : __fmul_rn(y[q], 0.0f);
                    }
                    mine[j] = make_float4(y[0], y[1], y[2], y[3]);
                }
                __syncwarp();
                // a column per lane, so that a store covers consecutive pixels of a channel (four columns per lane wrote every
                // sector four times: 256 x 64 x 56 x 56 -> 128 530 us, 491 so)
                const float *src = reinterpret_cast<const float *>(stg) + lane;
                float *dst       = out_img + (off[g] < 0 ? 0 : off[g]);
                if (off[g] >= 0 && half * 128 + g * 32 + lane < col_limit) {
                    int r = 0;
#pragma unroll 1
                    for (; r + 8 <= rows; r += 8) {
                        float x[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            x[u] = src[(r + u) * (kH_EpiRowBytes / 4)];
#pragma unroll
                        for (int u = 0; u < 8; ++u, dst += plane)
                            *dst = x[u];
                    }
#pragma unroll 1
                    for (; r < rows; ++r, dst += plane)
                        *dst = src[r * (kH_EpiRowBytes / 4)];
                }
                __syncwarp(); // the block is rewritten by the next columns
            }
            if (warp == 2 && lane == 0) {
                CH_ACCUM(5, e1 - e0);          // epilogue: waiting for a complete accumulator
                CH_ACCUM(6, CH_CLOCK() - e1);  // drain and store
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
    if (threadIdx.x == 0 && !failed && *abort_flag)
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

// ---- pre-pass -----------------------------------------------------------------------------
//
// Two launches: the range of every image, in slices, next to the filters (both forms of their planes, a block per
// filter); then the input as NHWC planes, in the form that the image's range allows.

// Blocks 0 .. ko - 1: filter [c][taps] -> planes [taps * c_pad], tap-major k (none if hi16 is null), and its inverse
// scale, 0 where the range of the filter does not fit float16 pairs.  The others: slice (blockIdx.x - ko) of the images
// ([batch][count] floats, `slices` to an image).
struct FilterPlanes {
    __half *hi16, *lo16;
    float *hi32, *lo32;
    float *scale;
};
__global__ void __launch_bounds__(256) conv_range_kernel(
    const float *__restrict__ w, int c, int taps, int c_pad, int ko, const FilterPlanes f, const float *__restrict__ x,
    int64_t count, int slices, int vec_ok, uint2 *__restrict__ ranges) {
    __shared__ uint2 part[8];
    griddep_launch_dependents();
    griddep_wait();
    const bool filter = (int64_t)blockIdx.x < ko;
    const int64_t o   = filter ? blockIdx.x : (blockIdx.x - ko) / slices;
    const int slice   = filter ? 0 : (int)(blockIdx.x - ko - o * slices);
    const float *src  = filter ? w + o * c * taps : x + o * count;
    const int64_t n   = filter ? (int64_t)c * taps : count;
    const int64_t step = filter ? 256 : (int64_t)slices * 256;
    uint2 r            = make_uint2(0u, kNoneSmallest);
    if (!filter && vec_ok) {
        const float4 *s4 = reinterpret_cast<const float4 *>(src);
#pragma unroll 8
        for (int64_t i = (int64_t)slice * 256 + threadIdx.x; i < n / 4; i += step) {
            const float4 q = s4[i];
            range_take(r, q.x), range_take(r, q.y), range_take(r, q.z), range_take(r, q.w);
        }
    } else {
#pragma unroll 8
        for (int64_t i = (int64_t)slice * 256 + threadIdx.x; i < n; i += step)
            range_take(r, src[i]);
    }
    r = range_warp(r);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = r;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j)
        r = range_join(r, part[j]);
    if (!filter) {
        if (threadIdx.x == 0)
            ranges[o * slices + slice] = r;
        return;
    }
    float scale, inverse;
    const bool fits = half_range_fits(r, scale, inverse);
    if (threadIdx.x == 0)
        f.scale[o] = fits ? inverse : 0.0f;
    if (f.hi16 == nullptr)
        return;
    for (int i = threadIdx.x; i < taps * c_pad; i += 256) {
        const int tap = i / c_pad, ic = i - tap * c_pad;
        const float v    = ic < c ? src[ic * taps + tap] : 0.0f;
        const int64_t at = o * taps * c_pad + i;
        split_half(v, scale, f.hi16[at], f.lo16[at]);
        split_tf32(v, f.hi32[at], f.lo32[at]);
    }
}

// x [batch][c][hw] -> NHWC planes [hw][c_pad], hi then lo, in the image's slot of 8 bytes per value: float16 pairs
// under the image's scale, or tf32 terms (image_scale 0) where the image or any filter does not fit those.  A
// block takes 64 channels by 64 positions through shared memory: reads of 256 contiguous bytes, writes of 128.  The
// images are taken last to first: the end of the tensor is what conv_range_kernel has just left in L2.
// Sub-images (ConvSubImages, hs x ws each): zeros where the image has no such row or column, those that no tap reads are
// left out.
//
// What bounds it is issue (0.83 of the slots at 128 x 64 x 56 x 56), so the moduli are constants, the one division left is a
// multiplication, and one warp works the image's scale out for all: 64 x 48 x 57 x 57 -> 96 at stride 2 76 -> 69 us (31 of it this kernel
// before), 256 x 64 x 56 x 56 -> 128 428 -> 425.
struct PlaneGeom {
    int h, w, hs, ws;
    uint32_t width_inv; // 2^32 / (ws * col_mod), rounded up; 0 for a width of 1
    ConvSubImages sub;
};
template <int ROW_MOD, int COL_MOD>
__global__ void __launch_bounds__(256) conv_planes_kernel(
    const float *__restrict__ x, int c, const PlaneGeom geom, int c_pad, const uint2 *__restrict__ ranges, int slices,
    const float *__restrict__ filter_scale, int ko, uint8_t *__restrict__ slots, float *__restrict__ image_scale) {
    __shared__ float tile[64][65];
    __shared__ float scale_s;
    __shared__ int fits_s;
    griddep_launch_dependents();
    griddep_wait();
    const int64_t img = gridDim.z - 1 - blockIdx.z;
    const int64_t q0  = (int64_t)blockIdx.x * 64;
    const int c0      = (int)blockIdx.y * 64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t in_hw = (int64_t)geom.h * geom.w;
    const int width  = geom.ws * COL_MOD;
    const int64_t hw = (int64_t)geom.hs * ROW_MOD * width; // positions of the image grown to whole multiples
    constexpr bool apart = ROW_MOD * COL_MOD > 1;
    const float *src = x + (img * c + c0) * in_hw;
    auto row_of = [&](int64_t q) { // q < 2^31: the rounded-up quotient is one too high at most
        const int row = geom.width_inv ? (int)__umulhi((uint32_t)q, geom.width_inv) : (int)q;
        return row - (row * width > (int)q ? 1 : 0);
    };
    // position q of the grown image in the input (-1: not there)
    auto source = [&](int64_t q) -> int64_t {
        if (!apart)
            return q < hw ? q : -1;
        const int row = row_of(q), col = (int)q - row * width;
        return q < hw && row < geom.h && col < geom.w ? (int64_t)row * geom.w + col : -1;
    };
    float v[16]; // every load before the first use of any
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int64_t from = source(q0 + lane + 32 * t);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int ch = warp + 8 * j;
            v[2 * j + t] = (c0 + ch < c && from >= 0) ? __ldcs(src + ch * in_hw + from) : 0.0f;
        }
    }
    if (warp == 0) {
        uint2 r = make_uint2(0u, kNoneSmallest);
        for (int s = lane; s < slices; s += 32)
            r = range_join(r, ranges[img * slices + s]);
        float s, inverse;
        const bool all = half_range_fits(range_warp(r), s, inverse);
        if (lane == 0)
            scale_s = s, fits_s = all;
    }
    int bad_filter = 0;
    for (int o = threadIdx.x; o < ko; o += 256)
        bad_filter |= filter_scale[o] == 0.0f ? 1 : 0;
#pragma unroll
    for (int j = 0; j < 16; ++j)
        tile[warp + 8 * (j >> 1)][lane + 32 * (j & 1)] = v[j];
    const bool fits   = !__syncthreads_or(bad_filter) && fits_s;
    const float scale = scale_s;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        image_scale[img] = fits ? 1.0f / scale : 0.0f; // a power of two
    const int64_t plane = hw * c_pad;
    uint8_t *slot       = slots + img * plane * 8;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int chunk = threadIdx.x & 7, q = (threadIdx.x >> 3) + 32 * t;
        if (q0 + q >= hw || c0 + chunk * 8 >= c_pad)
            continue;
        int64_t to = q0 + q;
        if (apart) {
            const int row = row_of(to), col = (int)to - row * width, sub = row % ROW_MOD * COL_MOD + col % COL_MOD;
            if (!(geom.sub.used >> sub & 1u))
                continue;
            if (fits || !geom.sub.tf32_plain)
                to = ((int64_t)sub * geom.hs + row / ROW_MOD) * geom.ws + col / COL_MOD;
            else if (row < geom.h && col < geom.w)
                to = (int64_t)row * geom.w + col;
            else
                continue;
        }
        const int64_t at = to * c_pad + c0 + chunk * 8;
        if (fits) {
            __half2 hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                split_half_pair(tile[chunk * 8 + 2 * j][q] * scale, tile[chunk * 8 + 2 * j + 1][q] * scale, hi[j], lo[j]);
            __half *p_hi = reinterpret_cast<__half *>(slot) + at;
            *reinterpret_cast<uint4 *>(p_hi)         = *reinterpret_cast<uint4 *>(hi);
            *reinterpret_cast<uint4 *>(p_hi + plane) = *reinterpret_cast<uint4 *>(lo);
        } else {
            float *p_hi = reinterpret_cast<float *>(slot) + at;
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                float hi[4], lo[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    split_tf32_flat(tile[chunk * 8 + j + u][q], hi[u], lo[u]);
                *reinterpret_cast<float4 *>(p_hi + j)         = make_float4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<float4 *>(p_hi + plane + j) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
}

struct HaloGeom {
    int pw, wo, ho, th, n_mma, box_rows, plane_bytes, stages;
    int hs, ws;         // extents of a sub-image
    int y_min, x_min;   // smallest row and column offset of a tap in its sub-image
    size_t smem;
};

int floor_div(int64_t a, int64_t b) { return (int)(a >= 0 ? a / b : -((-a + b - 1) / b)); }

// Tap (r, q) of output (oy, ox) reads input row oy * stride - pad + r = stride * (oy + a) + py: row oy + a of the
// sub-image py, and so for columns.  A tile is th rows of pw = wo + (largest - smallest b) positions.
bool halo_geometry(int64_t h, int64_t w, int64_t kh, int64_t kw, int64_t stride, int64_t pad, HaloGeom *g) {
    if (w + 2 * pad < kw || h + 2 * pad < kh || pad > 256 || kh > 256 || kw > 256)
        return false;
    const int64_t wo = (w + 2 * pad - kw) / stride + 1, ho = (h + 2 * pad - kh) / stride + 1;
    g->y_min = floor_div(-pad, stride), g->x_min = floor_div(-pad, stride);
    const int64_t span_y = floor_div(kh - 1 - pad, stride) - g->y_min, span_x = floor_div(kw - 1 - pad, stride) - g->x_min;
    const int64_t pw = wo + span_x;
    g->hs = (int)((h + stride - 1) / stride), g->ws = (int)((w + stride - 1) / stride);
    if (pw > 256)
        return false;
    // as many rows as 256 columns of the accumulator and the shared memory take
    for (int64_t th = std::min<int64_t>(256 / pw, ho); th >= 1; --th) {
        if (th + span_y > 256)
            continue;
        g->pw = (int)pw, g->wo = (int)wo, g->ho = (int)ho, g->th = (int)th;
        g->n_mma    = (int)((th * pw + 15) / 16 * 16);
        g->box_rows = (int)(th + span_y);
        // a tap's shifted window of n_mma rows may run past the box: reserve those rows too
        const int64_t rows = std::max<int64_t>(span_y * pw + span_x + g->n_mma, (int64_t)g->box_rows * pw);
        g->plane_bytes     = (int)((rows * kH_RowB + 1023) & ~1023ll);
        // 227 KB per CTA less the kernel's static shared memory
        const int rest = 225 * 1024 - kH_AStages * kH_AStageBytes - kH_EpiBytes - 1024;
        g->stages      = std::min(kH_HaloStages, rest / (2 * g->plane_bytes));
        g->smem = (size_t)kH_AStages * kH_AStageBytes + (size_t)g->stages * 2 * g->plane_bytes + kH_EpiBytes + 1024;
        if (g->stages >= 2)
            return true;
    }
    return false;
}

} // namespace

// Slices of an image in conv_range_kernel: 16 float4 to a thread where there are images enough, down to four where there
// are few.
int conv_range_slices(int64_t batch, int64_t count) {
    const int64_t few = std::min<int64_t>(count / 4096, 1024 / batch);
    return (int)std::min<int64_t>(64, std::max<int64_t>(1, std::max(count / 16384, few)));
}

// The pre-pass of a layer: the filters' scales and (filters16 non-null) planes, the images' planes and scales.
// ranges: batch * conv_range_slices(batch, c * hw) pairs of words.
ct_status conv_prepass(
    DeviceState *st, const float *x, const float *w, int64_t batch, int64_t c, int64_t h, int64_t wd, int64_t c_pad, int64_t ko,
    int64_t taps, void *filters16, void *filters32, size_t plane16, size_t plane32, float *filter_scale, void *ranges, float *image_scale,
    void *slots, const ConvSubImages &sub) {
    (void)st;
    const int64_t hw = h * wd;
    if (batch > 65535 || c_pad / 32 > 65535)
        return fail(CT_ERR_TOO_LARGE, "conv2d: batch or channel count too large for the layout pre-pass");
    const int64_t count = c * hw;
    const int slices    = conv_range_slices(batch, count);
    const int vec       = (count & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    uint8_t *f16 = static_cast<uint8_t *>(filters16), *f32 = static_cast<uint8_t *>(filters32);
    const FilterPlanes f{reinterpret_cast<__half *>(f16), reinterpret_cast<__half *>(f16 + plane16), reinterpret_cast<float *>(f32),
                         reinterpret_cast<float *>(f32 + plane32), filter_scale};
    ProfScope prof("conv_prepass");
    CT_CUDA(launch_dependent(conv_range_kernel, dim3((unsigned)(ko + batch * slices)), dim3(256), 0, stream(), w, (int)c, (int)taps,
                             (int)c_pad, (int)ko, f, x, count, slices, vec, static_cast<uint2 *>(ranges)));
    CT_LAUNCH_CHECK("conv_range");
    PlaneGeom geom{(int)h, (int)wd, (int)((h + sub.row_mod - 1) / sub.row_mod), (int)((wd + sub.col_mod - 1) / sub.col_mod), 0, sub};
    const int64_t width = (int64_t)geom.ws * sub.col_mod, positions = geom.hs * width * sub.row_mod;
    geom.width_inv = width > 1 ? (uint32_t)(((1ull << 32) + width - 1) / width) : 0;
    const dim3 grid((unsigned)((positions + 63) / 64), (unsigned)((c_pad + 63) / 64), (unsigned)batch);
    auto planes = [&](auto kernel) {
        return launch_dependent(kernel, grid, dim3(256), 0, stream(), x, (int)c, geom, (int)c_pad, static_cast<const uint2 *>(ranges), slices,
                                static_cast<const float *>(filter_scale), (int)ko, static_cast<uint8_t *>(slots), image_scale);
    };
    if (sub.row_mod == 1 && sub.col_mod == 1)
        CT_CUDA(planes(conv_planes_kernel<1, 1>));
    else if (sub.row_mod == 2 && sub.col_mod == 1)
        CT_CUDA(planes(conv_planes_kernel<2, 1>));
    else if (sub.row_mod == 2 && sub.col_mod == 2)
        CT_CUDA(planes(conv_planes_kernel<2, 2>));
    else
        CT_CUDA(planes(conv_planes_kernel<3, 3>));
    CT_LAUNCH_CHECK("conv_planes");
    return CT_OK;
}

// Whether the halo kernel takes this layer (float32 mode only): filters and strides within its tables, whole k-blocks
// of a tap list within one drain, and a tile that is reasonably full.
bool conv_halo_applicable(int64_t c_pad, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride,
                          int64_t pad) {
    HaloGeom g;
    if (stride < 1 || stride > kH_MaxStride || ko < kH_MinFilters || kh * kw > kH_MaxTaps || (c_pad % 32) != 0 ||
        c_pad > (1 << 20) || h > 0x3fff || w > 0x3fff)
        return false;
    if (!halo_geometry(h, w, kh, kw, stride, pad, &g))
        return false;
    // at least 70 % of the columns carry an output, and not a few rows only because shared memory holds no more
    return (int64_t)g.th * g.wo * 10 >= (int64_t)g.n_mma * 7 && (g.n_mma >= 128 || g.th == g.ho);
}

// Workspace: [filter scale][image scale][image ranges][w hi16][w lo16][w hi][w lo][image slots]; a slot holds an
// image's planes, float16 pairs or, where it does not fit those, tf32: no more than tf32 planes alone take.
ct_status conv_halo(
    DeviceState *st, const float *x, const float *w, int64_t batch, int64_t c, int64_t c_pad, int64_t h, int64_t wd, int64_t ko,
    int64_t kh, int64_t kw, int64_t stride, int64_t pad, const float *bias, int act, float *out) {
    HaloGeom g;
    if (!halo_geometry(h, wd, kh, kw, stride, pad, &g))
        return fail(CT_ERR_INVALID, "conv2d: internal tile shape not usable");
    auto align_up          = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    const int64_t taps     = kh * kw, subs = stride * stride, sub = (int64_t)g.hs * g.ws, hw = sub * subs;
    const size_t w16       = align_up((size_t)ko * taps * c_pad * 2), w32 = align_up((size_t)ko * taps * c_pad * 4);
    const size_t slot      = (size_t)hw * c_pad * 8;
    const size_t w_words   = align_up((size_t)ko * 4), x_words = align_up((size_t)batch * 4);
    const size_t ranges    = align_up((size_t)batch * conv_range_slices(batch, c * h * wd) * 8);
    CT_TRY(ensure_ws(&st->gemm_ws, &st->gemm_ws_bytes, w_words + x_words + ranges + 2 * w16 + 2 * w32 + (size_t)batch * slot));
    uint8_t *ws            = static_cast<uint8_t *>(st->gemm_ws);
    float *filter_scale    = reinterpret_cast<float *>(ws), *image_scale = reinterpret_cast<float *>(ws + w_words);
    uint8_t *w16_hi        = ws + w_words + x_words + ranges, *w32_hi = w16_hi + 2 * w16, *xp = w32_hi + 2 * w32;
    ConvHaloParams p;
    p.filter_scale = filter_scale, p.image_scale = image_scale;
    p.bias = bias, p.out = out, p.flags = st->flags_dev;
    p.ko = (int)ko, p.tiles_m = (int)((ko + 127) / 128);
    p.ho = g.ho, p.wo = g.wo, p.pw = g.pw, p.th = g.th;
    p.tiles_y = (g.ho + g.th - 1) / g.th;
    p.box_x0 = g.x_min, p.box_y0 = g.y_min;
    p.chunk_blocks = (int)std::max<int64_t>(1, kH_MaxK / (32 * taps));
    // a strided layer's tf32 images: no longer chains of truncating additions than the float16 ones have (3.0e-6 -> 3.7e-7 against
    // 64 bits at 48 channels, 3 x 3; all 64 images 110 -> 117 us); unstrided, with the cross products apart, 4.0e-6 -> 1.4e-6
    p.chunk_wide = stride > 1 ? 1 : 2 * p.chunk_blocks;
    p.c       = (int)c;
    p.last_first = c % 16 != 0;
    p.c_pad   = (int)c_pad;
    p.n_mma   = g.n_mma;
    p.box_bytes        = g.box_rows * g.pw * kH_RowB;
    p.halo_plane_bytes = g.plane_bytes, p.halo_stages = g.stages;
    p.act = act;
    p.halos = 0, p.halo_taps[0] = 0;
    uint32_t used = 0;
    for (int image = 0, listed = 0; image < (int)subs; ++image) {
        for (int t = 0; t < (int)taps; ++t) {
            const int r = t / (int)kw - (int)pad, q = t % (int)kw - (int)pad, a = floor_div(r, stride), b = floor_div(q, stride);
            if ((r - a * (int)stride) * (int)stride + (q - b * (int)stride) != image)
                continue;
            p.tap[listed]         = (uint8_t)t;
            p.tap_shift[listed++] = (uint16_t)((a - g.y_min) * g.pw + (b - g.x_min));
        }
        if (listed > p.halo_taps[p.halos]) {
            p.halo_image[p.halos]  = (uint8_t)image;
            p.halo_taps[++p.halos] = (uint8_t)listed;
            used |= 1u << image;
        }
    }
    CT_TRY(conv_prepass(st, x, w, batch, c, h, wd, c_pad, ko, taps, w16_hi, w32_hi, w16, w32, filter_scale, ws + w_words + x_words,
                        image_scale, xp, ConvSubImages{(int)stride, (int)stride, used, false}));
    const int64_t tiles = (int64_t)p.tiles_m * p.tiles_y * batch;
    if (tiles > 0x7fffffffll)
        return fail(CT_ERR_TOO_LARGE, "conv2d: too many tiles");
    ConvHaloMaps maps;
    auto encode = [&](CUtensorMap *mw, const uint8_t *wp, CUtensorMap *mx, const uint8_t *xpl, int elem) {
        const uint64_t kp = (uint64_t)(taps * c_pad), row = (uint64_t)(c_pad * elem);
        const uint64_t wdims[2] = {kp, (uint64_t)ko}, wstr[1] = {kp * (uint64_t)elem};
        const uint32_t wbox[2]  = {(uint32_t)(kH_RowB / elem), 128};
        const uint64_t xdims[5] = {(uint64_t)c_pad, (uint64_t)g.ws, (uint64_t)g.hs, (uint64_t)subs, (uint64_t)batch};
        const uint64_t xstr[4]  = {row, row * (uint64_t)g.ws, row * (uint64_t)sub, slot};
        const uint32_t xbox[5]  = {(uint32_t)(kH_RowB / elem), (uint32_t)g.pw, (uint32_t)g.box_rows, 1, 1};
        auto fn = elem == 4 ? encode_tiled_map_f32 : encode_tiled_map_f16;
        CT_TRY(fn(mw, wp, 2, wdims, wstr, wbox, kH_RowB));
        return fn(mx, xpl, 5, xdims, xstr, xbox, kH_RowB);
    };
    CT_TRY(encode(&maps.w16_hi, w16_hi, &maps.x16_hi, xp, 2));
    CT_TRY(encode(&maps.w16_lo, w16_hi + w16, &maps.x16_lo, xp + slot / 4, 2));
    CT_TRY(encode(&maps.w32_hi, w32_hi, &maps.x32_hi, xp, 4));
    CT_TRY(encode(&maps.w32_lo, w32_hi + w32, &maps.x32_lo, xp + slot / 2, 4));
    // the kernel also has a little static shared memory (barriers, the bias): ask for exactly what
    // this geometry needs, remembering the largest request per device
    static size_t attr_bytes_dev[16] = {};
    size_t &attr_bytes = attr_bytes_dev[st->device & 15];
    if (g.smem > attr_bytes) {
        CT_CUDA(cudaFuncSetAttribute(conv_halo_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
        attr_bytes = g.smem;
    }
    const unsigned grid = (unsigned)(tiles < st->sm_count ? tiles : st->sm_count);
    ProfScope prof("gemm_tc");
    CT_CUDA(launch_dependent(conv_halo_stream_kernel, dim3(grid), dim3(kH_Threads), g.smem, stream(), maps, p, (int)tiles));
    CT_LAUNCH_CHECK("conv_halo_stream");
    return CT_OK;
}

} // namespace ct
