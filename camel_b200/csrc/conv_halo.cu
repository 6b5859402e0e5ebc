// Implicit-GEMM conv2d (stride 1 to 3): the input halo of a tile is fetched once per channel block and serves all
// filter taps.
//
// The rows and columns of the input that are alike modulo the stride are sub-images, each written by the pre-pass as planes
// [position][channel] with the padding in them, pw positions to a row.  Position q of the output, q = y * pw + x (the pw - wo
// columns behind a row's end are computed and dropped), reads position q + shift of a tap's sub-image, whatever q: so a tile is any
// 128 consecutive positions, whole rows or not, its halo the 128 + (largest shift) positions from its first one on, and a tap
// the same shared memory through a descriptor moved by `shift` rows of 64 bytes.  Nothing is wasted on tiles that rows do not fill.
//
// Pixels are the accumulator's rows: a tile of 256 x n belongs to a pair of CTAs (cta_group::2), 128 positions each, n filters (a
// multiple of 32, at most 128) shared out between them.  What bounds such a kernel is shared memory, 128 bytes per clock: with the
// filters on the rows of a CTA by itself and 240 positions on its columns, the operands took 98 of them, the filters' stream 23, and
// the exchange through which the sums reached the pixels' order 18 more; a tile of 13,000 clocks of MMAs took 18,800.  Here the
// filters of a layer stay in shared memory where they fit beside two halos (64 -> 128 channels, 3 x 3: 144 KB a CTA; a ring of
// stages otherwise), half of a filter operand is read by each CTA, and a lane of the epilogue has a pixel and its registers
// channels, so that scale, bias, activation and the store need no exchange.
//
// Arithmetic: split float16 (half_split.cuh), scaled per filter and per image - a scale has to be constant
// along k, and an output's patch crosses the whole halo - with the cross products in an accumulator of their
// own, as in gemm_half.cu.  An image that spans too many powers of two - or every image, where a filter does - has tf32 planes in
// the same place (16 channels to a row of 64 bytes) and runs the same loop over those.  The two tiles of a pair may be of images of
// different forms: then the pair runs twice and each tile is stored once.
//
// MMAs per 16 channels and tap (8 in tf32), two ways of sharing the filters out.  THREE: X_hi x W_hi, X_hi x W_lo, X_lo x W_hi, n columns each, every
// CTA holding half of the hi and half of the lo terms.  Otherwise X_hi x [W_hi; W_lo], 2 n columns, the leader holding the hi and its peer the
// lo terms, and X_lo x W_hi from another copy of half of the hi terms in each.  An MMA takes half a clock per column but not less than 49,
// so the second is the faster one for n < 96; the first takes two thirds of the memory, and serves fewer filters too where that decides
// whether they stay, or has them streamed.
//
// k beyond 1024 values: both accumulators are drained every 1024 and added up in registers.  Additions into an accumulator truncate, and
// those of k-steps that are mostly padding cost least while the sums are small, so where channels do not fill the k-steps the last block
// is taken first (45 x 33 x 64 x 64 -> 35 6.0e-7 -> 4.0e-7 against 64 bits, 49 channels 7.5e-7 -> 6.2e-7, the same time).
//
// A pair per two SMs walks the tiles, filters outermost; two sets of accumulators, so that a tile is drained and stored under the next
// one's MMAs.  Every wait is bounded.  Measured: the roles run as whole warps with uniform control flow, so that descriptors stay in
// uniform registers; entered by one thread, the issuer took 11,000 clocks for a tile of 6900 clocks of MMAs, and is told what
// a halo holds by the producer (8400).  Sixteen epilogue warps: with eight a tile's drain and store took longer than its MMAs.
// 256 x 64 x 56 x 56 -> 128: kernel 307 -> 235 us, layer 484 -> 435; 64 x 48 x 57 x 57 -> 96 at stride 2, layer 69.5 -> 57.1.
#include "common.cuh"
#include "half_split.cuh"
#include "split.cuh"
#include "tc_ptx.cuh"
#include "tmap.cuh"

#include <algorithm>

namespace ct {
namespace {

using namespace ptx;

constexpr int kH_RowB       = 64;                     // bytes of k per operand row and k-block: 32 float16 / 16 tf32
constexpr int kH_MaxSlots   = 96;                     // groups of filter k-blocks in shared memory (a few taps of a channel block each)
constexpr int kH_HaloStages = 4;                      // at most; as many as shared memory holds
constexpr int kH_EpiWarps   = 16;
constexpr int kH_Threads    = 64 + 32 * kH_EpiWarps;
constexpr int kH_Smem       = 220 * 1024;             // 227 KB per CTA less the static shared memory
constexpr int kH_MinFilters = 17;
constexpr int kH_MaxTaps    = 32;
constexpr int kH_MaxStride  = 3;
constexpr int kH_MaxHalos   = kH_MaxStride * kH_MaxStride;
// What the leader's producer tells the MMA issuer about a halo, beside its first tap and the tap behind its last (six bits each)
constexpr uint32_t kH_Wide = 1u << 12, kH_Two = 1u << 13, kH_Load = 1u << 14, kH_Begin = 1u << 15, kH_End = 1u << 16, kH_Set = 1u << 17,
                   kH_Reload = 1u << 18, kH_Over = 1u << 19;
constexpr int kH_MaxK       = 1024; // values of k per drain of the accumulators

// n / d for n < 2^31, from inv = 2^32 / d rounded up (0 for d = 1): the rounded-up quotient is one too high at most.
struct FastDiv {
    uint32_t d, inv;
};
__device__ __forceinline__ int fast_div(int n, const FastDiv &f) {
    const uint32_t q = f.inv ? __umulhi((uint32_t)n, f.inv) : (uint32_t)n;
    return (int)(q - (q * f.d > (uint32_t)n ? 1u : 0u));
}
FastDiv fast_divisor(int64_t d) { return {(uint32_t)d, d > 1 ? (uint32_t)(((1ull << 32) + d - 1) / d) : 0u}; }

struct ConvHaloParams {
    float *out;       // [batch][ko][ho][wo]
    uint32_t *flags;
    int ko, n;        // n: filters of a tile
    int ho, wo, pw;   // pw: positions of a row
    int image_tiles;  // of 128 positions
    int total_tiles, pairs; // of the batch; pairs of them
    int items;        // pairs times filter tiles
    // The filter taps in the order of the halos that they read (one halo for stride 1; a sub-image each otherwise).
    int halos;                          // per channel block
    int halo_at[kH_MaxHalos];           // position of its sub-image in the planes
    uint8_t halo_taps[kH_MaxHalos + 1]; // its first tap in the list; the last entry is the number of taps
    uint16_t tap_shift[kH_MaxTaps];     // positions between an output and the tap's pixel in the sub-image, in units of descriptors
    int chunk_blocks;                   // blocks of 32 channels per drain of the accumulators
    int chunk_wide;                     // tf32 images: blocks of 16
    int chunks, chunks_wide;            // drains
    int c;                              // channels of the layer
    int last_first;                     // the channel blocks in descending order
    const float *filter_scale; // [ko rounded up to whole tiles] inverse scales
    const float *bias;         // the same, -0 where there is none: no sum notices
    const float *image_scale;  // [batch]; 0: this image's planes are tf32
    int c_pad;        // channels of the planes (k offset of a tap in the filter planes: tap * c_pad)
    int box_rows, boxes; // positions of a TMA box, boxes of a halo
    int halo_plane_bytes, halo_stages;
    int slots, slot_bytes; // groups of filter k-blocks in shared memory
    int group, tap_bytes, f1;        // taps of a group, bytes between two of them, and from the first operand's terms to the second's
    int act;
    FastDiv by_pairs, by_tiles, by_pw; // pairs, image_tiles, pw
};

struct ConvHaloMaps {
    CUtensorMap x16_hi, x16_lo, x32_hi, x32_lo;
    // THREE: hi and lo terms of n / 2 filters in one box.  Otherwise one plane's of n filters, and of n / 2.
    CUtensorMap w16[2], w32[2];
};

// Tile load of three dimensions into THIS CTA's shared memory whose bytes are counted on a barrier of this CTA or the leader.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst_smem, const void *map, uint32_t cluster_bar, int32_t c0, int32_t c1, int32_t c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];"
        :
        : "r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// The work of a pair, in the order that all its roles walk it: items (filter tile, pair of pixel tiles), each in one form or in
// both.  The scales of the images that say which are fetched an item ahead.
struct HaloWalk {
    const ConvHaloParams &p;
    int item, stride, form;
    int tn, tile[2], img[2];
    bool wide[2];
    float scale[2], next[2];

    __device__ __forceinline__ void fetch(int it) {
        if (it < p.items) {
            const int u = it - fast_div(it, p.by_pairs) * p.pairs;
#pragma unroll
            for (int r = 0; r < 2; ++r)
                next[r] = p.image_scale[fast_div(min(2 * u + r, p.total_tiles - 1), p.by_tiles)];
        }
    }
    __device__ __forceinline__ HaloWalk(const ConvHaloParams &params, int first, int step) : p(params), item(first - step), stride(step), form(1) {
        wide[0] = wide[1] = false;
        fetch(first);
    }
    // the next pass; false: none
    __device__ __forceinline__ bool advance() {
        if (form == 0 && (wide[0] || wide[1])) {
            form = 1;
            return true;
        }
        item += stride;
        if (item >= p.items)
            return false;
        tn          = fast_div(item, p.by_pairs);
        const int u = item - tn * p.pairs;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            tile[r] = min(2 * u + r, p.total_tiles - 1);
            img[r]  = fast_div(tile[r], p.by_tiles);
            scale[r] = next[r];
            wide[r]  = __any_sync(0xffffffffu, next[r] == 0.0f) != 0; // the same for all lanes, and known to be
        }
        form = wide[0] && wide[1] ? 1 : 0;
        fetch(item + stride);
        return true;
    }
    __device__ __forceinline__ int cblocks() const { return p.c_pad >> (form ? 4 : 5); }
    __device__ __forceinline__ int chunk() const { return form ? p.chunk_wide : p.chunk_blocks; }
    __device__ __forceinline__ int block(int b) const { return p.last_first ? cblocks() - 1 - b : b; }
    // Filter k-blocks come in sets of c_pad / 32 channel blocks (two to a tf32 pass); -1: not the first block of one
    __device__ __forceinline__ int set_of(int b) const {
        const int each = p.c_pad >> 5;
        return b == 0 ? tn * 3 + form : (b == each ? tn * 3 + 2 : -1);
    }
};

template <bool THREE, bool RING>
__global__ void __launch_bounds__(kH_Threads, 1) conv_halo_stream_kernel(
    const __grid_constant__ ConvHaloMaps maps, const __grid_constant__ ConvHaloParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_f_full[kH_MaxSlots], bar_f_empty[kH_MaxSlots], bar_reload;
    __shared__ uint64_t bar_h_full[kH_HaloStages], bar_h_empty[kH_HaloStages];
    __shared__ uint64_t bar_acc_full[2], bar_acc_empty[2];
    __shared__ uint32_t halo_word[kH_HaloStages];
    __shared__ int epi_word[2];
    __shared__ uint64_t bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s;
    // scales and bias of the filters of an epilogue warp: from global memory, between the stores, they cost more than the stores
    __shared__ __align__(16) float scale_s[kH_EpiWarps][32], bias_s[kH_EpiWarps][32];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); // known to be the same for the warp
    const int lane = threadIdx.x & 31;
    const int rank = (int)(blockIdx.x & 1); // in the cluster of two

    griddep_launch_dependents();
    const uint32_t smem_base  = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t halo_stage = 2u * (uint32_t)p.halo_plane_bytes;
    const uint32_t slot_base  = smem_base + (uint32_t)p.halo_stages * halo_stage;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.slots; ++s) {
            mbar_init(smem_u32(&bar_f_full[s]), 1);
            mbar_init(smem_u32(&bar_f_empty[s]), 1);
        }
        for (int s = 0; s < p.halo_stages; ++s) {
            mbar_init(smem_u32(&bar_h_full[s]), 1);
            mbar_init(smem_u32(&bar_h_empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), 2 * kH_EpiWarps); // both CTAs'
        }
        mbar_init(smem_u32(&bar_reload), 1);
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        prefetch_tensormap(&maps.x16_hi);
        prefetch_tensormap(&maps.x16_lo);
        prefetch_tensormap(&maps.w16[0]);
        prefetch_tensormap(&maps.w16[1]);
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish_pair();
    }
    griddep_wait(); // the planes, the scales and what the caller's earlier kernels wrote
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync(); // the partner's barriers exist before anything is signalled on them
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    const bool failed        = abort_flag_s != 0; // an earlier launch failed: no work
    __syncthreads(); // every thread has read abort_flag_s before a role may raise it
    const int first = (int)(blockIdx.x >> 1), stride = (int)(gridDim.x >> 1);

    if (failed) {
    } else if (warp == 0) {
        // ===== TMA producer: this CTA's halos and its share of the filters, counted on the leader's barriers =====
        int ka = 0, s = 0, kh2 = 0, hs = 0, held = -1, sets = 0; // filter k-blocks, halos and sets of filters issued so far
        uint32_t f_phase = 1, h_phase = 1;
        bool ok = true;
        HaloWalk walk(p, first, stride);
        while (ok && walk.advance()) {
            const CUtensorMap *x_hi = walk.form ? &maps.x32_hi : &maps.x16_hi, *x_lo = walk.form ? &maps.x32_lo : &maps.x16_lo;
            const CUtensorMap *w    = walk.form ? maps.w32 : maps.w16;
            const int block_k       = walk.form ? 16 : 32; // channels per k-block
            const int img  = rank ? walk.img[1] : walk.img[0], tile = rank ? walk.tile[1] : walk.tile[0];
            const int at   = (tile - img * p.image_tiles) * 128, cblocks = walk.cblocks();
            const int chunk = walk.chunk();
            bool load       = true;
            int in_chunk    = 0;
            for (int b = 0; b < cblocks && ok; ++b) {
                const int c0  = walk.block(b) * block_k;
                uint32_t word = walk.form ? kH_Wide | kH_Two : (p.c - c0 > 16 ? kH_Two : 0u); // k-steps that hold channels
                bool reload   = false;
                if (!RING) {
                    const int set = walk.set_of(b);
                    if (set >= 0) {
                        load   = set != held;
                        held   = set;
                        reload = load && sets++ > 0;
                        word |= kH_Set | (reload ? kH_Reload : 0u);
                    }
                }
                word |= (load ? kH_Load : 0u) | (in_chunk == 0 ? kH_Begin : 0u);
                const bool last = ++in_chunk == chunk || b + 1 == cblocks;
                if (last)
                    in_chunk = 0;
                for (int h = 0; h < p.halos && ok; ++h) {
                    ok = mbar_wait_patient_warp(smem_u32(&bar_h_empty[hs]), h_phase, abort_flag);
                    if (!ok)
                        break;
                    if (elect_one()) {
                        const uint32_t full = smem_u32(&bar_h_full[hs]), dst = smem_base + (uint32_t)hs * halo_stage;
                        if (rank == 0) {
                            halo_word[hs] = word | (uint32_t)p.halo_taps[h] | (uint32_t)p.halo_taps[h + 1] << 6 |
                                            (last && h + 1 == p.halos ? kH_End : 0u);
                            mbar_expect_tx(full, 2u * 2u * (uint32_t)(p.boxes * p.box_rows * kH_RowB));
                        }
                        for (int x = 0; x < p.boxes; ++x) {
                            const uint32_t off = (uint32_t)(x * p.box_rows * kH_RowB);
                            tma_load_3d_pair(dst + off, x_hi, leader_addr(full), c0, p.halo_at[h] + at + x * p.box_rows, img);
                            tma_load_3d_pair(dst + (uint32_t)p.halo_plane_bytes + off, x_lo, leader_addr(full), c0,
                                             p.halo_at[h] + at + x * p.box_rows, img);
                        }
                    }
                    __syncwarp();
                    ++kh2;
                    if (++hs == p.halo_stages)
                        hs = 0, h_phase ^= 1u;
                    word &= ~(kH_Begin | kH_Set | kH_Reload);
                    if (reload) // everything that read the last set has retired; the issuer has been told to say so
                        ok = mbar_wait_patient_warp(smem_u32(&bar_reload), (uint32_t)sets & 1u, abort_flag);
                    reload = false;
                    if (!ok)
                        break;
                    for (int t = p.halo_taps[h]; (RING || load) && t < p.halo_taps[h + 1]; t += RING ? p.group : 1) {
                        if (RING) {
                            ok = mbar_wait_patient_warp(smem_u32(&bar_f_empty[s]), f_phase, abort_flag);
                            if (!ok)
                                break;
                        }
                        if (elect_one()) {
                            const uint32_t full = smem_u32(&bar_f_full[s]), dst = slot_base + (uint32_t)(s * p.slot_bytes);
                            if (rank == 0)
                                mbar_expect_tx(full, 2u * (uint32_t)p.slot_bytes);
                            const int32_t cb = walk.block(b), row = walk.tn * p.n, half = row + rank * (p.n >> 1);
                            // (a group's box may run on past its halo's taps: what it then holds is not used)
                            if (THREE) {
                                tma_load_5d_pair(dst, &w[0], leader_addr(full), 0, half, t, cb, 0);
                            } else {
                                tma_load_5d_pair(dst, &w[0], leader_addr(full), 0, row, t, cb, rank);
                                tma_load_5d_pair(dst + (uint32_t)p.f1, &w[1], leader_addr(full), 0, half, t, cb, 0);
                            }
                        }
                        __syncwarp();
                        ++ka;
                        if (++s == p.slots)
                            s = 0, f_phase ^= 1u;
                    }
                }
            }
        }
        if (ok && rank == 0) {
            ok = mbar_wait_patient_warp(smem_u32(&bar_h_empty[hs]), h_phase, abort_flag);
            if (ok && elect_one()) {
                halo_word[hs] = kH_Over;
                mbar_arrive(smem_u32(&bar_h_full[hs]));
            }
            __syncwarp();
        }
        if (*abort_flag && rank == 0) {
            // unwind: let the copies still in flight land before the CTA goes away (the leader's barriers
            // count the partner's copies too, and neither CTA leaves before the other)
            for (int k2 = ka - p.slots < 0 ? 0 : ka - p.slots; k2 < ka; ++k2) {
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_f_full[k2 % p.slots]), (uint32_t)(k2 / p.slots) & 1u) &&
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
    } else if (warp == 1) {
        // ===== MMA issuer: the leader's, for the pair =====
        if (rank == 0) {
            // What a pass is made of is worked out by the producer (2400 clocks a pass here, while the tensor pipe ran dry), and
            // of a descriptor only the low word, the address, is computed.
            const uint32_t slot_step = (uint32_t)p.slot_bytes >> 4, tap_step = (uint32_t)p.tap_bytes >> 4, to_f1 = (uint32_t)p.f1 >> 4;
            const uint32_t q_step    = THREE ? tap_step : tap_step >> 1; // of the second operand's terms
            const uint32_t f_0       = (uint32_t)smem_desc_k<kH_RowB>(slot_base);
            const uint32_t to_lo     = (uint32_t)p.halo_plane_bytes >> 4;
            auto desc = [](uint32_t low) { return smem_desc_k<kH_RowB>(0) & 0xffffffff00000000ull | low; };
            int s = 0, hs = 0, acc = 0;
            uint32_t f_phase = 0, h_phase = 0, acc_phase = 3u; // a bit per set of accumulators
            uint32_t d_main = 0, d_cross = 0, f = f_0;
            bool ok = true;
            while (ok) {
                ok = mbar_wait_warp(smem_u32(&bar_h_full[hs]), h_phase, abort_flag);
                if (!ok)
                    break;
                tc_fence_after_sync();
                const uint32_t word = __shfl_sync(0xffffffffu, *const_cast<volatile uint32_t *>(&halo_word[hs]), 0);
                if (word & kH_Over)
                    break;
                if (word & kH_Reload)
                    tc_commit_warp(smem_u32(&bar_reload));
                if (word & kH_Set)
                    s = 0, f = f_0;
                uint32_t accumulate = 1u;
                if (word & kH_Begin) { // what the accumulators held before has been read
                    ok = mbar_wait_warp<kClusterRead>(smem_u32(&bar_acc_empty[acc]), acc_phase >> acc & 1u, abort_flag);
                    if (!ok)
                        break;
                    tc_fence_after_sync();
                    acc_phase ^= 1u << acc;
                    d_main = tmem_base + (uint32_t)(acc * 256), d_cross = d_main + (uint32_t)p.n;
                    accumulate = 0u;
                }
                const uint32_t idesc = make_idesc(word & kH_Wide ? 2u : 0u, 256, (uint32_t)p.n);
                const uint32_t idesc2 = make_idesc(word & kH_Wide ? 2u : 0u, 256, (uint32_t)(2 * p.n));
                const uint32_t x = (uint32_t)smem_desc_k<kH_RowB>(smem_base + (uint32_t)hs * halo_stage);
                const int t1 = (int)(word >> 6 & 63u);
                int in_group = 0;
                uint32_t f0 = f, f1 = f + to_f1;
                for (int t = (int)(word & 63u); t < t1; ++t) {
                    if (!RING || in_group == 0) {
                        f0 = f, f1 = f + to_f1;
                        if (RING || (word & kH_Load)) {
                            ok = mbar_wait_warp(smem_u32(&bar_f_full[s]), f_phase, abort_flag);
                            if (!ok)
                                break;
                            tc_fence_after_sync();
                        }
                    }
                    // the tap's pixels: the halo, so many rows of 64 bytes further on
                    const uint32_t xh = x + p.tap_shift[t], xl = xh + to_lo;
                    auto issue = [&](auto mma, uint32_t k) {
                        if (THREE) {
                            mma(d_main, desc(xh + k), desc(f0 + k), idesc, accumulate);
                            mma(d_cross, desc(xh + k), desc(f1 + k), idesc, accumulate);
                            mma(d_cross, desc(xl + k), desc(f0 + k), idesc, 1u);
                        } else {
                            mma(d_main, desc(xh + k), desc(f0 + k), idesc2, accumulate);
                            mma(d_cross, desc(xl + k), desc(f1 + k), idesc, 1u);
                        }
                        accumulate = 1u;
                    };
                    if (!(word & kH_Wide)) {
                        issue(mma_f16_warp<2>, 0);
                        if (word & kH_Two)
                            issue(mma_f16_warp<2>, 2);
                    } else {
                        issue(mma_tf32_pair_warp, 0);
                        issue(mma_tf32_pair_warp, 2);
                    }
                    bool next = true; // group
                    if (RING) {
                        f0 += tap_step, f1 += q_step;
                        next = ++in_group == p.group || t + 1 == t1;
                    }
                    if (next) {
                        if (RING) {
                            in_group = 0;
                            tc_commit_warp(smem_u32(&bar_f_empty[s]));
                        }
                        f += slot_step;
                        if (++s == p.slots) {
                            s = 0, f = f_0;
                            if (RING || (word & kH_Load))
                                f_phase ^= 1u;
                        }
                    }
                }
                if (!ok)
                    break;
                tc_commit_warp(smem_u32(&bar_h_empty[hs])); // the halo is free once its taps' MMAs have retired
                if (++hs == p.halo_stages)
                    hs = 0, h_phase ^= 1u;
                if (word & kH_End) {
                    tc_commit_warp(smem_u32(&bar_acc_full[acc]));
                    acc ^= 1;
                }
            }
            if (!ok || *abort_flag) {
                // unwind: wait until every MMA issued so far has retired
                __syncwarp();
                tc_commit_warp(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else {
        // ===== epilogue: a lane has a position, a warp a quarter of the channels =====
        const int quarter = warp & 3; // TMEM lanes this warp may read: 32 * quarter ..
        const int share   = (warp - 2) >> 2, each = p.n >> 2, groups = p.n >> 5; // its channels, and groups of eight of them
        const bool relu   = p.act == CT_ACT_RELU;
        const int64_t plane = (int64_t)p.ho * p.wo;
        float *scales = scale_s[warp - 2], *biases = bias_s[warp - 2];
        int acc = 0, held = -1, turn = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        HaloWalk walk(p, first, stride);
        while (ok && walk.advance()) {
            const bool wide    = walk.form != 0;
            const float weight = wide ? 1.0f : kHalfLoInv;
            const int img = rank ? walk.img[1] : walk.img[0], tile = rank ? walk.tile[1] : walk.tile[0];
            // stored in the form that its image has, and once: the last tile of an odd number has no partner
            const bool store = (rank ? walk.wide[1] : walk.wide[0]) == wide && !(rank && walk.tile[0] == walk.tile[1]);
            const float inv  = rank ? walk.scale[1] : walk.scale[0];
            const int q = (tile - img * p.image_tiles) * 128 + quarter * 32 + lane, y = fast_div(q, p.by_pw), x = q - y * p.pw;
            const int ch0 = walk.tn * p.n + share * each, chunks = wide ? p.chunks_wide : p.chunks;
            if (walk.tn != held) {
                held = walk.tn;
                __syncwarp();
                if (lane < each)
                    scales[lane] = p.filter_scale[ch0 + lane], biases[lane] = p.bias[ch0 + lane];
                __syncwarp();
            }
            float sum[32];
#pragma unroll 1
            for (int e = 0; e < chunks; ++e) {
                ok = group_wait(
                    warp == 2, [&] { return mbar_wait(smem_u32(&bar_acc_full[acc]), acc_phase >> acc & 1u, abort_flag); }, epi_word, turn++, 1,
                    32 * kH_EpiWarps);
                if (!ok)
                    break;
                acc_phase ^= 1u << acc;
                tc_fence_after_sync();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 256 + share * each);
                auto take = [&](int at, uint32_t main, uint32_t cross) {
                    const float v = __fadd_rn(__uint_as_float(main), __fmul_rn(__uint_as_float(cross), weight));
                    sum[at]       = e == 0 ? v : __fadd_rn(sum[at], v);
                };
#pragma unroll
                for (int g = 0; g < 4; g += 2) {
                    if (groups >= g + 2) {
                        uint32_t m[16], c[16];
                        tmem_ld_32x16(taddr + (uint32_t)(8 * g), m);
                        tmem_ld_32x16(taddr + (uint32_t)(p.n + 8 * g), c);
                        tmem_ld_wait();
#pragma unroll
                        for (int u = 0; u < 16; ++u)
                            take(8 * g + u, m[u], c[u]);
                    } else if (groups == g + 1) {
                        uint32_t m[8], c[8];
                        tmem_ld_32x8(taddr + (uint32_t)(8 * g), m);
                        tmem_ld_32x8(taddr + (uint32_t)(p.n + 8 * g), c);
                        tmem_ld_wait();
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            take(8 * g + u, m[u], c[u]);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive_peer_read(leader_addr(smem_u32(&bar_acc_empty[acc])));
                acc ^= 1;
            }
            if (!ok)
                break;
            if (store) {
                const bool live = x < p.wo && y < p.ho;
                float *at       = p.out + ((int64_t)img * p.ko + ch0) * plane + (int64_t)y * p.wo + x;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (g < groups && ch0 + 8 * g < p.ko) {
                        float fs[8], bs[8];
#pragma unroll
                        for (int u = 0; u < 8; u += 4) {
                            *reinterpret_cast<float4 *>(fs + u) = *reinterpret_cast<const float4 *>(scales + 8 * g + u);
                            *reinterpret_cast<float4 *>(bs + u) = *reinterpret_cast<const float4 *>(biases + 8 * g + u);
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u, at += plane) {
                            const float scale = wide ? 1.0f : __fmul_rn(fs[u], inv); // powers of two
                            float v = __fadd_rn(__fmul_rn(sum[8 * g + u], scale), bs[u]);
                            v       = !relu || v > 0.0f ? v : __fmul_rn(v, 0.0f);
                            if (live && ch0 + 8 * g + u < p.ko)
                                *at = v;
                        }
                    }
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    cluster_sync(); // neither CTA goes while the other's MMAs, copies or arrivals may still reach it
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
    if (threadIdx.x == 0 && !failed && *abort_flag)
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

// ---- pre-pass -----------------------------------------------------------------------------
//
// Two launches: the range of every image, in slices, next to the filters (both forms of their planes, a block per
// filter); then the input as NHWC planes, in the form that the image's range allows.

// Blocks 0 .. ko - 1: filter [c][taps] -> planes [taps in the order given][c_pad] (none if hi16 is null), and its inverse
// scale, 0 where the range of the filter does not fit float16 pairs.  The others: slice (blockIdx.x - ko) of the images
// ([batch][count] floats, `slices` to an image).
struct FilterPlanes {
    __half *hi16, *lo16;
    float *hi32, *lo32;
    float *scale;
    uint8_t order[kH_MaxTaps]; // place of each tap in the planes
    const float *bias; // the layer's, or null
    float *bias_out;   // its copy, -0 where there is none; null: not wanted
};
__global__ void __launch_bounds__(256) conv_range_kernel(
    const float *__restrict__ w, int c, int taps, int c_pad, int ko, const __grid_constant__ FilterPlanes f, const float *__restrict__ x,
    int64_t count, int slices, int vec_ok, uint2 *__restrict__ ranges) {
    __shared__ uint2 part[8];
    griddep_launch_dependents();
    griddep_wait();
    const bool filter = (int64_t)blockIdx.x < ko;
    const int64_t o   = filter ? blockIdx.x : (blockIdx.x - ko) / slices;
    const int slice   = filter ? 0 : (int)(blockIdx.x - ko - o * slices);
    const float *src  = filter ? w + o * c * taps : x + o * count;
    const int64_t n   = filter ? (int64_t)c * taps : count;
    const int step    = filter ? 256 : slices * 256;
    uint2 r            = make_uint2(0u, kNoneSmallest);
    // Eight loads in flight, also where fewer are left (zeros are not noticed): as a loop that was only to be unrolled they came one by one, 3 x
    // 31 x 30 x 29 4.2 us, so 3.3, 32 x 64 x 56 x 56 8.9 and 7.0, 73 x 122 x 47 x 47 27.8 and 23.7 (each load with a condition of its own 29.8).
    auto walk = [&](auto zero, auto take) {
        using V      = decltype(zero);
        const V *at  = reinterpret_cast<const V *>(src) + (int64_t)slice * 256 + threadIdx.x;
        const V *end = reinterpret_cast<const V *>(src) + n / (int64_t)(sizeof(V) / 4);
        for (; at + 7 * step < end; at += 8 * step) {
            V q[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                q[u] = at[u * step];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                take(q[u]);
        }
        if (at < end) {
            V q[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                q[u] = at + u * step < end ? at[u * step] : zero;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                take(q[u]);
        }
    };
    if (!filter && vec_ok)
        walk(make_float4(0.0f, 0.0f, 0.0f, 0.0f), [&](const float4 &q) { range_take(r, q.x), range_take(r, q.y), range_take(r, q.z), range_take(r, q.w); });
    else
        walk(0.0f, [&](float q) { range_take(r, q); });
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
    if (threadIdx.x == 0) {
        f.scale[o] = fits ? inverse : 0.0f;
        if (f.bias_out)
            f.bias_out[o] = f.bias ? f.bias[o] : -0.0f;
    }
    if (f.hi16 == nullptr)
        return;
    for (int i = threadIdx.x; i < taps * c_pad; i += 256) {
        const int tap = i / c_pad, ic = i - tap * c_pad;
        const float v    = ic < c ? src[ic * taps + tap] : 0.0f;
        const int64_t at = (o * taps + f.order[tap]) * c_pad + ic;
        split_half(v, scale, f.hi16[at], f.lo16[at]);
        split_tf32(v, f.hi32[at], f.lo32[at]);
    }
}

// x [batch][c][hw] -> NHWC planes [position][c_pad], hi then lo, in the image's slot of 8 bytes per value: float16 pairs
// under the image's scale, or tf32 terms (image_scale 0) where the image or any filter does not fit those.  Positions are those of the
// sub-images (ConvSubImages, hs x ws each, from row y0 and column x0 of the input on): zeros where the image has no such row or
// column, which is a layer's padding; those that no tap reads are left out.  The images are taken last to first: the end of the tensor
// is what conv_range_kernel has just left in L2.
//
// A warp takes 32 channels of 32 pixels, a pixel to a lane, all loads in flight at once: what a lane has split are then whole
// 16-byte pieces of the planes, and its own shared memory only brings them into an order in which four lanes write 64 contiguous bytes.  No barrier
// but the one behind which the block knows its image's form: blocks of 64 channels by 64 pixels, with barriers between reading and
// writing, took 96 us for 256 x 64 x 56 x 56 where this takes 81 (of 55 to 65 at the copy rate; without loads and stores 40: a block's wait for
// its image's range and its own start), and 22 for 64 x 48 x 57 x 57 at stride 2, where this takes 18.
struct PlaneGeom {
    int h, w, hs, ws, y0, x0;
    ConvSubImages sub;
    int groups, items; // groups of 32 channels; warps' shares of an image
    FastDiv by_w, by_groups, by_cols, by_chunks, by_pad; // image width, groups, columns of the grown image, eights of channels, padding columns
    int pad_top, pad_rows, mid_rows, pad_left, pad_cols; // the grown image's positions that no pixel has: rows above, all such rows ...
};
template <int ROW_MOD, int COL_MOD>
__global__ void __launch_bounds__(256, 3) conv_planes_kernel(
    const float *__restrict__ x, int c, const __grid_constant__ PlaneGeom g, int c_pad, const uint2 *__restrict__ ranges, int slices,
    const float *__restrict__ filter_scale, int ko, uint8_t *__restrict__ slots, float *__restrict__ image_scale) {
    __shared__ uint4 stage_s[8][128];
    __shared__ float scale_s;
    griddep_launch_dependents();
    griddep_wait();
    const int img  = (int)(gridDim.y - 1 - blockIdx.y);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int item = (int)blockIdx.x * 8 + warp, hw = g.h * g.w;
    const int px_tile = fast_div(item, g.by_groups), c0 = (item - px_tile * g.groups) * 32;
    const int q = px_tile * 32 + lane;
    const bool live  = item < g.items && q < hw;
    const float *src = x + ((int64_t)img * c + c0) * hw + q;
    float v[32]; // every load before the first use of any
    // (the address goes from channel to channel in two instructions; left to the compiler, each was worked out anew, in seven)
    auto channel = [&]() {
        const float value = __ldcs(src);
        asm volatile("add.s64 %0, %0, %1;" : "+l"(src) : "l"((int64_t)hw * 4));
        return value;
    };
    if (live && c0 + 32 <= c) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            v[j] = channel();
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            v[j] = live && c0 + j < c ? channel() : 0.0f;
    }
    if (warp == 0) {
        uint2 r = make_uint2(0u, kNoneSmallest);
        for (int s = lane; s < slices; s += 32)
            r = range_join(r, ranges[(int64_t)img * slices + s]);
        float scale, inverse;
        const bool all = half_range_fits(range_warp(r), scale, inverse);
        if (lane == 0)
            scale_s = all ? scale : 0.0f;
    }
    int bad_filter = 0;
    for (int o = threadIdx.x; o < ko; o += 256)
        bad_filter |= filter_scale[o] == 0.0f ? 1 : 0;
    const bool filters_fit = !__syncthreads_or(bad_filter);
    const float scale      = filters_fit ? scale_s : 0.0f;
    const bool fits        = scale != 0.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        image_scale[img] = fits ? 1.0f / scale : 0.0f; // a power of two
    const int rows = g.hs * ROW_MOD, cols = g.ws * COL_MOD;
    const bool plain    = !fits && g.sub.tf32_plain;
    const int64_t plane = (int64_t)__popc(g.sub.used) * g.hs * g.ws * c_pad;
    uint8_t *slot       = slots + (int64_t)img * plane * 8;
    auto place = [&](int row, int col) { // of the grown image; -1: not wanted
        if (ROW_MOD * COL_MOD == 1)
            return row * cols + col;
        const int sub = row % ROW_MOD * COL_MOD + col % COL_MOD;
        return g.sub.used >> sub & 1u ? (__popc(g.sub.used & ((1u << sub) - 1u)) * g.hs + row / ROW_MOD) * g.ws + col / COL_MOD : -1;
    };
    int to = -1;
    if (live) {
        const int y = fast_div(q, g.by_w), row = y - g.y0, col = q - y * g.w - g.x0;
        to = plain ? q : ((unsigned)row < (unsigned)rows && (unsigned)col < (unsigned)cols ? place(row, col) : -1);
    }
    // 64 bytes of each lane's pixel to `dst`, pixels `stride` bytes apart: chunk j of pixel p lies at j ^ ((p >> 1) & 3)
    uint4 *stage = stage_s[warp];
    auto emit = [&](const uint4 (&piece)[4], uint8_t *dst, int stride) {
        __syncwarp(); // the last one's have been read
#pragma unroll
        for (int j = 0; j < 4; ++j)
            stage[lane * 4 + (j ^ (lane >> 1 & 3))] = piece[j];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int p = 8 * k + (lane >> 2), j = lane & 3, at = __shfl_sync(0xffffffffu, to, p);
            if (at >= 0)
                *reinterpret_cast<uint4 *>(dst + (int64_t)at * stride + 16 * j) = stage[p * 4 + (j ^ (p >> 1 & 3))];
        }
    };
    if (item < g.items) {
        if (fits) {
            uint4 hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                __half2 h[4], l[4];
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    split_half_pair(__fmul_rn(v[8 * j + 2 * t], scale), __fmul_rn(v[8 * j + 2 * t + 1], scale), h[t], l[t]);
                hi[j] = *reinterpret_cast<uint4 *>(h), lo[j] = *reinterpret_cast<uint4 *>(l);
            }
            emit(hi, slot + c0 * 2, c_pad * 2);
            emit(lo, slot + plane * 2 + c0 * 2, c_pad * 2);
        } else {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint4 hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float h[4], l[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        split_tf32_flat(v[16 * half + 4 * j + t], h[t], l[t]);
                    hi[j] = *reinterpret_cast<uint4 *>(h), lo[j] = *reinterpret_cast<uint4 *>(l);
                }
                emit(hi, slot + (c0 + 16 * half) * 4, c_pad * 4);
                emit(lo, slot + plane * 4 + (c0 + 16 * half) * 4, c_pad * 4);
            }
        }
    }
    // positions that no pixel has: the layer's padding, shared out between the blocks of the image
    if (!plain) {
        const int chunks = c_pad >> 3, whole = g.pad_rows * cols, all = (whole + g.mid_rows * g.pad_cols) * chunks;
        for (int i = (int)blockIdx.x * 256 + (int)threadIdx.x; i < all; i += (int)gridDim.x * 256) {
            const int j = fast_div(i, g.by_chunks), chunk = i - j * chunks;
            int row, col;
            if (j < whole) {
                row = fast_div(j, g.by_cols), col = j - row * cols;
                row += row < g.pad_top ? 0 : g.mid_rows;
            } else {
                row = fast_div(j - whole, g.by_pad), col = j - whole - row * g.pad_cols;
                row += g.pad_top, col += col < g.pad_left ? 0 : cols - g.pad_cols;
            }
            const int at = place(row, col);
            if (at >= 0) {
                const int size = fits ? 16 : 32; // bytes of eight channels
                for (int b = 0; b < size; b += 16) {
                    uint8_t *dst = slot + ((int64_t)at * chunks + chunk) * size + b;
                    *reinterpret_cast<uint4 *>(dst)                              = make_uint4(0u, 0u, 0u, 0u);
                    *reinterpret_cast<uint4 *>(dst + plane * (fits ? 2 : 4)) = make_uint4(0u, 0u, 0u, 0u);
                }
            }
        }
    }
}

struct HaloGeom {
    int pw, wo, ho;
    int hs;             // rows of a sub-image; it has pw columns
    int y_min, x_min;   // smallest row and column offset of a tap in its sub-image
    int image_tiles, box_rows, boxes, plane_bytes, stages;
    int n, tiles_n, group, slots, slot_bytes, ring, three;
    size_t smem;
};

int floor_div(int64_t a, int64_t b) { return (int)(a >= 0 ? a / b : -((-a + b - 1) / b)); }

// Tap (r, q) of output (oy, ox) reads input row oy * stride - pad + r = stride * (oy + a) + py: row oy + a of the
// sub-image py, and so for columns.  The planes hold rows y_min .. of each sub-image and pw = wo + (largest - smallest b)
// columns from x_min on.
bool halo_geometry(int64_t c_pad, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride, int64_t pad, HaloGeom *g) {
    if (w + 2 * pad < kw || h + 2 * pad < kh || pad > 256 || kh > 256 || kw > 256)
        return false;
    const int64_t wo = (w + 2 * pad - kw) / stride + 1, ho = (h + 2 * pad - kh) / stride + 1;
    g->y_min = floor_div(-pad, stride), g->x_min = floor_div(-pad, stride);
    const int64_t span_y = floor_div(kh - 1 - pad, stride) - g->y_min, span_x = floor_div(kw - 1 - pad, stride) - g->x_min;
    const int64_t pw = wo + span_x;
    if (pw > 256) // as measured so far; nothing in the kernel needs it
        return false;
    g->pw = (int)pw, g->wo = (int)wo, g->ho = (int)ho, g->hs = (int)(ho + span_y);
    g->image_tiles = (int)((ho * pw + 127) / 128);
    // a halo: the tile's positions and those that its last one's taps reach, in boxes of whole swizzle atoms
    const int64_t rows = 128 + span_y * pw + span_x;
    g->boxes       = (int)((rows + 255) / 256);
    g->box_rows    = (int)(((rows + g->boxes - 1) / g->boxes + 7) / 8 * 8);
    g->plane_bytes = (g->boxes * g->box_rows * kH_RowB + 1023) & ~1023;
    // tiles of equal numbers of filters, in steps of 32 (the columns of an MMA of two CTAs)
    g->tiles_n    = (int)((ko + 127) / 128);
    g->n          = (int)(((ko + g->tiles_n - 1) / g->tiles_n + 31) / 32 * 32);
    const int budget = kH_Smem - 1024, halo = 2 * g->plane_bytes;
    // All filters of a tile, by halves (see the top) for many, and where the other way's memory does not hold them all.
    const int64_t all = kh * kw * (c_pad / 32);
    const int one = g->n * kH_RowB, both = one / 2 * 3;
    auto fits     = [&](int64_t bytes) { return all <= kH_MaxSlots && all * bytes + 2 * halo <= budget; };
    g->three      = g->n >= 96 || !fits(both);
    g->group      = 1;
    g->slot_bytes = g->three ? one : both;
    g->ring       = !fits(g->slot_bytes);
    if (!g->ring) {
        g->slots  = (int)all;
        g->stages = std::min(kH_HaloStages, (budget - g->slots * g->slot_bytes) / halo);
    } else {
        // In a ring, groups of taps, a row of them where a halo serves whole rows: with a tap by itself copies, waits and commits took 700
        // clocks, where those of 64 filters take 290 (40 x 100 x 50 x 50 -> 64, 5 x 5, 207 us, 168 so).  Room for three slots beside two halos is enough for that (12 x
        // 151 x 46 x 46 -> 115, 5 x 5, 116 us by single taps, 94 so).  Where a row is too much or the halos of a strided layer have parts of rows, by threes, from
        // 16 taps on (20 x 107 x 58 x 58 -> 108, 5 x 5 at stride 2, 104 and 88; nine taps lose by what the boxes bring for nothing, 43 x 200 x 45 x
        // 47 -> 67, 3 x 3, 102 and 110).  A third halo where that leaves 64 KB and two slots.
        const int row = stride == 1 && 2 * halo + 3 * kw * one <= budget ? (int)kw : (kh * kw >= 16 && 2 * halo + 3 * 3 * one <= budget ? 3 : 1);
        g->group      = row, g->slot_bytes *= row;
        g->stages = 3 * halo + std::max(64 * 1024, 2 * g->slot_bytes) <= budget ? 3 : 2;
        g->slots  = (int)std::min<int64_t>(std::min<int64_t>(16, all / g->group), (budget - g->stages * halo) / g->slot_bytes);
        if (budget < g->stages * halo || g->slots < std::min<int64_t>(g->group > 1 ? 2 : 4, all / g->group))
            return false;
    }
    g->smem = 1024 + (size_t)g->stages * halo + (size_t)g->slots * g->slot_bytes;
    return true;
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
    const float *x, const float *w, int64_t batch, int64_t c, int64_t h, int64_t wd, int64_t c_pad, int64_t ko, int64_t taps,
    void *filters16, void *filters32, size_t plane16, size_t plane32, const uint8_t *order, float *filter_scale, const float *bias, float *bias_copy,
    void *ranges, float *image_scale, void *slots, const ConvSubImages &sub) {
    if (batch > 65535)
        return fail(CT_ERR_TOO_LARGE, "conv2d: batch too large for the layout pre-pass");
    const int64_t count = c * h * wd;
    const int slices    = conv_range_slices(batch, count);
    const int vec       = (count & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    uint8_t *f16 = static_cast<uint8_t *>(filters16), *f32 = static_cast<uint8_t *>(filters32);
    FilterPlanes f{reinterpret_cast<__half *>(f16), reinterpret_cast<__half *>(f16 + plane16), reinterpret_cast<float *>(f32),
                   reinterpret_cast<float *>(f32 + plane32), filter_scale, {}, bias, bias_copy};
    for (int t = 0; order && t < (int)taps; ++t)
        f.order[t] = order[t];
    ProfScope prof("conv_prepass");
    CT_CUDA(launch_dependent(conv_range_kernel, dim3((unsigned)(ko + batch * slices)), dim3(256), 0, stream(), w, (int)c, (int)taps,
                             (int)c_pad, (int)ko, f, x, count, slices, vec, static_cast<uint2 *>(ranges)));
    CT_LAUNCH_CHECK("conv_range");
    const int64_t width = (int64_t)sub.cols * sub.col_mod, grown = (int64_t)sub.rows * sub.row_mod, hw = h * wd;
    if ((grown * width + 1) * (c_pad / 8) > 0x7fffffffll || (hw + 31) / 32 * (c_pad / 32) > 0x7ffffff0ll)
        return fail(CT_ERR_TOO_LARGE, "conv2d: image too large for the layout pre-pass");
    PlaneGeom geom{};
    geom.h = (int)h, geom.w = (int)wd, geom.hs = sub.rows, geom.ws = sub.cols, geom.y0 = sub.y0, geom.x0 = sub.x0, geom.sub = sub;
    geom.groups = (int)(c_pad / 32), geom.items = (int)((hw + 31) / 32) * geom.groups;
    const int64_t top = std::min<int64_t>(-geom.y0, grown), left = std::min<int64_t>(-geom.x0, width);
    geom.mid_rows = (int)std::min<int64_t>(h, grown - top), geom.pad_top = (int)top, geom.pad_rows = (int)grown - geom.mid_rows;
    geom.pad_left = (int)left, geom.pad_cols = (int)(width - std::min<int64_t>(wd, width - left));
    geom.by_w = fast_divisor(wd), geom.by_groups = fast_divisor(geom.groups), geom.by_cols = fast_divisor(width);
    geom.by_chunks = fast_divisor(c_pad / 8), geom.by_pad = fast_divisor(std::max(1, geom.pad_cols));
    const dim3 grid((unsigned)((geom.items + 7) / 8), (unsigned)batch);
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

// Whether the halo kernel takes this layer (float32 mode only): filters and strides within its tables, planes whose positions
// 32 bits count, and tiles that are reasonably full.
bool conv_halo_applicable(int64_t c_pad, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride,
                          int64_t pad) {
    HaloGeom g;
    if (stride < 1 || stride > kH_MaxStride || ko < kH_MinFilters || kh * kw > kH_MaxTaps || (c_pad % 32) != 0 ||
        c_pad > (1 << 20) || h > 0x3fff || w > 0x3fff)
        return false;
    if (!halo_geometry(c_pad, h, w, ko, kh, kw, stride, pad, &g))
        return false;
    // measured down to 47 % of the rows with an output (256 x 64 x 11 x 11 -> 128 38 us, 73 through patches)
    return (int64_t)g.ho * g.wo * 100 >= (int64_t)g.image_tiles * 128 * 45;
}

// Workspace: [filter scale][bias][image scale][image ranges][w hi16][w lo16][w hi][w lo][image slots]; a slot holds an
// image's planes, float16 pairs or, where it does not fit those, tf32: no more than tf32 planes alone take.
ct_status conv_halo(
    DeviceState *st, const float *x, const float *w, int64_t batch, int64_t c, int64_t c_pad, int64_t h, int64_t wd, int64_t ko,
    int64_t kh, int64_t kw, int64_t stride, int64_t pad, const float *bias, int act, float *out) {
    HaloGeom g;
    if (!halo_geometry(c_pad, h, wd, ko, kh, kw, stride, pad, &g))
        return fail(CT_ERR_INVALID, "conv2d: internal tile shape not usable");
    auto align_up          = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    const int64_t taps = kh * kw, subs = stride * stride, sub = (int64_t)g.hs * g.pw;
    ConvHaloParams p;
    p.halos = 0, p.halo_taps[0] = 0;
    uint8_t order[kH_MaxTaps] = {};
    uint32_t used = 0;
    for (int image = 0, listed = 0; image < (int)subs; ++image) {
        for (int t = 0; t < (int)taps; ++t) {
            const int r = t / (int)kw - (int)pad, q = t % (int)kw - (int)pad, a = floor_div(r, stride), b = floor_div(q, stride);
            if ((r - a * (int)stride) * (int)stride + (q - b * (int)stride) != image)
                continue;
            order[t]              = (uint8_t)listed;
            p.tap_shift[listed++] = (uint16_t)(((a - g.y_min) * g.pw + (b - g.x_min)) * (kH_RowB / 16));
        }
        if (listed > p.halo_taps[p.halos]) { // the planes hold the sub-images that a tap reads, one behind the other
            p.halo_at[p.halos]     = (int)(p.halos * sub);
            p.halo_taps[++p.halos] = (uint8_t)listed;
            used |= 1u << image;
        }
    }
    const int64_t positions = sub * p.halos;
    const size_t slot       = (size_t)positions * c_pad * 8;
    // At most 4 GB of planes, one image at least: the batch goes in parts, which the images, each with a scale of its own, do not notice.
    const int64_t most = std::max<int64_t>(1, (int64_t)((4ull << 30) / slot));
    if (batch > most) {
        const int64_t parts = (batch + most - 1) / most, part = (batch + parts - 1) / parts;
        for (int64_t at = 0; at < batch; at += part)
            CT_TRY(conv_halo(st, x + at * c * h * wd, w, std::min(part, batch - at), c, c_pad, h, wd, ko, kh, kw, stride, pad, bias, act,
                             out + at * ko * g.ho * g.wo));
        return CT_OK;
    }
    const int64_t tiles    = g.image_tiles * batch, pairs = (tiles + 1) / 2, items = pairs * g.tiles_n;
    if (items > 0x3fffffffll || positions > 0x3fffffffll)
        return fail(CT_ERR_TOO_LARGE, "conv2d: too many tiles");
    const size_t w16       = align_up((size_t)ko * taps * c_pad * 2), w32 = align_up((size_t)ko * taps * c_pad * 4);
    const size_t w_words   = align_up((size_t)g.n * g.tiles_n * 4), x_words = align_up((size_t)batch * 4);
    const size_t ranges    = align_up((size_t)batch * conv_range_slices(batch, c * h * wd) * 8);
    CT_TRY(ensure_ws(&st->gemm_ws, &st->gemm_ws_bytes, 2 * w_words + x_words + ranges + 2 * w16 + 2 * w32 + (size_t)batch * slot));
    uint8_t *ws            = static_cast<uint8_t *>(st->gemm_ws);
    float *filter_scale    = reinterpret_cast<float *>(ws), *bias_copy = reinterpret_cast<float *>(ws + w_words);
    float *image_scale     = reinterpret_cast<float *>(ws + 2 * w_words);
    uint8_t *range_words   = ws + 2 * w_words + x_words;
    uint8_t *w16_hi        = range_words + ranges, *w32_hi = w16_hi + 2 * w16, *xp = w32_hi + 2 * w32;
    p.filter_scale = filter_scale, p.bias = bias_copy, p.image_scale = image_scale;
    p.out = out, p.flags = st->flags_dev;
    p.ko = (int)ko, p.n = g.n;
    p.ho = g.ho, p.wo = g.wo, p.pw = g.pw;
    p.image_tiles = g.image_tiles, p.total_tiles = (int)tiles, p.pairs = (int)pairs, p.items = (int)items;
    p.chunk_blocks = (int)std::max<int64_t>(1, kH_MaxK / (32 * taps));
    // a strided layer's tf32 images: no longer chains of truncating additions than the float16 ones have (3.0e-6 -> 3.7e-7 against
    // 64 bits at 48 channels, 3 x 3; all 64 images 110 -> 117 us); unstrided, with the cross products apart, 4.0e-6 -> 1.4e-6
    p.chunk_wide = stride > 1 ? 1 : 2 * p.chunk_blocks;
    p.chunks     = (int)(c_pad / 32 + p.chunk_blocks - 1) / p.chunk_blocks, p.chunks_wide = (int)(c_pad / 16 + p.chunk_wide - 1) / p.chunk_wide;
    p.c       = (int)c;
    p.last_first = c % 16 != 0;
    p.c_pad   = (int)c_pad;
    p.box_rows = g.box_rows, p.boxes = g.boxes;
    p.halo_plane_bytes = g.plane_bytes, p.halo_stages = g.stages;
    p.slots = g.slots, p.slot_bytes = g.slot_bytes;
    p.act = act;
    p.by_pairs = fast_divisor(pairs), p.by_tiles = fast_divisor(g.image_tiles), p.by_pw = fast_divisor(g.pw);
    p.group = g.group, p.tap_bytes = g.three ? g.n / 2 * kH_RowB : g.n * kH_RowB, p.f1 = g.group * p.tap_bytes;
    const ConvSubImages images{(int)stride, (int)stride, used, false, g.hs, g.pw, g.y_min * (int)stride, g.x_min * (int)stride};
    CT_TRY(conv_prepass(x, w, batch, c, h, wd, c_pad, ko, taps, w16_hi, w32_hi, w16, w32, order, filter_scale, bias, bias_copy, range_words,
                        image_scale, xp, images));
    ConvHaloMaps maps;
    const bool three = g.three != 0;
    auto encode = [&](CUtensorMap *mw, const uint8_t *wp, size_t w_plane, CUtensorMap *mx_hi, CUtensorMap *mx_lo, int elem) {
        const uint64_t row = (uint64_t)(c_pad * elem), block = (uint64_t)(kH_RowB / elem);
        // a filter's channels of a block, filters, taps, blocks, hi and lo terms
        const uint64_t wdims[5] = {block, (uint64_t)ko, (uint64_t)taps, (uint64_t)c_pad / block, 2};
        const uint64_t wstr[4]  = {(uint64_t)taps * row, row, (uint64_t)kH_RowB, (uint64_t)w_plane};
        const uint32_t wbox[2][5] = {{(uint32_t)block, (uint32_t)(three ? g.n / 2 : g.n), (uint32_t)g.group, 1, three ? 2u : 1u},
                                     {(uint32_t)block, (uint32_t)(g.n / 2), (uint32_t)g.group, 1, 1}};
        const uint64_t xdims[3] = {(uint64_t)c_pad, (uint64_t)positions, (uint64_t)batch}, xstr[2] = {row, slot};
        const uint32_t xbox[3]  = {(uint32_t)block, (uint32_t)g.box_rows, 1};
        auto fn = elem == 4 ? encode_tiled_map_f32 : encode_tiled_map_f16;
        for (int i = 0; i < 2; ++i)
            CT_TRY(fn(&mw[i], wp, 5, wdims, wstr, wbox[i], kH_RowB));
        CT_TRY(fn(mx_hi, xp, 3, xdims, xstr, xbox, kH_RowB));
        return fn(mx_lo, xp + (size_t)positions * c_pad * elem, 3, xdims, xstr, xbox, kH_RowB);
    };
    CT_TRY(encode(maps.w16, w16_hi, w16, &maps.x16_hi, &maps.x16_lo, 2));
    CT_TRY(encode(maps.w32, w32_hi, w32, &maps.x32_hi, &maps.x32_lo, 4));
    static bool attr_set_dev[16] = {}; // the attribute belongs to a device's context
    if (!attr_set_dev[st->device & 15]) {
        for (auto kernel : {conv_halo_stream_kernel<false, false>, conv_halo_stream_kernel<true, false>, conv_halo_stream_kernel<true, true>})
            CT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kH_Smem));
        attr_set_dev[st->device & 15] = true;
    }
    const unsigned grid = 2u * (unsigned)std::min<int64_t>(items, st->sm_count / 2);
    ProfScope prof("gemm_tc");
    const auto kernel = g.ring ? conv_halo_stream_kernel<true, true> : (three ? conv_halo_stream_kernel<true, false> : conv_halo_stream_kernel<false, false>);
    CT_CUDA(launch_dependent_cluster(kernel, 2, dim3(grid), dim3(kH_Threads), g.smem, stream(), maps, p));
    CT_LAUNCH_CHECK("conv_halo_stream");
    return CT_OK;
}

} // namespace ct
