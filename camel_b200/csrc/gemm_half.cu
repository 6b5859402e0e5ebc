// Tensor-core GEMM for float32 operands in split float16: C[m,n] = act(A[m,k] . B[k,n] + bias).
//
// Each operand value is two 11-bit significands (half_split.cuh); three MMAs of kind::f16 per 16
// values of k - lo.hi, hi.lo and hi.hi - give the 3xTF32 product at twice its rate, from planes of
// half the size.  What bounds it: the tensor pipe (three MMAs per product: a third of the f16 rate) for large
// products - 16384^3: 35.5 -> 21.7 ms, 405 TFLOP/s under the power cap - and for one wave of tiles the set-up,
// first operands and final store around 14 us of MMAs - 4096 x 1024 x 1024: 36 -> 27 us.
//
// Accumulation.  The low terms are stored 2^11 times larger, so the two cross products have an
// accumulator of their own (joined with weight 2^-11 at the end); the leading accumulator then sees one
// addition per 16 values of k instead of six, and its rounding error - the tensor core truncates at
// every addition - is a sixth per value of k of what the single 3xTF32 accumulator collects.  It is
// drained into registers every 1024 values of k and summed there with round-to-nearest adds.
//
// Values that float16 pairs hold in fewer bits than tf32 pairs would are listed by the pre-pass, and their products
// are added in the epilogue of the rows and columns they belong to.  Where there are too many for that, the
// wide_planes kernel (which returns at once otherwise) writes tf32 planes, and the GEMM kernel runs
// the same loop over those: same stage layout, same descriptors, kind::tf32, 8 values of k per MMA, all
// three products into one accumulator drained every 256 values of k.
//
// Structure: one CTA per SM walks 128 x BN tiles (BN = 256 or 128); warp 0 fetches operand stages by
// TMA, one lane of warp 1 issues the MMAs, warps 2-9 drain and store.  Tensor memory (512 columns) holds
// 512 / (2 BN) pairs of accumulators, so that with BN = 128 tile i + 1 computes while tile i drains; with
// BN = 256 the next tile's cross products start as soon as that accumulator has been read.  Every wait
// is bounded.
#include "common.cuh"
#include "half_split.cuh"
#include "split.cuh"
#include "tc_ptx.cuh"
#include "tmap.cuh"

#include <algorithm>

namespace ct {
namespace {

using namespace ptx;

constexpr int kHM         = 128;
constexpr int kHEpiWarps  = 8;
constexpr int kHThreads   = 64 + 32 * kHEpiWarps;
constexpr int kHEpiBytes  = kHEpiWarps * 32 * 128; // per warp 32 rows x 32 columns, float4 slots XOR-swizzled
constexpr int kChunkHalf  = 1024; // values of k per drain of the leading accumulator
constexpr int kChunkWide  = 256;  // the same over tf32 planes

// CG = 2: the tile is 256 rows high and belongs to a pair of CTAs, each with 128 rows of A, half of the
// rows of B and 128 accumulator rows.  The MMAs of a single CTA read 12 KB of shared memory each while TMA
// writes 58 B/clk: 147 of the 128 B/clk there are (80 % of the cycles in the MMAs at 4736 x 8192 x 1024).
// In a pair each CTA reads 8 KB per MMA and receives two thirds of the bytes.
template <int BN, int CG> struct HalfCfg {
    static constexpr int kRowB       = CG == 2 ? 128 : 64; // bytes of one operand row per stage = swizzle span
    static constexpr int kSteps      = kRowB / 32;         // MMAs along k per stage and product
    static constexpr int kABytes     = kHM * kRowB;
    static constexpr int kBRows      = BN / CG;
    static constexpr int kBBytes     = kBRows * kRowB;
    static constexpr int kStageBytes = 2 * (kABytes + kBBytes);
    static constexpr int kStages     = 192 * 1024 / kStageBytes;
    static constexpr int kSets       = 512 / (2 * BN); // accumulator pairs
    static constexpr int kCols       = BN / 2;         // columns per epilogue thread
    static constexpr int kSmemBytes  = kStages * kStageBytes + kHEpiBytes + 1024;
};

struct HalfGemmParams {
    int64_t m, n;
    int k_groups;         // groups of 64 values of k
    int groups_per_split; // > 0: split-K, groups per slice (slices take the batch index)
    int cluster_split;    // > 1: the slices of a tile are the CTAs of one cluster, which adds them up itself
    int tiles_m, tiles_n;
    int group_m;            // row tiles that sweep the column tiles together
    int total_tiles;
    int batch;              // > 1: B holds that many right operands of n rows each, outputs out_batch_stride apart
    const float *row_scale; // [m]: inverse scale of each row of A, negative for a row with exceptions
    const float *col_scale; // [batch][n]
    const __half *a_hi, *a_lo, *b_hi, *b_lo; // the float16 planes and lists, for those rows
    int kp;
    HalfExceptions *exceptions_a, *exceptions_b;
    int a_line0;
    const float *bias;
    int bias_per_row;       // bias indexed by output row
    int act;
    float *out;
    int64_t out_batch_stride;
    uint32_t *flags;
    int force_wide;                         // the tf32 planes hold the operands, whatever the exceptions say
    uint32_t *only_if;                      // zero there: nothing to do (LEFT)
    HalfExceptions *reset;                  // the library's own list, if one of them is that: the last CTA clears it
    // row bands, see ct_matmul_packed_bands
    int bands;
    int band_first[9];
    int64_t band_out_off[8];
    uint32_t *band_done;
};

struct HalfMaps {
    CUtensorMap a16_hi, a16_lo, b16_hi, b16_lo;
    CUtensorMap a32_hi, a32_lo, b32_hi, b32_lo;
};

__device__ __forceinline__ void half_tile(const HalfGemmParams &p, int tile, int &tm, int &tn, int &tz, int &band) {
    band = 0;
    if (p.bands > 0) { // band by band; inside a band its row tiles sweep the column tiles together
        tz      = 0;
        int bid = tile;
        while (band + 1 < p.bands && bid >= (p.band_first[band + 1] - p.band_first[band]) * p.tiles_n) {
            bid -= (p.band_first[band + 1] - p.band_first[band]) * p.tiles_n;
            ++band;
        }
        const int gm = p.band_first[band + 1] - p.band_first[band];
        tm           = p.band_first[band] + bid % gm;
        tn           = bid / gm;
        return;
    }
    // groups of row tiles sweep the column tiles, so that CTAs running together share operands in L2: 16 of
    // 128 rows, or 8 of 256 (74 pairs then cover a near-square 8 x 9 block of tiles)
    const int per_batch = p.tiles_m * p.tiles_n;
    tz                  = tile / per_batch;
    const int bid       = tile - tz * per_batch;
    const int g         = bid / (p.group_m * p.tiles_n);
    const int first_m   = g * p.group_m;
    const int gm        = p.tiles_m - first_m < p.group_m ? p.tiles_m - first_m : p.group_m;
    const int in_group  = bid - g * p.group_m * p.tiles_n;
    tm                  = first_m + in_group % gm;
    tn                  = in_group / gm;
}

// ---- exceptions (half_split.cuh) -------------------------------------------------------------
//
// exception_a . b + held_a . exception_b is what the accumulators lack of an output whose row or column has
// exceptions, the planes holding zeros in their place.  Sums run in order of k, whatever order the pre-pass found them in.

__device__ __forceinline__ float half_held(const __half *hi, const __half *lo, int64_t at, float inverse) {
    return (__half2float(hi[at]) + __half2float(lo[at]) * kHalfLoInv) * fabsf(inverse);
}
// Entry of a line with the smallest k above `after`, -1 if there is none.
__device__ __forceinline__ int half_next(const HalfExceptions *x, int n, int operand, int64_t line, int after) {
    int best = -1, best_k = 0;
    for (int i = 0; i < n; ++i) {
        const int l = x->e[i].line, k = x->e[i].k;
        if (l == line * 2 + operand && k > after && (best < 0 || k < best_k))
            best = i, best_k = k;
    }
    return best;
}

// What `count` outputs of row `row` lack, columns (lines of B) line + 32 g for g < count, into sum[].
template <int G>
__device__ __forceinline__ void half_missing(
    const HalfGemmParams &p, int64_t row, bool a_has, int64_t line, int count, float (&sum)[G]) {
    const HalfExceptions *xa = p.exceptions_a, *xb = p.exceptions_b;
    const int nb = (int)xb->count;
    float sc[G];
#pragma unroll
    for (int g = 0; g < G; ++g)
        sum[g] = 0.0f, sc[g] = g < count ? p.col_scale[line + 32 * g] : 1.0f;
    if (a_has) {
        const int na = (int)xa->count;
        for (int k = -1, i; (i = half_next(xa, na, 0, row + p.a_line0, k)) >= 0;) {
            k             = xa->e[i].k;
            const float a = xa->e[i].value;
            float b[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                b[g] = g < count ? half_held(p.b_hi, p.b_lo, (line + 32 * g) * p.kp + k, sc[g]) : 0.0f;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (sc[g] < 0.0f) {
                    const int j = half_next(xb, nb, 1, line + 32 * g, k - 1);
                    if (j >= 0 && xb->e[j].k == k)
                        b[g] += xb->e[j].value;
                }
                sum[g] = __fmaf_rn(a, b[g], sum[g]);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g)
        if (sc[g] < 0.0f)
            for (int k = -1, j; (j = half_next(xb, nb, 1, line + 32 * g, k)) >= 0;) {
                k      = xb->e[j].k;
                sum[g] = __fmaf_rn(half_held(p.a_hi, p.a_lo, row * p.kp + k, p.row_scale[row]), xb->e[j].value, sum[g]);
            }
}

// Finishes what a warp has stored without bias and activation because it lacks the exceptions' products: the rows and
// columns of its 32 x (32 G) block that have exceptions.  Called when the tile's sums are out of registers: a call among the stores cost
// every tile 300 bytes of spills.  Only these outputs are read back, a row at once: one exception in 1537 x 771 x 2050
// costs its tile about 3 us.
template <int G>
__device__ __noinline__ void half_finish(
    const HalfGemmParams &p, float *out_z, int64_t row0, int rows, int64_t col0, int64_t line0, bool add) {
    const int lane = threadIdx.x & 31;
    __syncwarp(); // the stores of the other lanes
    auto finish = [&](float x, float missing, int64_t row, int64_t col) {
        if (add) // once, where k is sliced
            x = __fadd_rn(x, missing);
        if (p.bias)
            x = __fadd_rn(x, p.bias[p.bias_per_row ? row : col]);
        if (p.act == CT_ACT_RELU)
            x = __fmul_rn(x, x > 0.0f ? 1.0f : 0.0f);
        out_z[row * p.n + col] = x;
    };
    const bool row_has      = lane < rows && p.row_scale[row0 + lane] < 0.0f;
    const uint32_t row_mask = __ballot_sync(0xffffffffu, row_has);
    const int64_t col       = col0 + lane;
    const int count         = (int)(p.n <= col ? 0 : min((int64_t)G, (p.n - col + 31) / 32));
    for (uint32_t m = row_mask; m; m &= m - 1) {
        const int64_t row = row0 + __ffs(m) - 1;
        float x[G], missing[G];
#pragma unroll
        for (int g = 0; g < G; ++g)
            x[g] = g < count ? out_z[row * p.n + col + 32 * g] : 0.0f;
        half_missing<G>(p, row, true, line0 + col, count, missing);
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (g < count)
                finish(x[g], missing[g], row, col + 32 * g);
    }
    for (int g = 0; g < G; ++g)
        for (uint32_t m = __ballot_sync(0xffffffffu, g < count && p.col_scale[line0 + col + 32 * g] < 0.0f); m; m &= m - 1) { // lane = row
            const int64_t c = col0 + 32 * g + __ffs(m) - 1;
            if (lane < rows && !row_has) {
                float missing[1];
                const float x = out_z[(row0 + lane) * p.n + c];
                half_missing<1>(p, row0 + lane, false, line0 + c, 1, missing);
                finish(x, missing[0], row0 + lane, c);
            }
        }
}

// The same for a tile added up by its cluster: the rows r0 .. of this CTA's share and the columns that have exceptions,
// from the slices' sums at `sums` in the CTAs.  The flags of 32 rows or columns are looked at together; a warp takes
// every tenth of those that have any.
template <int BN>
__device__ __noinline__ void half_finish_slices(
    const HalfGemmParams &p, uint32_t sums, int slices, int r0, int rows, int64_t row0, int64_t col0) {
    constexpr int kWarps = kHThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto store = [&](int r, int c, float missing) {
        const int64_t row = row0 + r, col = col0 + c;
        float x = 0.0f;
        for (int z = 0; z < slices; ++z) {
            const float4 q = ld_cluster_f4(sums + (uint32_t)r * (uint32_t)(BN * 4) + (uint32_t)(((c >> 2) ^ (r & 7)) << 4), (uint32_t)z);
            const float v  = (c & 2) ? ((c & 1) ? q.w : q.z) : ((c & 1) ? q.y : q.x);
            x              = z == 0 ? v : __fadd_rn(x, v);
        }
        x = __fadd_rn(__fmul_rn(x, fabsf(p.col_scale[col])), missing);
        if (p.bias)
            x = __fadd_rn(x, p.bias[p.bias_per_row ? row : col]);
        if (p.act == CT_ACT_RELU)
            x = __fmul_rn(x, x > 0.0f ? 1.0f : 0.0f);
        p.out[row * p.n + col] = x;
    };
    auto row_has = [&](int r) { return row0 + r < p.m && p.row_scale[row0 + r] < 0.0f; };
    for (int b = 0; b < rows; b += 32)
        for (uint32_t m = __ballot_sync(0xffffffffu, b + lane < rows && row_has(r0 + b + lane)); m; m &= m - 1) {
            const int r = b + __ffs(m) - 1;
            if (r % kWarps != warp)
                continue;
            const int64_t col = col0 + lane;
            const int count   = (int)(p.n <= col ? 0 : min((int64_t)(BN / 32), (p.n - col + 31) / 32));
            float missing[BN / 32];
            half_missing<BN / 32>(p, row0 + r0 + r, true, col, count, missing);
#pragma unroll
            for (int u = 0; u < BN / 32; ++u)
                if (u < count)
                    store(r0 + r, lane + 32 * u, missing[u]);
        }
    for (int b = 0; b < BN; b += 32)
        for (uint32_t m = __ballot_sync(0xffffffffu, col0 + b + lane < p.n && p.col_scale[col0 + b + lane] < 0.0f); m; m &= m - 1) {
            const int c = b + __ffs(m) - 1;
            if (c % kWarps != warp)
                continue;
            for (int r = r0 + lane; r < r0 + rows; r += 32)
                if (row0 + r < p.m && !row_has(r)) {
                    float missing[1];
                    half_missing<1>(p, row0 + r, false, col0 + c, 1, missing);
                    store(r, c, missing[0]);
                }
        }
}

// LEFT: behind a panel product, for the operands that it leaves (p.only_if).  An instantiation of its own: with the early
// exit in the ordinary one the compiler arranged the rest less well, two layers of 4096 x 1024 x 1024 85.4 -> 89.3 us.
// LINES: rows of the result that are not 16-byte aligned, at most one tile to a CTA or pair.  The operand stages are idle when
// the tile is stored, so a warp's rows go through them whole and are stored in 128-byte lines, wherever in a line a row
// begins; with a fixed 32 columns to a store every store has two partial sectors.  Timed in turn without it, runs of one side 0.1 %
// apart: 1537 x 771 x 2050 42.6 -> 41.6 us, 2305 x 771 x 1057 41.1 -> 40.1, 3000 x 500 x 1001 34.9 -> 33.0, 9000 x 300 x 301 29.9 -> 28.0,
// 10453 x 199 x 222 29.4 -> 27.6, 4609 x 130 x 514 26.2 -> 24.0, 1281 x 65 x 1793 23.3 -> 21.1.  In the ordinary kernel (for a CTA's
// last tile) the same code cost others 3 %: 4096 x 1024 x 1024 twice 86.1 -> 88.6, 7853 x 118 x 8502 219 -> 237.
template <int BN, int CG, bool LEFT, bool LINES>
__global__ void __launch_bounds__(kHThreads, 1)
    gemm_half_kernel(const __grid_constant__ HalfMaps maps, const __grid_constant__ HalfGemmParams p) {
    using C            = HalfCfg<BN, CG>;
    constexpr int RB   = C::kRowB;
    const int rank     = CG == 2 ? (int)cluster_rank() : 0;
    // tile walk of the CTA or pair.  Slices of one cluster: blocks s * tiles + t in the order of the general
    // split, so that the tile index of block (t, slice) is slice * tiles + t
    const int slices   = CG == 1 ? p.cluster_split : 0;
    const int first    = CG == 2       ? (int)(blockIdx.x >> 1)
                         : slices > 1 ? (int)(blockIdx.x % slices) * (p.tiles_m * p.tiles_n) + (int)(blockIdx.x / slices)
                                      : (int)blockIdx.x;
    const int stride   = CG == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[C::kStages], bar_empty[C::kStages];
    // [set * 2 + which]: which 0 = leading accumulator, 1 = cross products
    __shared__ uint64_t bar_acc_full[2 * C::kSets], bar_acc_empty[2 * C::kSets];
    __shared__ uint64_t bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s, lacking_s;
    // epilogue warps that have stored a tile (bands only), a counter per tile that may be under way: accumulators
    // are handed back before the store, so a warp can be kSets tiles ahead of another (one that has no columns to
    // store always is)
    static_assert(C::kSets < 4, "tile_stores");
    __shared__ int tile_stores[4];
    volatile int *abort_flag = &abort_flag_s;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    griddep_launch_dependents();
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    auto stage_addr          = [&](int s) { return smem_base + (uint32_t)s * C::kStageBytes; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int b = 0; b < 2 * C::kSets; ++b) {
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), kHEpiWarps * CG);
        }
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        tile_stores[0] = tile_stores[1] = tile_stores[2] = tile_stores[3] = 0;
        lacking_s = 0;
        prefetch_tensormap(&maps.a16_hi);
        prefetch_tensormap(&maps.a16_lo);
        prefetch_tensormap(&maps.b16_hi);
        prefetch_tensormap(&maps.b16_lo);
    }
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
    if (CG == 2)
        cluster_sync(); // the partner's barriers exist before anything is signalled on them
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    const bool failed        = abort_flag_s != 0; // an earlier launch failed: no work, but bands are released
    __syncthreads(); // every thread has read abort_flag_s before a role may raise it
    // everything above is set-up that does not depend on earlier kernels; the planes, the words and the
    // output may
    griddep_wait();
    if (LEFT && *reinterpret_cast<volatile uint32_t *>(p.only_if) == 0u) {
        __syncthreads();
        if (slices > 1)
            cluster_sync();
        if (warp == 1)
            tmem_dealloc(tmem_base, 512);
        if (threadIdx.x == 0 && p.reset && atomicAdd(p.flags + FLAG_EXCEPTION_READERS, 1u) + 1u == gridDim.x) {
            p.flags[FLAG_EXCEPTION_READERS] = 0u;
            p.reset->wide = p.reset->count = 0u;
        }
        return;
    }
    // One stage by TMA: values of k from kc, rows of A from a_row and of B from b_row.
    auto load_stage = [&](const CUtensorMap *ma_hi, const CUtensorMap *ma_lo, const CUtensorMap *mb_hi, const CUtensorMap *mb_lo,
                          int s, int32_t kc, int32_t a_row, int32_t b_row) {
        uint32_t full      = smem_u32(&bar_full[s]);
        const uint32_t dst = stage_addr(s);
        if (CG == 2) {
            // both CTAs' bytes are counted on the leader's barrier
            if (rank == 0)
                mbar_expect_tx(full, 2u * (uint32_t)C::kStageBytes);
            full = leader_addr(full);
            tma_load_2d_pair(dst, ma_hi, full, kc, a_row);
            tma_load_2d_pair(dst + 2 * C::kABytes, mb_hi, full, kc, b_row);
            tma_load_2d_pair(dst + C::kABytes, ma_lo, full, kc, a_row);
            tma_load_2d_pair(dst + 2 * C::kABytes + C::kBBytes, mb_lo, full, kc, b_row);
        } else {
            mbar_expect_tx(full, (uint32_t)C::kStageBytes);
            tma_load_2d(dst, ma_hi, full, kc, a_row);
            tma_load_2d(dst + 2 * C::kABytes, mb_hi, full, kc, b_row);
            tma_load_2d(dst + C::kABytes, ma_lo, full, kc, a_row);
            tma_load_2d(dst + 2 * C::kABytes + C::kBBytes, mb_lo, full, kc, b_row);
        }
    };
    auto rows_of = [&](int tm, int tn, int tz, int32_t &a_row, int32_t &b_row) {
        a_row = (tm * CG + rank) * kHM;
        b_row = (p.batch > 1 ? tz * (int32_t)p.n : 0) + tn * BN + rank * C::kBRows;
    };
    // The first tile's first float16 stages are fetched before it is known whether there are too many exceptions (that word
    // comes from L2, 0.7 us behind the wait above); where there are, the issuer passes them over.
    int ahead = 0;
    if (!LEFT && !p.force_wide && !failed && first < p.total_tiles) {
        int tm, tn, tz, band;
        half_tile(p, first, tm, tn, tz, band);
        const int first_group = p.groups_per_split > 0 ? tz * p.groups_per_split : 0;
        const int left        = p.k_groups > first_group ? p.k_groups - first_group : 0;
        ahead = (p.groups_per_split > 0 && left > p.groups_per_split ? p.groups_per_split : left) * (64 / (RB / 2));
        ahead = ahead < C::kStages ? ahead : C::kStages;
        if (warp == 0 && elect_one()) {
            int32_t a_row, b_row;
            rows_of(tm, tn, tz, a_row, b_row);
            for (int s = 0; s < ahead; ++s)
                load_stage(&maps.a16_hi, &maps.a16_lo, &maps.b16_hi, &maps.b16_lo, s, first_group * 64 + s * (RB / 2), a_row, b_row);
        }
    }
    const bool wide = p.force_wide || half_wide(p.exceptions_a, p.exceptions_b);
    const int k_step    = wide ? RB / 4 : RB / 2; // values of k per stage
    const int per_group = 64 / k_step;            // stages per 64 values of k
    const int chunk     = (wide ? kChunkWide : kChunkHalf) / k_step;
    auto k_range        = [&](int tz, int &first_group, int &nkb) {
        first_group    = p.groups_per_split > 0 ? tz * p.groups_per_split : 0;
        const int left = p.k_groups > first_group ? p.k_groups - first_group : 0; // a cluster's last slices may be empty
        nkb = (p.groups_per_split > 0 && left > p.groups_per_split ? p.groups_per_split : left) * per_group;
    };

    if (failed) {
        // a stream waiting for a band is released also when the launch has failed; the failure is on record
        if (threadIdx.x == 0 && p.bands > 0)
            for (int tile = first; tile < p.total_tiles; tile += stride) {
                int tm, tn, tz, band;
                half_tile(p, tile, tm, tn, tz, band);
                atomicAdd(p.band_done + band, 1u);
            }
    } else if (warp == 0) {
        // ===== TMA producer: stages numbered across tiles =====
        if (elect_one()) {
            const CUtensorMap *ma_hi = wide ? &maps.a32_hi : &maps.a16_hi, *ma_lo = wide ? &maps.a32_lo : &maps.a16_lo;
            const CUtensorMap *mb_hi = wide ? &maps.b32_hi : &maps.b16_hi, *mb_lo = wide ? &maps.b32_lo : &maps.b16_lo;
            int s = ahead == C::kStages ? 0 : ahead, issued = ahead;
            uint32_t phase = ahead == C::kStages ? 0 : 1;
            bool ok        = true;
            for (int tile = first; tile < p.total_tiles && ok; tile += stride) {
                int tm, tn, tz, band, first_group, nkb;
                half_tile(p, tile, tm, tn, tz, band);
                k_range(tz, first_group, nkb);
                int32_t a_row, b_row;
                rows_of(tm, tn, tz, a_row, b_row);
                int kb     = tile == first && !wide ? ahead : 0;
                int32_t kc = first_group * 64 + kb * k_step;
                for (; kb < nkb; ++kb, kc += k_step, ++issued) {
                    if (!mbar_wait(smem_u32(&bar_empty[s]), phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    load_stage(ma_hi, ma_lo, mb_hi, mb_lo, s, kc, a_row, b_row);
                    if (++s == C::kStages)
                        s = 0, phase ^= 1u;
                }
            }
            if (*abort_flag && rank == 0) {
                // unwind: let the copies still in flight land before the CTA goes away (the leader's barriers
                // count the partner's copies too, and neither CTA leaves before the other)
                for (int k2 = issued - C::kStages < 0 ? 0 : issued - C::kStages; k2 < issued; ++k2) {
                    const uint64_t t0 = globaltimer_ns();
                    while (!mbar_try_wait(smem_u32(&bar_full[k2 % C::kStages]), (uint32_t)(k2 / C::kStages) & 1u) &&
                           globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer (the leader's, for the pair) =====
        if (elect_one() && rank == 0) {
            const uint32_t idesc = make_idesc(wide ? 2u : 0u, kHM * CG, BN);
            int s = 0, i = 0;
            uint32_t phase = 0;
            uint32_t empty_phase = (1u << (2 * C::kSets)) - 1u; // bit per accumulator: parity to wait for
            bool ok = true;
            auto mma = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t accumulate) {
                if (CG == 2)
                    mma_f16_pair(d, da, db, idesc, accumulate);
                else
                    mma_f16(d, da, db, idesc, accumulate);
            };
            auto mma32 = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t accumulate) {
                if (CG == 2)
                    mma_tf32_pair(d, da, db, idesc, accumulate);
                else
                    mma_tf32(d, da, db, idesc, accumulate);
            };
            auto commit = [&](uint32_t bar) {
                if (CG == 2)
                    tc_commit_pair(bar);
                else
                    tc_commit(bar);
            };
            auto wait_empty = [&](int acc) {
                const bool got = mbar_wait<CG == 2 ? kClusterRead : kCta>(smem_u32(&bar_acc_empty[acc]), (empty_phase >> acc) & 1u, abort_flag);
                empty_phase ^= 1u << acc;
                tc_fence_after_sync();
                return got;
            };
            for (int b = 0; wide && b < ahead && ok; ++b) {
                ok = mbar_wait(smem_u32(&bar_full[s]), phase, abort_flag);
                commit(smem_u32(&bar_empty[s]));
                if (++s == C::kStages)
                    s = 0, phase ^= 1u;
            }
            for (int tile = first; tile < p.total_tiles && ok; tile += stride, ++i) {
                int tm, tn, tz, band, first_group, nkb;
                half_tile(p, tile, tm, tn, tz, band);
                k_range(tz, first_group, nkb);
                const int set         = C::kSets == 1 ? 0 : (i & (C::kSets - 1));
                const uint32_t d_main = tmem_base + (uint32_t)(set * 2 * BN), d_cross = d_main + BN;
                int in_chunk = 0, which = 0;
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!mbar_wait(smem_u32(&bar_full[s]), phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_hi = stage_addr(s), a_lo = a_hi + C::kABytes;
                    const uint32_t b_hi = a_hi + 2 * C::kABytes, b_lo = b_hi + C::kBBytes;
                    const uint64_t da_hi = smem_desc_k<RB>(a_hi), db_hi = smem_desc_k<RB>(b_hi);
                    const uint64_t da_lo = smem_desc_k<RB>(a_lo), db_lo = smem_desc_k<RB>(b_lo);
                    const bool last = kb + 1 == nkb;
                    if (!wide) {
                        if (kb == 0 && !wait_empty(set * 2 + 1)) {
                            ok = false;
                            break;
                        }
#pragma unroll
                        for (int kk = 0; kk < C::kSteps; ++kk) {
                            mma(d_cross, da_lo + 2 * kk, db_hi + 2 * kk, kb == 0 && kk == 0 ? 0u : 1u);
                            mma(d_cross, da_hi + 2 * kk, db_lo + 2 * kk, 1u);
                        }
                        if (in_chunk == 0 && !wait_empty(set * 2)) {
                            ok = false;
                            break;
                        }
#pragma unroll
                        for (int kk = 0; kk < C::kSteps; ++kk)
                            mma(d_main, da_hi + 2 * kk, db_hi + 2 * kk, in_chunk == 0 && kk == 0 ? 0u : 1u);
                    } else {
                        if (in_chunk == 0 && !wait_empty(set * 2 + which)) {
                            ok = false;
                            break;
                        }
                        const uint32_t d = which ? d_cross : d_main;
#pragma unroll
                        for (int kk = 0; kk < C::kSteps; ++kk) {
                            mma32(d, da_lo + 2 * kk, db_hi + 2 * kk, in_chunk == 0 && kk == 0 ? 0u : 1u);
                            mma32(d, da_hi + 2 * kk, db_lo + 2 * kk, 1u);
                            mma32(d, da_hi + 2 * kk, db_hi + 2 * kk, 1u);
                        }
                    }
                    commit(smem_u32(&bar_empty[s])); // stage reusable once these MMAs retire
                    if (++s == C::kStages)
                        s = 0, phase ^= 1u;
                    if (++in_chunk == chunk || last) {
                        commit(smem_u32(&bar_acc_full[set * 2 + which]));
                        in_chunk = 0;
                        if (wide)
                            which ^= 1;
                    }
                    if (last && !wide)
                        commit(smem_u32(&bar_acc_full[set * 2 + 1]));
                }
            }
            if (!ok || *abort_flag) {
                // unwind: wait until every MMA issued so far has retired
                commit(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else {
        // ===== epilogue =====
        const int ew      = warp - 2;
        const int quarter = warp & 3; // TMEM lanes this warp may read: 32 * quarter ..
        const int half    = ew >> 2;  // which half of the tile's columns
        uint8_t *stg = smem_raw + (smem_base - smem_u32(smem_raw)) + (uint32_t)C::kStages * C::kStageBytes + (uint32_t)ew * 4096u;
        uint32_t full_phase = 0;
        int i               = 0;
        for (int tile = first; tile < p.total_tiles; tile += stride, ++i) {
            int tm, tn, tz, band, first_group, nkb;
            half_tile(p, tile, tm, tn, tz, band);
            k_range(tz, first_group, nkb);
            const int set         = C::kSets == 1 ? 0 : (i & (C::kSets - 1));
            const int num_chunks  = (nkb + chunk - 1) / chunk;
            const int64_t row0    = (int64_t)(tm * CG + rank) * kHM + quarter * 32;
            const int64_t tile_c0 = (int64_t)tn * BN;
            // column scale and bias of column 32 g + lane, fetched before the accumulator is waited for and
            // handed round by shuffles when the tile is stored (no barrier between the epilogue warps: after
            // a failed wait they leave one by one)
            float cs[C::kCols / 32], bb[C::kCols / 32];
            bool lacking = false; // a row or column of this warp's has exceptions
#pragma unroll
            for (int g = 0; g < C::kCols / 32; ++g) {
                const int64_t col = tile_c0 + half * C::kCols + g * 32 + lane;
                cs[g]             = (!wide && col < p.n) ? p.col_scale[(p.batch > 1 ? tz * p.n : 0) + col] : 1.0f;
                lacking |= cs[g] < 0.0f;
                cs[g] = fabsf(cs[g]);
                bb[g]             = (p.bias && !p.bias_per_row && col < p.n) ? p.bias[col] : 0.0f;
            }
            const float row_bias = (p.bias_per_row && row0 + lane < p.m) ? p.bias[row0 + lane] : 0.0f;
            float rs = (!wide && row0 + lane < p.m) ? p.row_scale[row0 + lane] : 1.0f;
            lacking  = __any_sync(0xffffffffu, lacking || rs < 0.0f);
            rs       = fabsf(rs);

            float acc[C::kCols];
            const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * 2 * BN + half * C::kCols);
            bool ok                  = true;
            auto await = [&](int which) {
                const int a    = set * 2 + which;
                const bool got = mbar_wait(smem_u32(&bar_acc_full[a]), (full_phase >> a) & 1u, abort_flag);
                full_phase ^= 1u << a;
                ok = __all_sync(0xffffffffu, got);
                tc_fence_after_sync();
                return ok;
            };
            auto hand_back = [&](int which) {
                const uint32_t bar = smem_u32(&bar_acc_empty[set * 2 + which]);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2)
                        mbar_arrive_peer_read(leader_addr(bar));
                    else
                        mbar_arrive(bar);
                }
            };
            // 3 x f16: leading accumulator of every chunk but the last, then the cross products (the next tile
            // starts with those: hand that accumulator back first), then the last chunk.  Sixteen columns at a time: all
            // of the first accumulator with one wait had every register twice and spilled (4096 x 1024 x 1024 38.8 us
            // against 38.5, 1537 x 771 x 2050 39.8 against 39.6).
            const int events = wide || nkb == 0 ? num_chunks : num_chunks + 1;
            auto which_of    = [&](int c) { return wide ? (c & 1) : (c == num_chunks - 1 ? 1 : 0); };
            if (events > 0 && await(which_of(0))) {
                const int which    = which_of(0);
                const float weight = !wide && which ? kHalfLoInv : 1.0f;
#pragma unroll
                for (int g = 0; g < C::kCols / 16; ++g) {
                    uint32_t r[16];
                    tmem_ld_32x16(lane_base + (uint32_t)(which * BN + g * 16), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[g * 16 + j] = __fmul_rn(__uint_as_float(r[j]), weight);
                }
                hand_back(which);
            } else {
#pragma unroll
                for (int j = 0; j < C::kCols; ++j)
                    acc[j] = 0.0f;
            }
#pragma unroll 1
            for (int c = 1; c < events && ok; ++c) {
                const int which    = which_of(c);
                const float weight = !wide && which ? kHalfLoInv : 1.0f;
                if (!await(which))
                    break;
#pragma unroll
                for (int g = 0; g < C::kCols / 16; ++g) {
                    uint32_t r[16];
                    tmem_ld_32x16(lane_base + (uint32_t)(which * BN + g * 16), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[g * 16 + j] = __fadd_rn(acc[g * 16 + j], __fmul_rn(__uint_as_float(r[j]), weight));
                }
                hand_back(which);
            }
            if (!ok)
                break;

            if (slices > 1) {
                if (lacking && lane == 0)
                    lacking_s = 1; // every slice sees the same rows and columns
                // this slice's 128 x 128 sums go to the idle operand stages (every MMA has retired), rows of 512
                // bytes, float4 slots XOR-swizzled; the cluster adds them up below
                uint8_t *part = smem_raw + (smem_base - smem_u32(smem_raw)) + (uint32_t)(quarter * 32 + lane) * (BN * 4u);
#pragma unroll
                for (int j = 0; j < C::kCols / 4; ++j)
                    *reinterpret_cast<float4 *>(part + (((half * (C::kCols / 4) + j) ^ (lane & 7)) << 4)) =
                        make_float4(__fmul_rn(acc[4 * j], rs), __fmul_rn(acc[4 * j + 1], rs), __fmul_rn(acc[4 * j + 2], rs),
                                    __fmul_rn(acc[4 * j + 3], rs));
                break; // one tile per CTA
            }

            float *out_z        = p.out + (int64_t)tz * p.out_batch_stride + (p.bands > 0 ? p.band_out_off[band] : 0);
            const bool vec      = (p.n & 3) == 0 && (reinterpret_cast<uintptr_t>(out_z) & 15u) == 0;
            const int rows_left = (int)(p.m - row0 < 32 ? (p.m - row0 < 0 ? 0 : p.m - row0) : 32);
            if (LINES && !lacking) { // every MMA has retired
                uint8_t *block = smem_raw + (smem_base - smem_u32(smem_raw)) + (uint32_t)ew * (32u * C::kCols * 4u);
                float2 *columns = reinterpret_cast<float2 *>(stg); // scale and bias
#pragma unroll
                for (int g = 0; g < C::kCols / 32; ++g)
                    columns[g * 32 + lane] = make_float2(cs[g], bb[g]);
#pragma unroll
                for (int j = 0; j < C::kCols / 4; ++j)
                    *reinterpret_cast<float4 *>(block + lane * (C::kCols * 4) + ((j ^ (lane & 7)) << 4)) =
                        make_float4(__fmul_rn(acc[4 * j], rs), __fmul_rn(acc[4 * j + 1], rs), __fmul_rn(acc[4 * j + 2], rs),
                                    __fmul_rn(acc[4 * j + 3], rs));
                __syncwarp();
                const int64_t left = p.n - tile_c0 - half * C::kCols;
                const int width    = (int)(left < C::kCols ? (left < 0 ? 0 : left) : C::kCols);
                float *dst         = out_z + row0 * p.n + tile_c0 + half * C::kCols;
#pragma unroll 1
                for (int r = 0; r < rows_left; ++r, dst += p.n) {
                    const int first = lane - (int)((reinterpret_cast<uintptr_t>(dst) >> 2) & 31u);
                    const float rb  = __shfl_sync(0xffffffffu, row_bias, r);
                    float x[C::kCols / 32 + 1];
                    float2 cb[C::kCols / 32 + 1];
#pragma unroll
                    for (int j = 0; j <= C::kCols / 32; ++j) {
                        const int col  = first + 32 * j;
                        const bool in  = col >= 0 && col < width;
                        const int from = in ? col : 0;
                        x[j]  = *reinterpret_cast<const float *>(block + r * (C::kCols * 4) + (((from >> 2) ^ (r & 7)) << 4) + (from & 3) * 4);
                        cb[j] = columns[from];
                    }
#pragma unroll
                    for (int j = 0; j <= C::kCols / 32; ++j) {
                        const int col = first + 32 * j;
                        float y       = __fmul_rn(x[j], cb[j].x);
                        if (p.bias)
                            y = __fadd_rn(y, p.bias_per_row ? rb : cb[j].y);
                        if (p.act == CT_ACT_RELU)
                            y = __fmul_rn(y, y > 0.0f ? 1.0f : 0.0f);
                        if (col >= 0 && col < width)
                            dst[col] = y;
                    }
                }
                __syncwarp();
            } else
#pragma unroll
            for (int g = 0; g < C::kCols / 32; ++g) {
                const int c0        = half * C::kCols + g * 32; // column of the tile
                const int64_t left  = p.n - tile_c0 - c0;
                const int cols_left = (int)(left < 32 ? (left < 0 ? 0 : left) : 32);
                if (cols_left == 0)
                    break;
                // 32 x 32 values through the warp's staging block (float4 slots XOR-swizzled by row: no
                // bank conflicts either way), written out as runs of 128 contiguous bytes per row
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<float4 *>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                        make_float4(__fmul_rn(acc[g * 32 + 4 * j], rs), __fmul_rn(acc[g * 32 + 4 * j + 1], rs),
                                    __fmul_rn(acc[g * 32 + 4 * j + 2], rs), __fmul_rn(acc[g * 32 + 4 * j + 3], rs));
                __syncwarp();
                if (vec && cols_left == 32) {
                    const int sub = lane & 7, rr = lane >> 3;
                    float c4[4], b4[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        c4[q] = __shfl_sync(0xffffffffu, cs[g], sub * 4 + q);
                        b4[q] = __shfl_sync(0xffffffffu, bb[g], sub * 4 + q);
                    }
                    float *dst      = out_z + (row0 + rr) * p.n + tile_c0 + c0 + sub * 4;
#pragma unroll 4
                    for (int it = 0; it < 8; ++it) {
                        const int r = it * 4 + rr;
                        float4 v    = *reinterpret_cast<const float4 *>(stg + r * 128 + ((sub ^ (r & 7)) << 4));
                        v = make_float4(__fmul_rn(v.x, c4[0]), __fmul_rn(v.y, c4[1]), __fmul_rn(v.z, c4[2]), __fmul_rn(v.w, c4[3]));
                        if (p.bias_per_row) {
                            const float rb = __shfl_sync(0xffffffffu, row_bias, r);
                            b4[0] = b4[1] = b4[2] = b4[3] = rb;
                        }
                        if (p.bias)
                            v = make_float4(__fadd_rn(v.x, b4[0]), __fadd_rn(v.y, b4[1]), __fadd_rn(v.z, b4[2]), __fadd_rn(v.w, b4[3]));
                        if (p.act == CT_ACT_RELU)
                            v = make_float4(__fmul_rn(v.x, v.x > 0.0f ? 1.0f : 0.0f), __fmul_rn(v.y, v.y > 0.0f ? 1.0f : 0.0f),
                                            __fmul_rn(v.z, v.z > 0.0f ? 1.0f : 0.0f), __fmul_rn(v.w, v.w > 0.0f ? 1.0f : 0.0f));
                        if (r < rows_left)
                            *reinterpret_cast<float4 *>(dst) = v;
                        dst += 4 * p.n;
                    }
                } else {
                    // ragged edge or rows that are not 16-byte aligned: a column per lane
                    float *dst = out_z + row0 * p.n + tile_c0 + c0 + lane;
#pragma unroll 4
                    for (int r = 0; r < rows_left; ++r) {
                        float x = *reinterpret_cast<const float *>(stg + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
                        x       = __fmul_rn(x, cs[g]);
                        const float rb = __shfl_sync(0xffffffffu, row_bias, r);
                        if (p.bias)
                            x = __fadd_rn(x, p.bias_per_row ? rb : bb[g]);
                        if (p.act == CT_ACT_RELU)
                            x = __fmul_rn(x, x > 0.0f ? 1.0f : 0.0f);
                        if (lane < cols_left)
                            dst[(int64_t)r * p.n] = x;
                    }
                }
                if (lacking) { // their outputs without bias and activation again: half_finish has the rest
                    const bool col_has      = lane < cols_left && p.col_scale[(p.batch > 1 ? tz * p.n : 0) + tile_c0 + c0 + lane] < 0.0f;
                    const uint32_t row_mask = __ballot_sync(0xffffffffu, lane < rows_left && p.row_scale[row0 + lane] < 0.0f);
#pragma unroll 1
                    for (int r = 0; r < rows_left; ++r)
                        if (((row_mask >> r & 1u) || col_has) && lane < cols_left)
                            out_z[(row0 + r) * p.n + tile_c0 + c0 + lane] = __fmul_rn(
                                *reinterpret_cast<const float *>(stg + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4), cs[g]);
                }
                __syncwarp(); // the block is rewritten by the next 32 columns
            }
            if (lacking)
                half_finish<C::kCols / 32>(p, out_z, row0, rows_left, tile_c0 + half * C::kCols, p.batch > 1 ? tz * p.n : 0, first_group == 0);
            if (p.bands > 0) {
                // the last warp to have stored the tile counts it; tile i + 4 comes to the same counter only after
                // every warp is past tile i
                __threadfence();
                __syncwarp();
                if (lane == 0 && atomicAdd(&tile_stores[i & 3], 1) == kHEpiWarps - 1) {
                    tile_stores[i & 3] = 0;
                    __threadfence();
                    atomicAdd(p.band_done + band, 1u);
                }
            }
        }
    }

    if (CG == 1 && slices > 1) {
        // Each CTA of the cluster adds up its share of the tile's rows over all slices, in slice order,
        // through distributed shared memory: no partial sums in memory and no second launch.
        __syncthreads();
        cluster_sync();
        int tm, tn, tz, band;
        half_tile(p, first, tm, tn, tz, band);
        const int rows_each = kHM / slices;
        const bool vec      = (p.n & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
        if (!failed && !abort_flag_s)
            for (int i = threadIdx.x; i < rows_each * (BN / 4); i += kHThreads) {
                const int r = (int)cluster_rank() * rows_each + i / (BN / 4), slot = i % (BN / 4);
                const int64_t row = (int64_t)tm * kHM + r, col = (int64_t)tn * BN + slot * 4;
                if (row >= p.m || col >= p.n)
                    continue;
                const uint32_t at = smem_base + (uint32_t)r * (BN * 4u) + (uint32_t)((slot ^ (r & 7)) << 4);
                float4 v          = ld_cluster_f4(at, 0);
#pragma unroll 4
                for (int z = 1; z < slices; ++z) {
                    const float4 q = ld_cluster_f4(at, (uint32_t)z);
                    v = make_float4(__fadd_rn(v.x, q.x), __fadd_rn(v.y, q.y), __fadd_rn(v.z, q.z), __fadd_rn(v.w, q.w));
                }
                float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (col + q < p.n) {
                        x[q] = __fmul_rn(x[q], wide ? 1.0f : fabsf(p.col_scale[col + q]));
                        if (p.bias)
                            x[q] = __fadd_rn(x[q], p.bias[p.bias_per_row ? row : col + q]);
                        if (p.act == CT_ACT_RELU)
                            x[q] = __fmul_rn(x[q], x[q] > 0.0f ? 1.0f : 0.0f);
                    }
                }
                float *dst = p.out + row * p.n + col;
                if (vec && col + 3 < p.n) {
                    *reinterpret_cast<float4 *>(dst) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (col + q < p.n)
                            dst[q] = x[q];
                }
            }
        if (lacking_s && !failed && !abort_flag_s) {
            __syncthreads(); // what follows writes some of these outputs again
            half_finish_slices<BN>(p, smem_base, slices, (int)cluster_rank() * rows_each, rows_each, (int64_t)tm * kHM, (int64_t)tn * BN);
        }
        cluster_sync(); // a CTA's sums stay until every other CTA has read them
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
    if (threadIdx.x == 0) {
        if (!failed && *abort_flag) {
            atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
            // waiting streams are released: at least the whole count of every band (a band's count may
            // then overshoot; the failure is on record)
            for (int tile = first; p.bands > 0 && tile < p.total_tiles; tile += stride) {
                int tm, tn, tz, band;
                half_tile(p, tile, tm, tn, tz, band);
                atomicAdd(p.band_done + band, 1u);
            }
        }
        if (p.reset) {
            // the last CTA to get here clears it for the next product
            if (atomicAdd(p.flags + FLAG_EXCEPTION_READERS, 1u) + 1u == gridDim.x) {
                p.flags[FLAG_EXCEPTION_READERS] = 0u;
                p.reset->wide = p.reset->count = 0u;
                if (LEFT)
                    *p.only_if = 0u;
            }
        }
    }
}

// ---- operand pre-pass ---------------------------------------------------------------------

// What a pre-pass writes: float16 planes, inverse scales (negative: a row with exceptions), the exceptions and, for
// small operands (hi32 non-null), the tf32 planes as well, which then need no launch of their own.
struct HalfPlanes {
    __half *hi16, *lo16;
    float *scale;
    HalfExceptions *exceptions;
    int operand;
    float *hi32, *lo32;
};

HalfPlanes planes_of(const HalfOperand &o, bool both_forms) {
    return HalfPlanes{static_cast<__half *>(const_cast<void *>(o.hi16)), static_cast<__half *>(const_cast<void *>(o.lo16)),
                      const_cast<float *>(o.scale), o.exceptions, o.operand,
                      both_forms ? static_cast<float *>(const_cast<void *>(o.hi32)) : nullptr,
                      both_forms ? static_cast<float *>(const_cast<void *>(o.lo32)) : nullptr};
}

// A line whose range is not plain - it has exceptions, infinities or NaN - is split as if it had none and then put
// right here: zeros and an entry in the list for each exception, no low term for the others.  Called by `threads`
// threads, whole warps; true if there are exceptions.
__device__ __noinline__ bool half_repair(
    const float *src, int64_t stride, int64_t k, float scale, __half *hi, __half *lo, HalfExceptions *x, int operand, int64_t line, int t,
    int threads) {
    bool found = false;
    for (int64_t c = t; __any_sync(0xffffffffu, c < k); c += threads) {
        if (__all_sync(0xffffffffu, half_overfull(x)))
            return true; // the planes will not be read
        const float v = c < k ? src[c * stride] : 0.0f;
        found |= half_record(x, v, scale, operand, line, c);
        if (half_exception(v, scale))
            hi[c] = __half(0.0f), lo[c] = __half(0.0f);
        else if (!isfinite(v))
            lo[c] = __half(0.0f);
    }
    return found;
}
// Whether a line with this range (half_split.cuh) and scale needs it.
__device__ __forceinline__ bool half_not_plain(uint2 range, float scale) {
    return range.x >= 0x7f800000u || (range.y != kNoneSmallest && __uint_as_float(range.y + 1u) * scale < kHalfSmallest);
}

// in [rows][k] -> float16 planes [rows][kp], inverse row scales.  TPR threads per row keep the row in
// registers (V float4 each, rows of up to 16384) between finding its largest magnitude and splitting it;
// longer rows are read twice (the second time from L2).  Bound by memory: 4 bytes read and 4 written per value.
template <int TPR, int V>
__device__ __forceinline__ void half_rows(
    int64_t block, const float *__restrict__ in, int64_t rows, int64_t k, int64_t kp, const HalfPlanes &p, int vec_ok) {
    __shared__ uint2 range_s[8];
    constexpr int RPB = 256 / TPR;
    const int t       = threadIdx.x % TPR;
    const int64_t row = block * RPB + threadIdx.x / TPR;
    if (TPR == 32 && row >= rows)
        return;
    const float *src = in + row * k;
    auto load        = [&](int64_t c) {
        if (vec_ok && c + 3 < k)
            return __ldcs(reinterpret_cast<const float4 *>(src + c));
        float4 q;
        q.x = c < k ? src[c] : 0.0f;
        q.y = c + 1 < k ? src[c + 1] : 0.0f;
        q.z = c + 2 < k ? src[c + 2] : 0.0f;
        q.w = c + 3 < k ? src[c + 3] : 0.0f;
        return q;
    };
    float4 v[V];
    uint2 range = make_uint2(0u, kNoneSmallest);
    auto take   = [&](const float4 &q) {
        range_take(range, q.x), range_take(range, q.y), range_take(range, q.z), range_take(range, q.w);
    };
    auto reduce = [&]() {
        range = range_warp(range);
        if (TPR == 256) {
            if ((threadIdx.x & 31) == 0)
                range_s[threadIdx.x >> 5] = range;
            __syncthreads();
#pragma unroll
            for (int w = 0; w < 8; ++w)
                range = range_join(range, range_s[w]);
        }
    };
    const bool fits = kp <= TPR * V * 4;
    if (fits) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int64_t c = (int64_t)(t + j * TPR) * 4;
            v[j]            = c < k ? load(c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int j = 0; j < V; ++j)
            take(v[j]);
    } else {
        for (int64_t c = t * 4; c < k; c += TPR * 4)
            take(load(c));
    }
    reduce();
    const bool finite = range.x < 0x7f800000u;
    if (!finite) { // rare: the scale is that of the finite values
        if (TPR == 256)
            __syncthreads();
        range = make_uint2(0u, kNoneSmallest);
        for (int64_t c = t; c < k; c += TPR)
            range_take(range, isfinite(src[c]) ? src[c] : 0.0f);
        reduce();
    }
    float scale, inverse;
    const bool ok = half_scale(range.x, scale, inverse);
    auto put      = [&](int64_t c, const float4 &q) {
        __half2 hi[2], lo[2];
        split_half_pair(q.x * scale, q.y * scale, hi[0], lo[0]);
        split_half_pair(q.z * scale, q.w * scale, hi[1], lo[1]);
        *reinterpret_cast<uint2 *>(p.hi16 + row * kp + c) = *reinterpret_cast<uint2 *>(hi);
        *reinterpret_cast<uint2 *>(p.lo16 + row * kp + c) = *reinterpret_cast<uint2 *>(lo);
        if (p.hi32) {
            float4 h, l;
            split_tf32_flat(q.x, h.x, l.x);
            split_tf32_flat(q.y, h.y, l.y);
            split_tf32_flat(q.z, h.z, l.z);
            split_tf32_flat(q.w, h.w, l.w);
            *reinterpret_cast<float4 *>(p.hi32 + row * kp + c) = h;
            *reinterpret_cast<float4 *>(p.lo32 + row * kp + c) = l;
        }
    };
    if (fits) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int64_t c = (int64_t)(t + j * TPR) * 4;
            if (c < kp)
                put(c, v[j]);
        }
    } else {
        for (int64_t c = t * 4; c < kp; c += TPR * 4)
            put(c, c < k ? load(c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    }
    bool bad = false;
    if (!finite || half_not_plain(range, scale)) { // rare, and the same for all threads of the row
        if (TPR == 256)
            __syncthreads();
        else
            __syncwarp();
        bad = half_repair(src, 1, k, scale, p.hi16 + row * kp, p.lo16 + row * kp, p.exceptions, p.operand, row, t, TPR);
        if (TPR == 256)
            bad = __syncthreads_or(bad) != 0;
    }
    if (t == 0) {
        p.scale[row] = bad ? -inverse : inverse;
        if (!ok)
            p.exceptions->wide = 1u;
    }
}

template <int TPR, int V>
__global__ void __launch_bounds__(256) half_rows_kernel(
    const float *__restrict__ in, int64_t rows, int64_t k, int64_t kp, const HalfPlanes p, int vec_ok,
    uint32_t *__restrict__ zero, int64_t zero_count) {
    griddep_launch_dependents();
    griddep_wait();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < zero_count; i += (int64_t)gridDim.x * 256)
        zero[i] = 0u; // scales and column maxima of the right operand, accumulated by the next kernels
    half_rows<TPR, V>((int64_t)blockIdx.x, in, rows, k, kp, p, vec_ok);
}

// Behind a panel product, which seldom leaves anything: a block to an SM, which walks the rows if *only_if says so.
__global__ void __launch_bounds__(256) half_rows_left_kernel(
    const float *__restrict__ in, int64_t rows, int64_t k, int64_t kp, const HalfPlanes p, int vec_ok,
    const uint32_t *__restrict__ only_if) {
    griddep_launch_dependents();
    griddep_wait();
    if (*reinterpret_cast<const volatile uint32_t *>(only_if) == 0u)
        return;
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        half_rows<256, 8>(row, in, rows, k, kp, p, vec_ok);
        __syncthreads();
    }
}

// Largest finite magnitude of each column of in [k][n], by atomic maximum into col_max (zeroed before).  128 columns to a block,
// a row of them to a warp.
__global__ void __launch_bounds__(256) half_col_max_kernel(
    const float *__restrict__ in, int64_t k, int64_t n, int64_t rows_per_block, int vec_ok, uint32_t *__restrict__ col_max) {
    __shared__ uint32_t max_s[8][128];
    griddep_launch_dependents();
    griddep_wait();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t n0 = (int64_t)blockIdx.x * 128;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_block, r1 = min(k, r0 + rows_per_block);
    uint32_t mx[4] = {0, 0, 0, 0};
    if (vec_ok) {
        if (n0 + tx * 4 < n)
#pragma unroll 8
            for (int64_t r = r0 + ty; r < r1; r += 8) {
                const float4 v = *reinterpret_cast<const float4 *>(in + r * n + n0 + tx * 4);
                mx[0] = max(mx[0], finite_magnitude(v.x)), mx[1] = max(mx[1], finite_magnitude(v.y));
                mx[2] = max(mx[2], finite_magnitude(v.z)), mx[3] = max(mx[3], finite_magnitude(v.w));
            }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            max_s[ty][tx * 4 + q] = mx[q];
    } else {
#pragma unroll 4
        for (int64_t r = r0 + ty; r < r1; r += 8)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                mx[q] = max(mx[q], n0 + tx + 32 * q < n ? finite_magnitude(in[r * n + n0 + tx + 32 * q]) : 0u);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            max_s[ty][tx + 32 * q] = mx[q];
    }
    __syncthreads();
    if (threadIdx.x < 128 && n0 + threadIdx.x < n) {
        uint32_t all = max_s[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < 8; ++w)
            all = max(all, max_s[w][threadIdx.x]);
        atomicMax(col_max + n0 + threadIdx.x, all);
    }
}

// in [k][n] -> transposed float16 planes [n][kp], inverse column scales.  Blocks of 64 k x 64 columns, eight values of k to a
// thread and 16-byte stores: 16384 x 16384 with the maxima 813 us, with one half2 to a store and 32 columns to a block
// 1030.  The first block of a column writes its scale, any of them its sign (both by OR, the scales start at zero).
__global__ void __launch_bounds__(256) half_cols_kernel(
    const float *__restrict__ in, int64_t k, int64_t n, int64_t kp, const HalfPlanes p, int vec_ok, const uint32_t *__restrict__ col_max) {
    __shared__ float tile[64][65];
    griddep_launch_dependents();
    griddep_wait();
    const int64_t n0 = (int64_t)blockIdx.x * 64, k0 = (int64_t)blockIdx.y * 64;
    transpose_load(tile, in, k, n, k0, n0, vec_ok);
    __syncthreads();
    const int kc = (threadIdx.x & 7) * 8;
    const int64_t kk = k0 + kc;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int col    = (threadIdx.x >> 3) + 32 * j;
        const int64_t nn = n0 + col;
        const bool there = nn < n && kk < kp;
        float scale, inverse;
        const bool ok  = half_scale(nn < n ? col_max[nn] : 0u, scale, inverse);
        uint32_t *word = reinterpret_cast<uint32_t *>(p.scale + (nn < n ? nn : 0));
        if (nn < n && kk == 0) {
            atomicOr(word, __float_as_uint(inverse));
            if (!ok)
                p.exceptions->wide = 1u;
        }
        float v[8];
        bool special = false;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            v[u] = tile[kc + u][col];
            special |= half_exception(v[u], scale) || !isfinite(v[u]);
        }
        special = special && there;
        if (there) {
            __half2 hi[4], lo[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                split_half_pair(v[2 * u] * scale, v[2 * u + 1] * scale, hi[u], lo[u]);
            if (special)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    split_half(v[2 * u], scale, hi[u].x, lo[u].x);
                    split_half(v[2 * u + 1], scale, hi[u].y, lo[u].y);
                }
            *reinterpret_cast<uint4 *>(p.hi16 + nn * kp + kk) = *reinterpret_cast<uint4 *>(hi);
            *reinterpret_cast<uint4 *>(p.lo16 + nn * kp + kk) = *reinterpret_cast<uint4 *>(lo);
            if (p.hi32)
#pragma unroll
                for (int u = 0; u < 8; u += 4) {
                    float4 h, l;
                    split_tf32_flat(v[u], h.x, l.x);
                    split_tf32_flat(v[u + 1], h.y, l.y);
                    split_tf32_flat(v[u + 2], h.z, l.z);
                    split_tf32_flat(v[u + 3], h.w, l.w);
                    *reinterpret_cast<float4 *>(p.hi32 + nn * kp + kk + u) = h;
                    *reinterpret_cast<float4 *>(p.lo32 + nn * kp + kk + u) = l;
                }
        }
        if (__any_sync(0xffffffffu, special))
#pragma unroll 1
            for (int u = 0; u < 8; ++u) {
                const float value = there ? tile[kc + u][col] : 0.0f;
                half_record(p.exceptions, value, scale, p.operand, nn, kk + u);
                if (half_exception(value, scale))
                    atomicOr(word, 0x80000000u);
            }
    }
}

// The same for k <= kShortK in one pass: a block keeps the whole length of 8 columns (32 bytes of each row, a
// sector) in shared memory between the maximum and the split, a warp per column.  Up to 1024, where six such blocks
// share an SM: at 4096 there was one, with too few loads in flight (two passes over the columns are faster).
constexpr int kShortCols = 8;
constexpr int kShortK    = 1024;
constexpr int kShortPad  = kShortCols + 1;

__device__ __forceinline__ void half_cols_short(
    float *tile, int block, const float *__restrict__ in, int64_t k, int64_t n, int64_t kp, const HalfPlanes &p) {
    const int tx = threadIdx.x & (kShortCols - 1), ty = threadIdx.x / kShortCols; // 32 rows at a time
    const int64_t n0 = (int64_t)block * kShortCols;
    const bool col_ok = n0 + tx < n;
    const float *src  = in + n0 + tx;
#pragma unroll 8
    for (int kk = ty; kk < (int)kp; kk += 32)
        tile[kk * kShortPad + tx] = (col_ok && kk < k) ? src[(int64_t)kk * n] : 0.0f;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint2 range    = make_uint2(0u, kNoneSmallest);
    for (int kk = lane; kk < (int)kp; kk += 32)
        range_take(range, tile[kk * kShortPad + warp]);
    range             = range_warp(range);
    const bool finite = range.x < 0x7f800000u;
    if (!finite) {
        range = make_uint2(0u, kNoneSmallest);
        for (int kk = lane; kk < (int)kp; kk += 32)
            range_take(range, isfinite(tile[kk * kShortPad + warp]) ? tile[kk * kShortPad + warp] : 0.0f);
        range = range_warp(range);
    }
    float scale, inverse;
    const bool ok    = half_scale(range.x, scale, inverse);
    const int64_t nn = n0 + warp;
    if (nn >= n)
        return;
    for (int kk = lane * 2; kk < (int)kp; kk += 64) {
        __half2 hi, lo;
        const float v0 = tile[kk * kShortPad + warp], v1 = tile[(kk + 1) * kShortPad + warp];
        split_half_pair(v0 * scale, v1 * scale, hi, lo);
        *reinterpret_cast<__half2 *>(p.hi16 + nn * kp + kk) = hi;
        *reinterpret_cast<__half2 *>(p.lo16 + nn * kp + kk) = lo;
        if (p.hi32) {
            float2 h, l;
            split_tf32_flat(v0, h.x, l.x);
            split_tf32_flat(v1, h.y, l.y);
            *reinterpret_cast<float2 *>(p.hi32 + nn * kp + kk) = h;
            *reinterpret_cast<float2 *>(p.lo32 + nn * kp + kk) = l;
        }
    }
    bool bad = false;
    if (!finite || half_not_plain(range, scale)) {
        __syncwarp();
        bad = half_repair(in + nn, n, k, scale, p.hi16 + nn * kp, p.lo16 + nn * kp, p.exceptions, p.operand, nn, lane, 32);
    }
    if (lane == 0) {
        p.scale[nn] = bad ? -inverse : inverse;
        if (!ok)
            p.exceptions->wide = 1u;
    }
}

__global__ void __launch_bounds__(256) half_cols_short_kernel(
    const float *__restrict__ in, int64_t k, int64_t n, int64_t kp, const HalfPlanes p) {
    extern __shared__ float tile_short[];
    griddep_launch_dependents();
    griddep_wait();
    half_cols_short(tile_short, (int)blockIdx.x, in, k, n, kp, p);
}

// Both operands of a product with k <= 1024 in one launch: the first row_blocks blocks split rows of A (a warp
// per row), the others columns of B.  At these sizes a launch costs as much as the pass itself.
template <int V>
__global__ void __launch_bounds__(256) half_both_kernel(
    const float *__restrict__ a, int64_t m, int a_vec_ok, const HalfPlanes pa, int row_blocks,
    const float *__restrict__ b, int64_t n, const HalfPlanes pb, int64_t k, int64_t kp) {
    extern __shared__ float tile_short[];
    griddep_launch_dependents();
    griddep_wait();
    if ((int)blockIdx.x < row_blocks)
        half_rows<32, V>((int64_t)blockIdx.x, a, m, k, kp, pa, a_vec_ok);
    else
        half_cols_short(tile_short, (int)blockIdx.x - row_blocks, b, k, n, kp, pb);
}

// The tf32 planes of operands that float16 pairs cannot hold; returns at once where both can be held.  Blocks of 64 k
// x 64 rows, sixteen loads to a thread in flight, two blocks to an SM: with four loads the pass took 57 us for
// 4096 x 1024 x 1024, and more blocks make the idle launch longer.
struct WideOperand {
    const float *in;   // [rows][k], or [k][rows] when transposed
    int64_t rows;      // 0: nothing to do
    int transposed;
    float *hi, *lo;    // [rows][kp]
};

__global__ void __launch_bounds__(256) wide_planes_kernel(
    const HalfExceptions *__restrict__ ea, const HalfExceptions *__restrict__ eb, const WideOperand a, const WideOperand b,
    int64_t k, int64_t kp) {
    __shared__ float tile[64][65];
    griddep_launch_dependents();
    griddep_wait();
    if (!half_wide(ea, eb))
        return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int which = 0; which < 2; ++which) {
        const WideOperand &o  = which ? b : a;
        const int64_t tiles_k = (kp + 63) / 64, tiles = ((o.rows + 63) / 64) * tiles_k;
        for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int64_t r0 = t / tiles_k * 64, k0 = t % tiles_k * 64;
            float v[16]; // row r0 + ty + 8 (u >> 1), value k0 + tx + 32 (u & 1)
            if (o.transposed) {
                // value k0 + ty + 8 (u >> 1) of row r0 + tx + 32 (u & 1)
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int64_t kk = k0 + ty + 8 * (u >> 1), rr = r0 + tx + 32 * (u & 1);
                    v[u]             = (kk < k && rr < o.rows) ? o.in[kk * o.rows + rr] : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    tile[tx + 32 * (u & 1)][ty + 8 * (u >> 1)] = v[u];
                __syncthreads();
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    v[u] = tile[ty + 8 * (u >> 1)][tx + 32 * (u & 1)];
                __syncthreads();
            } else {
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int64_t rr = r0 + ty + 8 * (u >> 1), kk = k0 + tx + 32 * (u & 1);
                    v[u]             = (rr < o.rows && kk < k) ? o.in[rr * k + kk] : 0.0f;
                }
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int64_t rr = r0 + ty + 8 * (u >> 1), kk = k0 + tx + 32 * (u & 1);
                if (rr < o.rows && kk < kp) {
                    float hi, lo;
                    split_tf32_flat(v[u], hi, lo);
                    o.hi[rr * kp + kk] = hi;
                    o.lo[rr * kp + kk] = lo;
                }
            }
        }
    }
}

// tf32 planes from float16 planes (both terms convert exactly) and the exceptions, for a row range of a packed left
// operand whose right operand is wide; returns at once where the left operand is wide itself and has them already.
__global__ void __launch_bounds__(256) widen_planes_kernel(
    const HalfExceptions *__restrict__ x, int line0, const __half *__restrict__ hi16, const __half *__restrict__ lo16,
    const float *__restrict__ row_scale, int64_t rows, int64_t kp, float *__restrict__ hi32, float *__restrict__ lo32) {
    if (half_wide(x, x))
        return;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < rows * kp; i += (int64_t)gridDim.x * 256) {
        const int64_t row = i / kp;
        const float s = row_scale[row], inverse = fabsf(s);
        float hi = __half2float(hi16[i]) * inverse, lo = __half2float(lo16[i]) * kHalfLoInv * inverse;
        if (s < 0.0f)
            for (int e = 0; e < (int)x->count; ++e)
                if (x->e[e].line == (row + line0) * 2 && x->e[e].k == i - row * kp)
                    split_tf32(x->e[e].value, hi, lo);
        hi32[i] = hi;
        lo32[i] = lo;
    }
}

__global__ void __launch_bounds__(256) half_splitk_reduce_kernel(
    const float *__restrict__ partial, int splits, int64_t total, int64_t n, const float *__restrict__ bias,
    int act, float *__restrict__ out, const uint32_t *__restrict__ flags) {
    griddep_launch_dependents();
    griddep_wait();
    // the slices were not computed if an earlier failure is on record
    if (*reinterpret_cast<const volatile uint32_t *>(flags + FLAG_TIMEOUT) != 0)
        return;
    const int64_t step = (int64_t)gridDim.x * 256;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += step) {
        float v = partial[i];
#pragma unroll 4
        for (int z = 1; z < splits; ++z)
            v = __fadd_rn(v, partial[(int64_t)z * total + i]);
        if (bias)
            v = __fadd_rn(v, bias[i % n]);
        if (act == CT_ACT_RELU)
            v = __fmul_rn(v, v > 0.0f ? 1.0f : 0.0f);
        out[i] = v;
    }
}

// A plane [rows][kp] as a 2-D map whose box is row_bytes of k by box_rows rows; what lies outside reads zero.
ct_status plane_map(CUtensorMap *map, const void *base, int elem, int64_t rows, int64_t kp, int box_rows, int row_bytes) {
    const uint64_t dims[2] = {(uint64_t)kp, (uint64_t)rows}, strides[1] = {(uint64_t)kp * (uint64_t)elem};
    const uint32_t box[2]  = {(uint32_t)(row_bytes / elem), (uint32_t)box_rows};
    return elem == 4 ? encode_tiled_map_f32(map, base, 2, dims, strides, box, row_bytes)
                     : encode_tiled_map_f16(map, base, 2, dims, strides, box, row_bytes);
}

template <int BN, int CG, bool LEFT = false, bool LINES = false>
ct_status launch_half(DeviceState *st, const HalfOperand &a, const HalfOperand &b, int64_t kp, HalfGemmParams &p, int splits) {
    using C = HalfCfg<BN, CG>;
    HalfMaps maps;
    CT_TRY(plane_map(&maps.a16_hi, a.hi16, 2, a.rows, kp, kHM, C::kRowB));
    CT_TRY(plane_map(&maps.a16_lo, a.lo16, 2, a.rows, kp, kHM, C::kRowB));
    CT_TRY(plane_map(&maps.b16_hi, b.hi16, 2, b.rows, kp, C::kBRows, C::kRowB));
    CT_TRY(plane_map(&maps.b16_lo, b.lo16, 2, b.rows, kp, C::kBRows, C::kRowB));
    CT_TRY(plane_map(&maps.a32_hi, a.hi32, 4, a.rows, kp, kHM, C::kRowB));
    CT_TRY(plane_map(&maps.a32_lo, a.lo32, 4, a.rows, kp, kHM, C::kRowB));
    CT_TRY(plane_map(&maps.b32_hi, b.hi32, 4, b.rows, kp, C::kBRows, C::kRowB));
    CT_TRY(plane_map(&maps.b32_lo, b.lo32, 4, b.rows, kp, C::kBRows, C::kRowB));
    p.tiles_m           = (int)((p.m + kHM * CG - 1) / (kHM * CG));
    p.tiles_n           = (int)((p.n + BN - 1) / BN);
    const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n * splits * (p.batch > 1 ? p.batch : 1);
    if (tiles > 0x7fffffffll)
        return fail(CT_ERR_TOO_LARGE, "gemm: too many tiles");
    p.total_tiles = (int)tiles;
    p.group_m     = 16 / CG;
    static bool attr_set_dev[16] = {}; // the attribute belongs to a device's context
    if (!attr_set_dev[st->device & 15]) {
        CT_CUDA(cudaFuncSetAttribute(gemm_half_kernel<BN, CG, LEFT, LINES>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
        attr_set_dev[st->device & 15] = true;
    }
    const int units     = st->sm_count / CG;
    const unsigned grid = (unsigned)(tiles < units ? tiles : units) * CG;
    const int cluster   = p.cluster_split > 1 ? p.cluster_split : CG;
    ProfScope prof("gemm_tc");
    CT_CUDA(launch_dependent_cluster(gemm_half_kernel<BN, CG, LEFT, LINES>, cluster, dim3(grid), dim3(kHThreads), (size_t)C::kSmemBytes, stream(), maps, p));
    CT_LAUNCH_CHECK("gemm_half");
    return CT_OK;
}

} // namespace

ct_status half_split_rows(
    DeviceState *st, const float *in, int64_t k, int64_t kp, const HalfOperand &o, bool both_forms, uint32_t *zero,
    int64_t zero_count, const uint32_t *only_if) {
    const int64_t rows = o.rows;
    const int vec      = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    const HalfPlanes p = planes_of(o, both_forms);
    if (only_if) {
        CT_CUDA(launch_dependent(half_rows_left_kernel, dim3((unsigned)std::min<int64_t>(rows, st->sm_count)), dim3(256), 0, stream(), in, rows,
                                 k, kp, p, vec, only_if));
        CT_LAUNCH_CHECK("half_rows_left");
        return CT_OK;
    }
    // a warp per row while a row fits its registers (eight float4 per lane), else a block per row
#define CT_ROWS(TPR, V, GRID)                                                                                       \
    CT_CUDA(launch_dependent(half_rows_kernel<TPR, V>, dim3((unsigned)(GRID)), dim3(256), 0, stream(), in, rows, k, \
                             kp, p, vec, zero, zero_count))
    if (kp <= 512)
        CT_ROWS(32, 4, (rows + 7) / 8);
    else if (kp <= 1024)
        CT_ROWS(32, 8, (rows + 7) / 8);
    else if (kp <= 4096)
        CT_ROWS(256, 4, rows);
    else if (kp <= 8192)
        CT_ROWS(256, 8, rows);
    else
        CT_ROWS(256, 16, rows);
#undef CT_ROWS
    CT_LAUNCH_CHECK("half_rows");
    return CT_OK;
}

// in [k][n].  col_max: n words, zeroed before in stream order (unused where half_cols_is_short(k)).
bool half_cols_is_short(int64_t kp) { return kp <= kShortK; }

ct_status half_split_cols(
    DeviceState *st, const float *in, int64_t k, int64_t kp, const HalfOperand &o, bool both_forms, uint32_t *col_max) {
    const int64_t n    = o.rows;
    const HalfPlanes p = planes_of(o, both_forms);
    const unsigned strips = (unsigned)((n + 127) / 128);
    const int vec         = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    if (half_cols_is_short(kp)) {
        CT_CUDA(launch_dependent(half_cols_short_kernel, dim3((unsigned)((n + kShortCols - 1) / kShortCols)), dim3(256),
                                 (size_t)kp * kShortPad * 4, stream(), in, k, n, kp, p));
        CT_LAUNCH_CHECK("half_cols_short");
        return CT_OK;
    }
    int64_t slices = std::max<int64_t>(1, (int64_t)st->sm_count * 8 / strips);
    int64_t rows   = std::max<int64_t>(64, (k + slices - 1) / slices);
    slices         = std::max<int64_t>(1, (k + rows - 1) / rows);
    const int64_t slabs = (kp + 63) / 64;
    if (slabs > 65535 || slices > 65535)
        return fail(CT_ERR_TOO_LARGE, "gemm: k too large for the operand pre-pass");
    CT_CUDA(launch_dependent(half_col_max_kernel, dim3(strips, (unsigned)slices), dim3(256), 0, stream(), in, k, n, rows, vec, col_max));
    CT_LAUNCH_CHECK("half_col_max");
    CT_CUDA(launch_dependent(half_cols_kernel, dim3((unsigned)((n + 63) / 64), (unsigned)slabs), dim3(256), 0, stream(), in, k, n, kp, p, vec,
                             static_cast<const uint32_t *>(col_max)));
    CT_LAUNCH_CHECK("half_cols");
    return CT_OK;
}

// Both operands in one launch where k is short enough; false: the caller splits them one by one.
ct_status half_split_both(
    DeviceState *st, const float *a, const HalfOperand &oa, const float *b, const HalfOperand &ob, int64_t k, int64_t kp,
    bool both_forms, bool *done) {
    (void)st;
    *done = kp <= 1024;
    if (!*done)
        return CT_OK;
    const int64_t m = oa.rows, n = ob.rows;
    const int vec        = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0;
    const int row_blocks = (int)((m + 7) / 8);
    const unsigned grid  = (unsigned)(row_blocks + (n + kShortCols - 1) / kShortCols);
    const size_t smem    = (size_t)kp * kShortPad * 4; // at most 36 KB
    if (kp <= 512)
        CT_CUDA(launch_dependent(half_both_kernel<4>, dim3(grid), dim3(256), smem, stream(), a, m, vec, planes_of(oa, both_forms),
                                 row_blocks, b, n, planes_of(ob, both_forms), k, kp));
    else
        CT_CUDA(launch_dependent(half_both_kernel<8>, dim3(grid), dim3(256), smem, stream(), a, m, vec, planes_of(oa, both_forms),
                                 row_blocks, b, n, planes_of(ob, both_forms), k, kp));
    CT_LAUNCH_CHECK("half_both");
    return CT_OK;
}

ct_status half_wide_planes(
    DeviceState *st, const HalfExceptions *ea, const HalfExceptions *eb, const float *a, int64_t m, bool a_is_km, void *a_hi, void *a_lo, const float *b,
    int64_t n, void *b_hi, void *b_lo, int64_t k, int64_t kp) {
    const WideOperand oa{a, m, a_is_km ? 1 : 0, static_cast<float *>(a_hi), static_cast<float *>(a_lo)};
    const WideOperand ob{b, n, 1, static_cast<float *>(b_hi), static_cast<float *>(b_lo)};
    CT_CUDA(launch_dependent(wide_planes_kernel, dim3((unsigned)st->sm_count * 2), dim3(256), 0, stream(), ea, eb, oa, ob, k, kp));
    CT_LAUNCH_CHECK("wide_planes");
    return CT_OK;
}

ct_status half_widen_rows(DeviceState *st, const HalfOperand &o, int64_t kp) {
    widen_planes_kernel<<<(unsigned)st->sm_count * 4, 256, 0, stream()>>>(
        o.exceptions, (int)o.line0, static_cast<const __half *>(o.hi16), static_cast<const __half *>(o.lo16), o.scale, o.rows, kp,
        static_cast<float *>(const_cast<void *>(o.hi32)), static_cast<float *>(const_cast<void *>(o.lo32)));
    CT_LAUNCH_CHECK("widen_planes");
    return CT_OK;
}

// How many clusters of `size` CTAs of the 128 x 128 product run at the same time.
static int half_clusters(const DeviceState *st, int size) {
    static int known[16][4] = {}; // per device, by log2(size); under the entry points' lock
    int &count = known[st->device & 15][size == 8 ? 3 : size / 2];
    if (count == 0) {
        using C = HalfCfg<128, 1>;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(st->sm_count / size * size)), cfg.blockDim = dim3(kHThreads);
        cfg.dynamicSmemBytes = C::kSmemBytes;
        cfg.attrs = attr, cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(gemm_half_kernel<128, 1, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&count, gemm_half_kernel<128, 1, false, false>, &cfg) != cudaSuccess || count < 1) {
            cudaGetLastError();
            count = st->sm_count / size / 2 + 1; // not known: half of the machine
        }
    }
    return count;
}

// Tile width: 128 x 256 where such tiles fill at least half of the machine, else 128 x 128.
int gemm_tile_columns(const DeviceState *st, int64_t m, int64_t n, int64_t batch) {
    const int64_t tiles256 = ((m + kHM - 1) / kHM) * ((n + 255) / 256) * batch;
    return n > 128 && tiles256 >= st->sm_count / 2 ? 256 : 128;
}

ct_status gemm_half(
    DeviceState *st, const HalfOperand &a, const HalfOperand &b, int64_t kp, const float *bias, int act, float *out,
    bool force_wide, bool allow_splitk, const HalfBands *bands, int batch, bool bias_per_row, uint32_t *only_if) {
    const int64_t m = a.rows, n = b.rows / batch;
    const int bn    = gemm_tile_columns(st, m, n, batch);
    HalfGemmParams p{};
    p.m = m, p.n = n;
    p.batch            = batch;
    p.out_batch_stride = m * n;
    p.bias_per_row     = bias_per_row && bias ? 1 : 0;
    p.k_groups    = (int)((kp + 63) / 64);
    p.row_scale   = a.scale;
    p.col_scale   = b.scale;
    p.flags       = st->flags_dev;
    p.only_if     = only_if;
    p.a_hi = static_cast<const __half *>(a.hi16), p.a_lo = static_cast<const __half *>(a.lo16);
    p.b_hi = static_cast<const __half *>(b.hi16), p.b_lo = static_cast<const __half *>(b.lo16);
    p.kp           = (int)kp;
    p.exceptions_a = a.exceptions, p.exceptions_b = b.exceptions;
    p.a_line0      = (int)a.line0;
    p.force_wide   = force_wide ? 1 : 0;
    p.reset        = a.exceptions == st->exceptions_dev || b.exceptions == st->exceptions_dev ? st->exceptions_dev : nullptr;
    if (bands) {
        p.bands     = bands->bands;
        p.band_done = bands->done;
        for (int i = 0; i <= p.bands; ++i)
            p.band_first[i] = bands->first[i];
        for (int i = 0; i < p.bands; ++i)
            p.band_out_off[i] = bands->out_off[i];
    }
    // Few output tiles: slice k across CTAs so that more of the machine works.  Up to eight slices of a tile
    // are a cluster that adds them up itself; only where ten to sixteen tiles and a k beyond 4500 (a 12544 -> 128 layer
    // on 1153 to 2048 rows; fewer tiles with such a k take the tf32 planes) leave room for more do the partial sums go
    // through a workspace and a second launch.
    const int64_t tiles = ((m + kHM - 1) / kHM) * ((n + bn - 1) / bn);
    int splits          = 1;
    if (allow_splitk && !bands && batch == 1 && bn == 128 && tiles * 2 <= st->sm_count) {
        splits = (int)std::min<int64_t>(std::min<int64_t>(st->sm_count / tiles, p.k_groups / 8), 32);
        if (splits <= 8) {
            splits = 1;
            // at least 128 values of k each, and as many slices as whole clusters of them fit the machine at once, which
            // is fewer than its SMs would hold: 33 of four and 15 of eight (36 of four ran in two waves, 1498 x 2747 x 320
            // 57 us where two slices take 49; 16 of eight, 2000 x 1024 x 100, 32 us where four take 25)
            while (splits < 8 && tiles <= half_clusters(st, splits * 2) && p.k_groups >= splits * 4)
                splits *= 2;
            p.cluster_split = splits;
        }
        p.groups_per_split = splits > 1 ? (p.k_groups + splits - 1) / splits : 0;
        if (splits > 8)
            splits = (p.k_groups + p.groups_per_split - 1) / p.groups_per_split; // no empty slice
    }
    if (only_if && (bn != 128 || splits > 8))
        return fail(CT_ERR_INVALID, "gemm: product behind a panel not usable");
    if (splits <= 8) {
        p.bias = bias, p.act = act, p.out = out;
        if (only_if)
            return launch_half<128, 1, true>(st, a, b, kp, p, splits);
        if (bn == 256 && !bands && m > kHM) {
            const int64_t pairs = (m + 2 * kHM - 1) / (2 * kHM) * ((n + 255) / 256) * batch;
            return (n & 3) != 0 && pairs <= st->sm_count / 2 ? launch_half<256, 2, false, true>(st, a, b, kp, p, 1)
                                                             : launch_half<256, 2>(st, a, b, kp, p, 1);
        }
        return bn == 256 ? launch_half<256, 1>(st, a, b, kp, p, 1) : launch_half<128, 1>(st, a, b, kp, p, splits);
    }
    CT_TRY(ensure_ws(&st->splitk_ws, &st->splitk_ws_bytes, (size_t)splits * m * n * sizeof(float)));
    float *partial     = static_cast<float *>(st->splitk_ws);
    p.bias             = nullptr;
    p.act              = CT_ACT_NONE;
    p.out              = partial;
    CT_TRY((launch_half<128, 1>(st, a, b, kp, p, splits)));
    const int64_t total = m * n;
    const int64_t blocks = std::min<int64_t>((total + 255) / 256, (int64_t)st->sm_count * 16);
    ProfScope prof("gemm_splitk_reduce");
    CT_CUDA(launch_dependent(half_splitk_reduce_kernel, dim3((unsigned)blocks), dim3(256), 0, stream(),
                             static_cast<const float *>(partial), splits, total, n, bias, act, out,
                             static_cast<const uint32_t *>(st->flags_dev)));
    CT_LAUNCH_CHECK("half_splitk_reduce");
    return CT_OK;
}

} // namespace ct
