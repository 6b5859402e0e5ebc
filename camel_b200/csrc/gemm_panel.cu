// Tall float32 products with at most 128 columns and a long k: C[m,n] = act(A[m,k] . B[k,n] + bias), A read once, as it is.
//
// With one tile of columns every value of A belongs to one tile, so writing A's float16 planes first (8 bytes of traffic for
// each 4-byte value) and reading them again (4) was two thirds of the time: 8192 x 12544 x 128 took 130 us of pre-pass and 120 us
// of product.  Here sixteen warps load A in chunks of 128 rows by 128 values of k into registers, split them into float16
// pairs (half_split.cuh) in shared memory and, one chunk behind, add the chunk's sums to their own.  A scale has to be constant
// along the values that an accumulator sums, so each row of each chunk has its own, and the accumulators - one set
// computes while the other is read - are drained every chunk, in float32 with round-to-nearest adds.  B's planes come
// by TMA as for the other products; the slices of a tile's k are CTAs of a cluster, which add up through distributed
// shared memory.  8192 x 12544 x 128: 261 -> 184 us, 9000 x 2100 x 64: 64 -> 56.  What bounds it: what the SMs draw from L2, 64 KB of
// A and 64 KB of B's planes a chunk, 4600 clocks at the 28 bytes a clock that each SM gets when all draw; a chunk takes about 5800,
// where A alone from memory would take 2480.
//
// Values of A that float16 pairs cannot hold are listed, zeros in their place, and their products with B's row added to the sums
// in float32, B's own list likewise.  More than the lists hold, infinities, NaN or exponents beyond the scales leave a mark:
// the kernels that are launched behind this one return at once where there is none and compute the whole product from
// planes otherwise.
#include "common.cuh"
#include "half_split.cuh"
#include "tc_ptx.cuh"
#include "tmap.cuh"

#include <algorithm>

namespace ct {
namespace {

using namespace ptx;

constexpr int kGP_Workers = 16;
constexpr int kGP_Threads = 64 + 32 * kGP_Workers;
constexpr int kGP_K       = 128;              // values of k of a chunk
constexpr int kGP_Block   = 128 * 128;        // bytes: 128 rows of 64 values
constexpr int kGP_Plane   = 2 * kGP_Block;
constexpr int kGP_Buffer  = 2 * kGP_Plane;    // A hi and lo of a chunk; two of them
constexpr int kGP_BStages = 3;                // 64 values of k each, hi and lo
constexpr int kGP_B       = 2 * kGP_Buffer;
constexpr int kGP_Listed  = 16;               // exceptions of a CTA's part of A
constexpr int kGP_Smem    = kGP_B + kGP_BStages * 2 * kGP_Block; // with the static 3 KB all that a CTA can have

struct PanelParams {
    const float *a, *bias, *col_scale;
    const __half *b_hi, *b_lo; // the planes [n][kp]
    int64_t kp;
    float *out;
    int64_t m, n, k;
    int chunks, chunks_each, slices; // chunks of k, and of a slice
    int act, vec_a, vec_out;
    const HalfExceptions *exceptions_b;
    uint32_t *flags;
};

struct PanelException {
    int row, chunk_k; // row of the tile, position in the slice
    float value;
};

__global__ void __launch_bounds__(kGP_Threads, 1) gemm_panel_kernel(
    const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, const __grid_constant__ PanelParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ uint64_t bar_a_full[2], bar_a_empty[2], bar_acc_full[2], bar_acc_empty[2];
    __shared__ uint64_t bar_b_full[kGP_BStages], bar_b_empty[kGP_BStages], bar_done;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s, leave_s, listed_s;
    __shared__ PanelException list_s[kGP_Listed];
    __shared__ float row_inv[4][128]; // of a chunk's rows: written before its MMAs, read until the chunk after the next is multiplied
    volatile int *abort_flag = &abort_flag_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = smem_u32(smem_raw);
    uint8_t *smem            = smem_raw;

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_a_full[b]), kGP_Workers);
            mbar_init(smem_u32(&bar_a_empty[b]), 1);
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), kGP_Workers);
        }
        for (int s = 0; s < kGP_BStages; ++s) {
            mbar_init(smem_u32(&bar_b_full[s]), 1);
            mbar_init(smem_u32(&bar_b_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_done), 1);
        mbar_fence_init();
        prefetch_tensormap(&map_hi);
        prefetch_tensormap(&map_lo);
        abort_flag_s = 0;
        listed_s     = 0;
    }
    griddep_wait();
    if (threadIdx.x == 0) {
        // whether an earlier launch failed (no work, but the cluster's CTAs stay together), or B is not for this kernel
        const bool b_bad  = half_wide(p.exceptions_b, p.exceptions_b);
        const bool failed = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0;
        if (b_bad && blockIdx.x == 0)
            p.flags[FLAG_PANEL] = 1u;
        leave_s = b_bad ? 2 : (failed ? 1 : 0);
    }
    __syncthreads();
    const bool failed = leave_s == 1;
    if (leave_s == 2)
        return;
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    const int rank = (int)(blockIdx.x % p.slices);
    const int64_t row0 = (int64_t)(blockIdx.x / p.slices) * 128;
    const int chunk0 = rank * p.chunks_each;
    const int chunks = failed || p.chunks - chunk0 < 0 ? 0 : (p.chunks - chunk0 < p.chunks_each ? p.chunks - chunk0 : p.chunks_each);

    // worker warps: rows 8 w .. of the chunks, and 32 rows by 32 columns of the sums
    const int w = warp - 2, quarter = warp & 3, cg = w >> 2;
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j)
        acc[j] = 0.0f;
    bool ok = true;
    if (warp == 0) {
        // ===== B's planes =====
        if (elect_one()) {
            int i = 0;
            for (; i < 2 * chunks; ++i) {
                const int s = i % kGP_BStages;
                if (!mbar_wait(smem_u32(&bar_b_empty[s]), ((uint32_t)(i / kGP_BStages) & 1u) ^ 1u, abort_flag))
                    break;
                const uint32_t full = smem_u32(&bar_b_full[s]), dst = smem_base + (uint32_t)(kGP_B + s * 2 * kGP_Block);
                const int32_t kc = chunk0 * kGP_K + i * 64;
                mbar_expect_tx(full, 2u * kGP_Block);
                tma_load_2d(dst, &map_hi, full, kc, 0);
                tma_load_2d(dst + kGP_Block, &map_lo, full, kc, 0);
            }
            if (*abort_flag) // let the copies still in flight land before the CTA goes away
                for (int k2 = i - kGP_BStages < 0 ? 0 : i - kGP_BStages; k2 < i; ++k2) {
                    const uint64_t t0 = globaltimer_ns();
                    while (!mbar_try_wait(smem_u32(&bar_b_full[k2 % kGP_BStages]), (uint32_t)(k2 / kGP_BStages) & 1u) &&
                           globaltimer_ns() - t0 < kWaitBudgetNs) {
                    }
                }
        }
    } else if (warp == 1) {
        // ===== MMA issuer =====
        if (elect_one()) {
            const uint32_t idesc = make_idesc(0u, 128, 128);
            bool go = true;
            for (int c = 0, i = 0; c < chunks && go; ++c) {
                const int b = c & 1;
                const uint32_t d_main = tmem_base + (uint32_t)(b * 256), d_cross = d_main + 128u;
                go = mbar_wait(smem_u32(&bar_acc_empty[b]), ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag) &&
                     mbar_wait(smem_u32(&bar_a_full[b]), (uint32_t)(c >> 1) & 1u, abort_flag);
                for (int h = 0; h < 2 && go; ++h, ++i) {
                    const int s = i % kGP_BStages;
                    go          = mbar_wait(smem_u32(&bar_b_full[s]), (uint32_t)(i / kGP_BStages) & 1u, abort_flag);
                    if (!go)
                        break;
                    tc_fence_after_sync();
                    const uint64_t ah = smem_desc_k<128>(smem_base + (uint32_t)(b * kGP_Buffer + h * kGP_Block));
                    const uint64_t bh = smem_desc_k<128>(smem_base + (uint32_t)(kGP_B + s * 2 * kGP_Block));
                    const uint64_t al = ah + (kGP_Plane >> 4), bl = bh + (kGP_Block >> 4);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        mma_f16(d_cross, al + 2 * kk, bh + 2 * kk, idesc, h || kk ? 1u : 0u);
                        mma_f16(d_main, ah + 2 * kk, bh + 2 * kk, idesc, h || kk ? 1u : 0u);
                        mma_f16(d_cross, ah + 2 * kk, bl + 2 * kk, idesc, 1u);
                    }
                    tc_commit(smem_u32(&bar_b_empty[s]));
                }
                if (go) {
                    tc_commit(smem_u32(&bar_a_empty[b]));
                    tc_commit(smem_u32(&bar_acc_full[b]));
                }
            }
            if (!go || *abort_flag) {
                tc_commit(smem_u32(&bar_done));
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bar_done), 0) && globaltimer_ns() - t0 < kWaitBudgetNs) {
                }
            }
        }
    } else {
        // ===== workers =====
        float4 v[8];
        auto load = [&](int c) {
            const int64_t k0 = (int64_t)(chunk0 + c) * kGP_K + 4 * lane;
            const int left   = (int)(p.k - k0 < 4 ? (p.k - k0 < 0 ? 0 : p.k - k0) : 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int64_t row = row0 + w * 8 + i;
                const float *src  = p.a + row * p.k + k0;
                const int take    = c < chunks && row < p.m ? left : 0;
                if (p.vec_a) {
                    v[i] = take ? __ldcs(reinterpret_cast<const float4 *>(src)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                } else {
                    v[i].x = take > 0 ? src[0] : 0.0f, v[i].y = take > 1 ? src[1] : 0.0f;
                    v[i].z = take > 2 ? src[2] : 0.0f, v[i].w = take > 3 ? src[3] : 0.0f;
                }
            }
        };
        // the lines of a chunk, four to a row, brought into L2 ahead of the loads, which have registers for one chunk only
        auto prefetch = [&](int c) {
            const int64_t row = row0 + w * 8 + (lane >> 2), k0 = (int64_t)(chunk0 + c) * kGP_K + (lane & 3) * 32;
            if (c < chunks && row < p.m && k0 < p.k)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.a + row * p.k + k0));
        };
        auto drain = [&](int c) {
            const int b    = c & 1;
            const bool got = mbar_wait(smem_u32(&bar_acc_full[b]), (uint32_t)(c >> 1) & 1u, abort_flag);
            ok             = __all_sync(0xffffffffu, got) != 0;
            if (!ok)
                return;
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 256 + cg * 32);
            const float rs       = row_inv[c & 3][quarter * 32 + lane];
#pragma unroll
            for (int h = 0; h < 32; h += 16) {
                uint32_t x[16], y[16];
                tmem_ld_32x16(taddr + h, x);
                tmem_ld_32x16(taddr + 128 + h, y);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) // the products with powers of two are exact
                    acc[h + j] = __fmaf_rn(__fmaf_rn(__uint_as_float(y[j]), kHalfLoInv, __uint_as_float(x[j])), rs, acc[h + j]);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&bar_acc_empty[b]));
        };
        prefetch(1);
        prefetch(2);
        load(0);
        bool bad = false;
        for (int c = 0; c < chunks && ok; ++c) {
            const int b = c & 1;
            ok          = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_a_empty[b]), ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag)) != 0;
            if (!ok)
                break;
            uint8_t *dst = smem + b * kGP_Buffer + (lane >> 4) * kGP_Block + w * 8 * 128 + (lane & 1) * 8;
            // the largest magnitudes of the eight rows; lane i has the scale of row i & 7 and the smallest magnitude it takes
            uint32_t top = 0, low[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint2 r = make_uint2(0u, kNoneSmallest);
                range_take(r, v[i].x), range_take(r, v[i].y), range_take(r, v[i].z), range_take(r, v[i].w);
                const uint32_t all = __reduce_max_sync(0xffffffffu, r.x);
                top                = (lane & 7) == i ? all : top;
                low[i]             = r.y;
            }
            float scale, inverse;
            bad |= !half_scale(top, scale, inverse) || top >= 0x7f800000u;
            const uint32_t smallest = __float_as_uint(__fmul_rn(kHalfSmallest, inverse)) - 1u;
            if (lane < 8)
                row_inv[c & 3][w * 8 + lane] = inverse;
            bool small = false;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                small |= low[i] < __shfl_sync(0xffffffffu, smallest, i);
            if (__any_sync(0xffffffffu, small)) { // rare
                auto take = [&](float &x, int i, int q) {
                    const float s = __shfl_sync(0xffffffffu, scale, i);
                    if (!half_exception(x, s))
                        return;
                    const int at = atomicAdd(&listed_s, 1);
                    if (at < kGP_Listed)
                        list_s[at] = PanelException{w * 8 + i, c * kGP_K + 4 * lane + q, x};
                    else
                        bad = true;
                    x = 0.0f;
                };
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    take(v[i].x, i, 0), take(v[i].y, i, 1), take(v[i].z, i, 2), take(v[i].w, i, 3);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float s = __shfl_sync(0xffffffffu, scale, i);
                __half2 hi[2], lo[2];
                split_half_pair(v[i].x * s, v[i].y * s, hi[0], lo[0]);
                split_half_pair(v[i].z * s, v[i].w * s, hi[1], lo[1]);
                uint8_t *at = dst + i * 128 + ((((lane & 15) >> 1) ^ i) << 4); // 128-byte swizzle; row & 7 = i
                *reinterpret_cast<uint2 *>(at)             = *reinterpret_cast<uint2 *>(hi);
                *reinterpret_cast<uint2 *>(at + kGP_Plane) = *reinterpret_cast<uint2 *>(lo);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // written here, read by the tensor core
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&bar_a_full[b]));
            prefetch(c + 3);
            // one half of the warps loads while the other drains: 8192 x 12544 x 128 184 us, 194 with all in one order
            const bool later = (w >> 2) & 1;
            if (!later)
                load(c + 1);
            if (c > 0)
                drain(c - 1);
            if (later)
                load(c + 1);
        }
        if (ok && chunks > 0)
            drain(chunks - 1);
        if (bad)
            p.flags[FLAG_PANEL] = 1u;
    }
    __syncthreads(); // the list is complete
    if (warp >= 2) {
// What the sums lack, before their column scales: A's exceptions times B's planes, A times B's exceptions.  Both in order of
        // k, whatever order the lists were filled in: that varies from run to run.
        const int row = quarter * 32 + lane, listed = listed_s < kGP_Listed ? listed_s : kGP_Listed;
        for (int after = -1;;) {
            int next = -1;
            for (int i = 0; i < listed; ++i)
                if (list_s[i].row == row && list_s[i].chunk_k > after && (next < 0 || list_s[i].chunk_k < list_s[next].chunk_k))
                    next = i;
            if (next < 0)
                break;
            const PanelException x = list_s[next];
            const int64_t kk = (int64_t)chunk0 * kGP_K + x.chunk_k;
            after            = x.chunk_k;
#pragma unroll 1
            for (int j = 0; j < 32 && cg * 32 + j < p.n; ++j) {
                const int64_t at = (cg * 32 + j) * p.kp + kk;
                const float b    = __half2float(p.b_hi[at]) + __half2float(p.b_lo[at]) * kHalfLoInv;
#pragma unroll
                for (int q = 0; q < 32; ++q) // no index that is not constant: the sums would leave their registers for the whole kernel
                    acc[q] = q == j ? __fmaf_rn(x.value, b, acc[q]) : acc[q];
            }
        }
        const int listed_b = (int)p.exceptions_b->count;
        const int64_t first = (int64_t)chunk0 * kGP_K, last = first + (int64_t)chunks * kGP_K;
        for (int64_t after = first - 1;;) {
            int64_t next = last;
            for (int i = 0; i < listed_b; ++i) {
                const HalfException x = p.exceptions_b->e[i];
                if ((x.line & 1) && x.line >> 6 == cg && x.k > after && x.k < next)
                    next = x.k;
            }
            if (next == last)
                break;
            after = next;
            for (int i = 0; i < listed_b; ++i) { // a column each
                const HalfException x = p.exceptions_b->e[i];
                const int col = x.line >> 1;
                if (!(x.line & 1) || x.line >> 6 != cg || x.k != next || row0 + row >= p.m)
                    continue;
                const float add = __fmul_rn(p.a[(row0 + row) * p.k + x.k], x.value / fabsf(p.col_scale[col]));
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    acc[j] = (col & 31) == j ? __fadd_rn(acc[j], add) : acc[j];
            }
        }
    }

    // ---- the slices' sums: rows of 512 bytes, float4 slots XOR-swizzled, slice after slice, to the CTA that adds them up ----
    __syncwarp();
    cluster_sync(); // every MMA of every slice has been read: the operands' memory is free
    const int rows_each = 128 / p.slices;
    if (warp >= 2) {
        const int row       = quarter * 32 + lane;
        const uint32_t part = mapa(smem_base + (uint32_t)((rank * rows_each + row % rows_each) * 512), (uint32_t)(row / rows_each));
#pragma unroll
        for (int j = 0; j < 8; ++j)
            st_cluster_f4(part + (uint32_t)(((cg * 8 + j) ^ (row & 7)) << 4), make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
    }
    tc_fence_before_sync();
    __syncwarp();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
    const int64_t col = lane * 4;
    float c4[4], b4[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        c4[q] = col + q < p.n ? fabsf(p.col_scale[col + q]) : 1.0f;
        b4[q] = p.bias && col + q < p.n ? p.bias[col + q] : 0.0f;
    }
    if (!failed && !*abort_flag && col < p.n)
        for (int r = warp; r < rows_each; r += kGP_Threads / 32) {
            const int64_t row = row0 + rank * rows_each + r;
            if (row >= p.m)
                break;
            const uint8_t *at = smem + r * 512 + ((lane ^ (r & 7)) << 4);
            float4 s          = *reinterpret_cast<const float4 *>(at);
            for (int z = 1; z < p.slices; ++z) {
                const float4 q = *reinterpret_cast<const float4 *>(at + z * rows_each * 512);
                s = make_float4(__fadd_rn(s.x, q.x), __fadd_rn(s.y, q.y), __fadd_rn(s.z, q.z), __fadd_rn(s.w, q.w));
            }
            float x[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[q] = __fmul_rn(x[q], c4[q]);
                if (p.bias)
                    x[q] = __fadd_rn(x[q], b4[q]);
                if (p.act == CT_ACT_RELU)
                    x[q] = __fmul_rn(x[q], x[q] > 0.0f ? 1.0f : 0.0f);
            }
            float *dst = p.out + row * p.n + col;
            if (p.vec_out) {
                *reinterpret_cast<float4 *>(dst) = make_float4(x[0], x[1], x[2], x[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (col + q < p.n)
                        dst[q] = x[q];
            }
        }
    if (threadIdx.x == 0 && *abort_flag)
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

// How many clusters of `size` CTAs run at the same time.
int panel_clusters(const DeviceState *st, int size) {
    static int known[16][4] = {}; // per device, by log2(size); under the entry points' lock
    int &count = known[st->device & 15][size == 8 ? 3 : size / 2];
    if (count == 0) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(st->sm_count / size * size)), cfg.blockDim = dim3(kGP_Threads);
        cfg.dynamicSmemBytes = kGP_Smem;
        cfg.attrs = attr, cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(gemm_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGP_Smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&count, gemm_panel_kernel, &cfg) != cudaSuccess || count < 1) {
            cudaGetLastError();
            count = -1; // not known: the other kernels
        }
    }
    return count;
}

// Slices of k; 0: the product is not for this kernel.  It takes those with one tile of columns whose k is sliced (the others
// have the bytes of ct_matmul_packed_rows), which fill two thirds of the machine, and where A is most of the work.  With slices
// a power of two, and 74 clusters of two, 33 of four and 15 of eight at once, that is 25 to 33 row tiles where k is 4096 and
// more, and 50 to 74 from 2048 on.
int panel_slices(const DeviceState *st, int64_t m, int64_t k, int64_t n) {
    const int64_t tiles = (m + 127) / 128;
    if (n > 128 || k < 2048 || tiles * 2 > st->sm_count || st->sm_count / tiles > 8) // gemm_half, behind it, would use more slices than a cluster has
        return 0;
    int slices = 2;
    while (slices < 8 && tiles <= panel_clusters(st, slices * 2) && k >= slices * 2 * 1024)
        slices *= 2;
    return tiles <= panel_clusters(st, slices) && tiles * slices * 3 >= st->sm_count * 2 ? slices : 0;
}

} // namespace

bool gemm_panel_applicable(const DeviceState *st, int64_t m, int64_t k, int64_t n) { return panel_slices(st, m, k, n) > 0; }

ct_status gemm_panel(
    DeviceState *st, const float *a, const HalfOperand &b, int64_t kp, const float *bias, int64_t m, int64_t k, int64_t n, int act, float *out) {
    CUtensorMap maps[2];
    const uint64_t dims[2] = {(uint64_t)kp, (uint64_t)n}, strides[1] = {(uint64_t)kp * 2};
    const uint32_t box[2]  = {64, 128};
    CT_TRY(encode_tiled_map_f16(&maps[0], b.hi16, 2, dims, strides, box, 128));
    CT_TRY(encode_tiled_map_f16(&maps[1], b.lo16, 2, dims, strides, box, 128));
    auto aligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    PanelParams p{};
    p.a = a, p.bias = bias, p.col_scale = b.scale, p.out = out;
    p.m = m, p.n = n, p.k = k;
    p.slices      = panel_slices(st, m, k, n);
    p.chunks      = (int)((k + kGP_K - 1) / kGP_K);
    p.chunks_each = (p.chunks + p.slices - 1) / p.slices;
    p.act   = act;
    p.vec_a = (k & 3) == 0 && aligned(a), p.vec_out = (n & 3) == 0 && aligned(out);
    p.b_hi = static_cast<const __half *>(b.hi16), p.b_lo = static_cast<const __half *>(b.lo16), p.kp = kp;
    p.exceptions_b = b.exceptions;
    p.flags        = st->flags_dev;
    const unsigned grid = (unsigned)((m + 127) / 128 * p.slices);
    ProfScope prof("gemm_tc");
    CT_CUDA(launch_dependent_cluster(gemm_panel_kernel, p.slices, dim3(grid), dim3(kGP_Threads), (size_t)kGP_Smem, stream(), maps[0], maps[1], p));
    CT_LAUNCH_CHECK("gemm_panel");
    return CT_OK;
}

} // namespace ct
