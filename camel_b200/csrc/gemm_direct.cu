// Small float32 products in one launch: C[m,n] = act(A[m,k] . B[k,n] + bias) straight from float32 operands.
//
// A product of a few tiles is latency: the pre-pass that writes operand planes, the wait for it and a pipeline that fetches
// them again took 15 us at 512 x 512 x 512, of which the MMAs are one.  Here a CTA has one 128 x 128 tile and at most 128
// values of k; it loads its float32 operands once into registers (sixteen 16-byte loads a thread, all in flight), splits
// them into float16 pairs in shared memory and multiplies; the CTAs of a cluster are the slices of a tile's k and add up
// through distributed shared memory: 15.3 -> 8.7 us, a 64-sample request of two hidden layers and a classifier 36 -> 24.6.  A's
// planes are K-major, B's stay as they lie (rows of n, an MN-major operand), so nothing is transposed.
//
// What bounds it is the chain: operands 1.4 us after the wait, their ranges 1.1, planes 1.3, the last MMA 0.7 behind them, sums
// to the others 2.0, added up and stored 0.6.  So nothing is done for rows and columns that a tile does not have (a tile
// of 64 columns has every lane of B's loads at work, of 64 rows half of A's), a range takes two instructions a value,
// and the first half of k is multiplied while B's second half is written: 9.6 -> 9.3 us and 25.9 -> 24.6.
//
// A scale has to be constant along the values that one accumulator sums, here the slice: the rows of A and the columns
// of B are scaled by their largest magnitude in the slice, which can only hold more than the whole row's.  A slice with
// a value that float16 pairs cannot hold (half_split.cuh), an infinity or a NaN is multiplied in three bfloat16 terms
// instead, which have float32's exponents: h.h, the cross products h.m, m.h, m.m, and in a second round h.l and l.h with
// the l terms where the m terms were.  Every CTA decides that for itself.
#include "common.cuh"
#include "half_split.cuh"
#include "tc_ptx.cuh"

#include <algorithm>

#include <cuda_bf16.h>

namespace ct {
namespace {

using namespace ptx;

constexpr int kGD_Threads = 512, kGD_Warps = kGD_Threads / 32;
constexpr int kGD_K       = 128;                      // values of k of a slice
constexpr int kGD_Block   = 128 * 128;                // bytes: 128 rows of 64 values of k (A), 128 k of 64 columns (B)
constexpr int kGD_Plane   = 2 * kGD_Block;
constexpr int kGD_B       = 2 * kGD_Plane;            // A hi, A lo, B hi, B lo
constexpr int kGD_Sums    = 4 * kGD_Plane;            // 64 KB that the cluster's CTAs send
constexpr int kGD_Ranges  = kGD_Sums + 128 * 128 * 4; // of the columns, a row of them per warp
constexpr int kGD_Smem    = kGD_Ranges + kGD_Warps * 128 * 8 + 1024;

struct DirectParams {
    const float *a, *b, *bias;
    float *out;
    int64_t m, n, k;
    int kc, slices, tiles_m, bn; // values of k per slice, a multiple of 16; columns of a tile, 64 or 128
    int act, vec_a, vec_b, vec_out;
    uint32_t *flags;
};

// Start address >> 4; leading byte offset: the next 64 columns; stride byte offset: the next 8 values of k; 128-byte swizzle.
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)(kGD_Block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// The range of half_split.cuh in half the instructions: .x the largest magnitude (7fffffff once there is a NaN), .y twice the
// bits of the smallest non-zero one less 1 (all ones: there is none).
__device__ __forceinline__ void range_take_two(uint2 &r, float v, float w) {
    float m;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(__uint_as_float(r.x)), "f"(fabsf(v)), "f"(fabsf(w)));
    r.x = __float_as_uint(m);
    r.y = __vimin3_u32(r.y, 2u * __float_as_uint(v) - 1u, 2u * __float_as_uint(w) - 1u);
}

__global__ void __launch_bounds__(kGD_Threads, 1) gemm_direct_kernel(const __grid_constant__ DirectParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag_s, wide_s;
    __shared__ float row_inv[128];
    __shared__ __align__(16) float col_scale[128], col_inv[128];
    volatile int *abort_flag = &abort_flag_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem            = smem_raw + (smem_base - smem_u32(smem_raw));
    uint2(*ranges)[128]      = reinterpret_cast<uint2(*)[128]>(smem + kGD_Ranges);

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        wide_s = 0;
        mbar_init(smem_u32(&bar), 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_base_slot), 256);
        tmem_relinquish();
    }
    const int rank = (int)(blockIdx.x % p.slices), tile = (int)(blockIdx.x / p.slices);
    const int64_t row0 = (int64_t)(tile % p.tiles_m) * 128, col0 = (int64_t)(tile / p.tiles_m) * p.bn, k0 = (int64_t)rank * p.kc;
    const int kn     = (int)(p.k - k0 < 0 ? 0 : (p.k - k0 < p.kc ? p.k - k0 : p.kc)); // the last slices may be empty
    const int ksteps = (kn + 15) >> 4;
    cluster_arrive(); // this CTA runs: the others may write to its shared memory
    griddep_wait();
    if (threadIdx.x == 0)
        abort_flag_s = *reinterpret_cast<volatile uint32_t *>(p.flags + FLAG_TIMEOUT) != 0 ? 1 : 0;

    // ---- the operands: a warp has eight rows of A, a lane four values of k; four values of k of each half of B, a lane four
    // columns, or in a tile of 64 columns a half of the warp the even ones of those k and the other the odd ones ----
    const int valid   = (int)(p.m - row0 < 128 ? p.m - row0 : 128);
    const bool narrow = p.bn == 64, has_rows = warp * 8 < valid;
    const int quad    = narrow ? lane & 15 : lane; // the lane's columns
    auto k_of         = [&](int i) { return narrow ? (i >> 1) * 64 + warp * 4 + (i & 1) * 2 + (lane >> 4) : (i >> 2) * 64 + warp * 4 + (i & 3); };
    float4 av[8], bv[8];
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t row = row0 + warp * 8 + i;
        const float *src  = p.a + row * p.k + k0 + 4 * lane;
        const int left    = row < p.m ? kn - 4 * lane : 0;
        if (p.vec_a) {
            av[i] = left > 0 ? *reinterpret_cast<const float4 *>(src) : zero;
        } else {
            av[i].x = left > 0 ? src[0] : 0.0f, av[i].y = left > 1 ? src[1] : 0.0f;
            av[i].z = left > 2 ? src[2] : 0.0f, av[i].w = left > 3 ? src[3] : 0.0f;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int kk     = k_of(i);
        const float *src = p.b + (k0 + kk) * p.n + col0 + 4 * quad;
        const int left   = kk < kn && (i < 4 || !narrow) ? (int)(p.n - col0 < p.bn ? p.n - col0 : p.bn) - 4 * quad : 0;
        if (p.vec_b) {
            bv[i] = left > 0 ? *reinterpret_cast<const float4 *>(src) : zero;
        } else {
            bv[i].x = left > 0 ? src[0] : 0.0f, bv[i].y = left > 1 ? src[1] : 0.0f;
            bv[i].z = left > 2 ? src[2] : 0.0f, bv[i].w = left > 3 ? src[3] : 0.0f;
        }
    }

    // ---- their ranges ----
    auto plain = [](uint2 r, float &scale, float &inverse) {
        const bool ok = half_scale(r.x, scale, inverse);
        return ok && r.x < 0x7f800000u && (r.y == kNoneSmallest || __uint_as_float((r.y + 1u) >> 1) * scale >= kHalfSmallest);
    };
    float a_scale[8];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint2 r = make_uint2(0u, kNoneSmallest);
        if (!has_rows)
            break;
        range_take_two(r, av[i].x, av[i].y), range_take_two(r, av[i].z, av[i].w);
        float inverse;
        bad |= !plain(range_warp(r), a_scale[i], inverse);
        if (lane == 0)
            row_inv[warp * 8 + i] = inverse;
    }
    {
        uint2 r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            r[q] = make_uint2(0u, kNoneSmallest);
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            if (i == 4 && narrow)
                break;
            range_take_two(r[0], bv[i].x, bv[i + 1].x), range_take_two(r[1], bv[i].y, bv[i + 1].y);
            range_take_two(r[2], bv[i].z, bv[i + 1].z), range_take_two(r[3], bv[i].w, bv[i + 1].w);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            ranges[warp][4 * lane + q] = r[q];
    }
    __syncthreads();
    if ((int)threadIdx.x < p.bn) {
        uint2 r = ranges[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < kGD_Warps; ++w)
            r = range_join(r, ranges[w][threadIdx.x]);
        if (narrow) // the odd values of k
#pragma unroll
            for (int w = 0; w < kGD_Warps; ++w)
                r = range_join(r, ranges[w][64 + threadIdx.x]);
        float scale, inverse;
        bad |= !plain(r, scale, inverse);
        col_scale[threadIdx.x] = scale, col_inv[threadIdx.x] = inverse;
    }
    if (bad)
        wide_s = 1;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const bool wide   = wide_s != 0;
    const bool failed = abort_flag_s != 0;
    const uint32_t tmem_base = tmem_base_slot;

    // ---- their planes: rows of 128 bytes, 128-byte swizzle; a lane has eight bytes of a row ----
    auto put = [&](int plane, int block, int row, uint2 v) {
        *reinterpret_cast<uint2 *>(smem + plane * kGD_Plane + block * kGD_Block + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8) = v;
    };
    auto put_a = [&](int plane, int i, uint2 v) { put(plane, lane >> 4, warp * 8 + i, v); };
    auto put_b = [&](int plane, int i, uint2 v) { put(2 + plane, narrow ? 0 : lane >> 4, k_of(i), v); };
    auto bf16_terms = [](float v, float &h, float &m, float &l) { // v = h + m + l exactly, for finite v
        const bool finite = isfinite(v);
        h = finite ? __uint_as_float(__float_as_uint(v) & 0xffff0000u) : v; // truncated: rounding could reach infinity
        const float d = v - h;
        m = finite ? __bfloat162float(__float2bfloat16_rn(d)) : 0.0f;
        l = finite ? d - m : 0.0f;
    };
    auto bf16_pair = [](float x, float y, float z, float w) {
        __nv_bfloat162 q[2] = {__floats2bfloat162_rn(x, y), __floats2bfloat162_rn(z, w)};
        return *reinterpret_cast<uint2 *>(q);
    };
    auto split_bf16 = [&](auto &&to, int i, const float4 &v, bool last) {
        float h[4], m[4], l[4];
        bf16_terms(v.x, h[0], m[0], l[0]), bf16_terms(v.y, h[1], m[1], l[1]);
        bf16_terms(v.z, h[2], m[2], l[2]), bf16_terms(v.w, h[3], m[3], l[3]);
        if (last) {
            to(1, i, bf16_pair(l[0], l[1], l[2], l[3]));
        } else {
            to(0, i, bf16_pair(h[0], h[1], h[2], h[3]));
            to(1, i, bf16_pair(m[0], m[1], m[2], m[3]));
        }
    };
    auto split_bf16_all = [&](bool last) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (has_rows)
                split_bf16(put_a, i, av[i], last);
            if (i < 4 || !narrow)
                split_bf16(put_b, i, bv[i], last);
        }
    };

    // ---- the product: leading accumulator in columns 0 .. 127, cross products behind it ----
    const uint32_t d_main = tmem_base, d_cross = tmem_base + 128u;
    const uint32_t idesc  = make_idesc(wide ? 1u : 0u, 128, (uint32_t)p.bn) | 1u << 16; // B is MN-major
    auto a_desc = [&](int plane, int ks) { return smem_desc_k<128>(smem_base + (uint32_t)(plane * kGD_Plane + (ks >> 2) * kGD_Block)) + 2 * (ks & 3); };
    auto b_desc = [&](int plane, int ks) { return desc_mn(smem_base + (uint32_t)(kGD_B + plane * kGD_Plane + ks * 2048)); };
    auto mma    = [&](int ks) {
        const uint64_t ah = a_desc(0, ks), al = a_desc(1, ks), bh = b_desc(0, ks), bl = b_desc(1, ks);
        mma_f16(d_cross, al, bh, idesc, ks > 0);
        mma_f16(d_main, ah, bh, idesc, ks > 0);
        mma_f16(d_cross, ah, bl, idesc, 1u);
        if (wide)
            mma_f16(d_cross, al, bl, idesc, 1u);
    };
    bool ok = !failed;
    if (!wide) {
        // The first 64 values of k are multiplied while B's others are written.
        const float4 s = *reinterpret_cast<const float4 *>(col_scale + 4 * quad);
        auto split_b   = [&](int i) {
            __half2 hi[2], lo[2];
            split_half_pair(bv[i].x * s.x, bv[i].y * s.y, hi[0], lo[0]);
            split_half_pair(bv[i].z * s.z, bv[i].w * s.w, hi[1], lo[1]);
            put_b(0, i, *reinterpret_cast<uint2 *>(hi));
            put_b(1, i, *reinterpret_cast<uint2 *>(lo));
        };
        if (has_rows)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                __half2 hi[2], lo[2];
                split_half_pair(av[i].x * a_scale[i], av[i].y * a_scale[i], hi[0], lo[0]);
                split_half_pair(av[i].z * a_scale[i], av[i].w * a_scale[i], hi[1], lo[1]);
                put_a(0, i, *reinterpret_cast<uint2 *>(hi));
                put_a(1, i, *reinterpret_cast<uint2 *>(lo));
            }
        split_b(0), split_b(1);
        if (!narrow)
            split_b(2), split_b(3);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // written here, read by the tensor core
        __syncthreads();
        if (ok && warp == 0 && elect_one())
            for (int ks = 0; ks < ksteps && ks < 4; ++ks)
                mma(ks);
        if (narrow)
            split_b(2), split_b(3);
        else
            split_b(4), split_b(5), split_b(6), split_b(7);
    } else {
        split_bf16_all(false);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (ok && ksteps > 0) {
        if (warp == 0 && elect_one()) {
            for (int ks = wide ? 0 : 4; ks < ksteps; ++ks)
                mma(ks);
            tc_commit(smem_u32(&bar));
        }
        ok = mbar_wait(smem_u32(&bar), 0u, abort_flag);
        tc_fence_after_sync();
        if (wide) {
            __syncthreads();
            split_bf16_all(true);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            if (warp == 0 && elect_one()) {
                for (int ks = 0; ks < ksteps; ++ks) {
                    mma_f16(d_cross, a_desc(1, ks), b_desc(0, ks), idesc, 1u);
                    mma_f16(d_cross, a_desc(0, ks), b_desc(1, ks), idesc, 1u);
                }
                tc_commit(smem_u32(&bar));
            }
            ok = mbar_wait(smem_u32(&bar), 1u, abort_flag) && ok;
            tc_fence_after_sync();
        }
    }

    // ---- its sums, 32 columns of 32 rows to a warp, to the CTAs that add up those rows: rows of 512 bytes, float4 slots
    // XOR-swizzled, slice after slice ----
    // Between the CTAs they move at some 11 bytes per clock (64 KB in 3.8 us), so only what the output has is sent, the rows
    // there are, dealt out evenly, and tiles of 64 columns where the machine holds twice as many; a CTA's own rows stay.  A
    // thread drains a row, four pieces of 128 bytes go out in one instruction: the turn through the warp's 4 KB takes less than
    // 32 pieces of 16 bytes do (512 x 512 x 512 9.3 -> 8.8 us; alike where the tiles have 128 columns).  Read by the CTAs that
    // add them up they need a second cluster barrier: 10.1.
    const int rows_each = (valid + p.slices - 1) / p.slices;
    // Its part of the rows is added up by all threads, four columns to a thread; their bias is on its way meanwhile.
    const int quads   = p.bn >> 2, slot = threadIdx.x & (quads - 1);
    const int64_t col = col0 + slot * 4;
    float b4[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        b4[q] = p.bias && col + q < p.n ? p.bias[col + q] : 0.0f;
    cluster_wait();
    const int quarter = warp & 3, cg = warp >> 2, row = quarter * 32 + lane;
    if (quarter * 32 < valid && cg * 32 < p.bn) {
        uint32_t main[32], cross[32];
        __syncwarp();
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cg * 32), main);
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(128 + cg * 32), cross);
        tmem_ld_wait();
        const float weight = wide ? 1.0f : kHalfLoInv, rs = wide ? 1.0f : row_inv[row];
        uint8_t *stage     = smem + warp * 4096; // the planes have been read
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 c = wide ? make_float4(1.0f, 1.0f, 1.0f, 1.0f) : *reinterpret_cast<const float4 *>(col_inv + cg * 32 + 4 * j);
            auto value = [&](int u, float s) {
                const float v = __fadd_rn(__uint_as_float(main[4 * j + u]), __fmul_rn(__uint_as_float(cross[4 * j + u]), weight));
                return ksteps > 0 ? __fmul_rn(__fmul_rn(v, rs), s) : 0.0f;
            };
            *reinterpret_cast<float4 *>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_float4(value(0, c.x), value(1, c.y), value(2, c.z), value(3, c.w));
        }
        __syncwarp();
        const int j = lane & 7;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int l = i * 4 + (lane >> 3), r = quarter * 32 + l, to = r / rows_each, at = r - to * rows_each;
            const float4 v = *reinterpret_cast<const float4 *>(stage + l * 128 + ((j ^ (l & 7)) << 4));
            const uint32_t dst = (uint32_t)((rank * rows_each + at) * 512 + (((cg * 8 + j) ^ (at & 7)) << 4));
            if (r < valid && to == rank)
                *reinterpret_cast<float4 *>(smem + kGD_Sums + dst) = v;
            else if (r < valid)
                st_cluster_f4(mapa(smem_base + (uint32_t)kGD_Sums + dst, (uint32_t)to), v);
        }
    }
    tc_fence_before_sync();
    __syncwarp();
    cluster_sync(); // every slice's sums have arrived; nobody writes to this CTA any more
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 256);
    }
    if (!failed && !*abort_flag)
        for (int r = threadIdx.x / quads; r < rows_each; r += kGD_Threads / quads) {
            const int64_t row = row0 + rank * rows_each + r;
            if (rank * rows_each + r >= valid || col >= p.n)
                break;
            const uint8_t *at = smem + kGD_Sums + r * 512 + ((slot ^ (r & 7)) << 4);
            float4 v          = *reinterpret_cast<const float4 *>(at);
            for (int z = 1; z < p.slices; ++z) {
                const float4 q = *reinterpret_cast<const float4 *>(at + z * rows_each * 512);
                v = make_float4(__fadd_rn(v.x, q.x), __fadd_rn(v.y, q.y), __fadd_rn(v.z, q.z), __fadd_rn(v.w, q.w));
            }
            float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
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
    // every thread has waited by a clock of its own: one that gave up has kept the CTA from storing, whatever thread 0 saw
    if (threadIdx.x == 0 && !failed && (!ok || *abort_flag))
        atomicExch(p.flags + FLAG_TIMEOUT, 1u + (uint32_t)blockIdx.x);
}

// How many clusters of `size` CTAs run at the same time.
int direct_clusters(const DeviceState *st, int size) {
    static int known[16][4] = {}; // per device, by log2(size); under the entry points' lock
    int &count = known[st->device & 15][size == 8 ? 3 : size / 2];
    if (count == 0) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)size, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(st->sm_count / size * size)), cfg.blockDim = dim3(kGD_Threads);
        cfg.dynamicSmemBytes = kGD_Smem;
        cfg.attrs = attr, cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(gemm_direct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGD_Smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&count, gemm_direct_kernel, &cfg) != cudaSuccess || count < 1) {
            cudaGetLastError();
            count = -1; // not known: the other kernels
        }
    }
    return count;
}

// Slices of k, a power of two of at most 128 values each; 0: the product is not for this kernel.  It takes those whose slices
// run at once, all clusters of them; k of one slice is left to the kernels whose bytes ct_matmul_packed_rows has.
int direct_slices(const DeviceState *st, int64_t m, int64_t k, int64_t n, int *bn) {
    if (k <= 192 || k > 8 * kGD_K || m > (1 << 20) || n > (1 << 20))
        return 0;
    int slices = 2;
    while (slices * kGD_K < k)
        slices *= 2;
    const int64_t rows = (m + 127) / 128, most = direct_clusters(st, slices);
    *bn                = n <= 64 || rows * ((n + 63) / 64) <= most ? 64 : 128;
    return rows * ((n + 127) / 128) <= most ? slices : 0;
}

} // namespace

bool gemm_direct_applicable(const DeviceState *st, int64_t m, int64_t k, int64_t n) {
    int bn;
    return direct_slices(st, m, k, n, &bn) > 0;
}

ct_status gemm_direct(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k, int64_t n, int act, float *out) {
    auto aligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    DirectParams p{};
    p.a = a, p.b = b, p.bias = bias, p.out = out;
    p.m = m, p.n = n, p.k = k;
    p.slices  = direct_slices(st, m, k, n, &p.bn);
    p.kc      = (int)((k + p.slices - 1) / p.slices + 15) & ~15;
    p.tiles_m = (int)((m + 127) / 128);
    p.act     = act;
    p.vec_a = (k & 3) == 0 && aligned(a), p.vec_b = (n & 3) == 0 && aligned(b), p.vec_out = (n & 3) == 0 && aligned(out);
    p.flags = st->flags_dev;
    const unsigned grid = (unsigned)(p.tiles_m * ((n + p.bn - 1) / p.bn) * p.slices);
    ProfScope prof("gemm_tc");
    CT_CUDA(launch_dependent_cluster(gemm_direct_kernel, p.slices, dim3(grid), dim3(kGD_Threads), (size_t)kGD_Smem, stream(), p));
    CT_LAUNCH_CHECK("gemm_direct");
    return CT_OK;
}

} // namespace ct
