// CUDA-core contractions for the shapes and dtypes the tensor-core kernel does not take:
//  - matmul_generic: any dtype pair, float64 accumulation per output element, exactly the
//    reference loop (modules/tensor/operators.cpp:757-766); used for int64/bool operands and
//    for tiny problems.
//  - gemm_f32_skinny: float32 x float32 with n <= 32 output columns (the classifier layer of
//    an MLP): one warp per output row, float64 accumulation, with bias / relu / row-softmax /
//    argmax fused, so the logits never round-trip through HBM.
#include "common.cuh"
#include "fastmath.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace ct {
namespace {

__device__ __forceinline__ double ld_as_double(int dt, const void *p, int64_t i) {
    switch (dt) {
    case CT_F32:
        return (double)static_cast<const float *>(p)[i];
    case CT_I64:
        return (double)static_cast<const int64_t *>(p)[i];
    default:
        return static_cast<const uint8_t *>(p)[i] != 0 ? 1.0 : 0.0;
    }
}

__device__ __forceinline__ void st_from_double(int dt, void *p, int64_t i, double v) {
    switch (dt) {
    case CT_F32:
        static_cast<float *>(p)[i] = (float)v;
        break;
    case CT_I64:
        static_cast<int64_t *>(p)[i] = (int64_t)v;
        break;
    default:
        static_cast<uint8_t *>(p)[i] = v != 0.0 ? 1 : 0;
        break;
    }
}

// 16x16 outputs per block, operands staged through shared memory as float64.
__global__ void __launch_bounds__(256) matmul_generic_kernel(
    int adt, const void *a, int bdt, const void *b, int64_t m, int64_t k, int64_t n, int odt,
    void *out) {
    __shared__ double sa[16][17];
    __shared__ double sb[16][17];
    int tx      = threadIdx.x & 15;
    int ty      = threadIdx.x >> 4;
    int64_t row = (int64_t)blockIdx.y * 16 + ty;
    int64_t col = (int64_t)blockIdx.x * 16 + tx;
    double acc  = 0.0;
    for (int64_t k0 = 0; k0 < k; k0 += 16) {
        int64_t ka = k0 + tx, kb = k0 + ty;
        sa[ty][tx] = (row < m && ka < k) ? ld_as_double(adt, a, row * k + ka) : 0.0;
        sb[ty][tx] = (kb < k && col < n) ? ld_as_double(bdt, b, kb * n + col) : 0.0;
        __syncthreads();
        int lim = (int)((k - k0) < 16 ? (k - k0) : 16);
        for (int kk = 0; kk < lim; ++kk)
            acc += sa[ty][kk] * sb[kk][tx]; // k ascending, like the reference
        __syncthreads();
    }
    if (row < m && col < n)
        st_from_double(odt, out, row * n + col, acc);
}

// One warp per output row; lanes split k.  N_MAX bounds the register accumulators.
template <int N_MAX>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(
    const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
    int64_t m, int64_t k, int n, int act, float *__restrict__ out, int64_t *__restrict__ argmax) {
    int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= m)
        return;
    int lane        = threadIdx.x & 31;
    const float *xr = x + row * k;
    double acc[N_MAX];
#pragma unroll
    for (int j = 0; j < N_MAX; ++j)
        acc[j] = 0.0;
    for (int64_t kk = lane; kk < k; kk += 32) {
        double xv       = (double)xr[kk];
        const float *wr = w + kk * n;
#pragma unroll
        for (int j = 0; j < N_MAX; ++j)
            if (j < n)
                acc[j] = __fma_rn(xv, (double)__ldg(wr + j), acc[j]); // float32 x float32 is exact in float64: same bits as mul, add
    }
#pragma unroll
    for (int j = 0; j < N_MAX; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    // Every lane now holds all n sums; lane j finishes column j.
    float logit = 0.0f;
#pragma unroll
    for (int j = 0; j < N_MAX; ++j) {
        if (j == lane && j < n) {
            double v = acc[j];
            if (bias)
                v += (double)bias[j]; // the bias is the last term of the float64 sum
            logit = (float)v;
        }
    }
    bool live = lane < n;
    if (act == CT_ACT_RELU) {
        logit = __fmul_rn(logit, logit > 0.0f ? 1.0f : 0.0f);
    }
    if (act != CT_ACT_SOFTMAX) {
        if (live)
            out[row * n + lane] = logit;
        return;
    }
    // Row softmax and argmax across the first n lanes, with the reference's scan semantics:
    // element 0 seeds, a later element wins only on strict '>'.
    float best   = __shfl_sync(0xffffffffu, logit, 0);
    int best_idx = 0;
    for (int j = 1; j < n; ++j) {
        float v = __shfl_sync(0xffffffffu, logit, j);
        if (v > best) {
            best     = v;
            best_idx = j;
        }
    }
    float e  = live ? exp_f32(__fsub_rn(logit, best)) : 0.0f;
    double s = 0.0;
    for (int j = 0; j < n; ++j)
        s += (double)__shfl_sync(0xffffffffu, e, j);
    float d = (float)s;
    if (live)
        out[row * n + lane] = __fdiv_rn(e, d);
    if (argmax && lane == 0)
        argmax[row] = best_idx;
}

// Lane j < n holds the rounded logit of column j of one row: activation, and for softmax the
// row softmax / argmax with the reference's scan semantics (element 0 seeds, a later element
// wins only on strict '>').  Called by a whole warp.
__device__ __forceinline__ void skinny_finish_logit(
    float logit, int64_t row, int n, int act, int lane, float *__restrict__ out,
    int64_t *__restrict__ argmax) {
    bool live = lane < n;
    if (act == CT_ACT_RELU)
        logit = __fmul_rn(logit, logit > 0.0f ? 1.0f : 0.0f);
    if (act != CT_ACT_SOFTMAX) {
        if (live)
            out[row * n + lane] = logit;
        return;
    }
    float best   = __shfl_sync(0xffffffffu, logit, 0);
    int best_idx = 0;
    for (int j = 1; j < n; ++j) {
        float v = __shfl_sync(0xffffffffu, logit, j);
        if (v > best) {
            best     = v;
            best_idx = j;
        }
    }
    float e  = live ? exp_f32(__fsub_rn(logit, best)) : 0.0f;
    double s = 0.0;
    for (int j = 0; j < n; ++j)
        s += (double)__shfl_sync(0xffffffffu, e, j);
    float d = (float)s;
    if (live)
        out[row * n + lane] = __fdiv_rn(e, d);
    if (argmax && lane == 0)
        argmax[row] = best_idx;
}

// Finishes one output row held as per-lane partial sums: butterfly reduction, then bias,
// activation, and (for softmax) the row softmax / argmax across the first n lanes.
template <int N_MAX>
__device__ __forceinline__ void skinny_finish_row(
    double (&acc)[N_MAX], const float *__restrict__ bias, int64_t row, int n, int act, int lane,
    float *__restrict__ out, int64_t *__restrict__ argmax) {
#pragma unroll
    for (int j = 0; j < N_MAX; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    float logit = 0.0f;
#pragma unroll
    for (int j = 0; j < N_MAX; ++j) {
        if (j == lane && j < n) {
            double v = acc[j];
            if (bias)
                v += (double)bias[j]; // the bias is the last term of the float64 sum
            logit = (float)v;
        }
    }
    skinny_finish_logit(logit, row, n, act, lane, out, argmax);
}

// Same contraction with the whole weight matrix [k][n] staged once per block in shared memory
// (k*n*4 bytes <= 200 KB): the weight reads that made the kernel above latency-bound become
// shared-memory reads, the activations stream in with 128-bit loads, and a persistent grid
// of 2 blocks per SM walks the rows.
template <int N_MAX>
__global__ void __launch_bounds__(256) gemm_skinny_smem_kernel(
    const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
    int64_t m, int64_t k, int n, int act, float *__restrict__ out, int64_t *__restrict__ argmax) {
    extern __shared__ __align__(16) double w_s[];
    // staged transposed [n][k] and already widened to float64: the float32 -> float64
    // conversions run on the slow special-function pipe, so they are paid once per weight
    // and block here instead of once per multiply-add
    const int total = (int)(k * n); // <= 25600 by the dispatch condition
    for (int base = threadIdx.x; base < total; base += 256 * 8) {
        float tmp[8]; // eight independent loads in flight per thread, then the scattered stores
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int i  = base + u * 256;
            tmp[u] = i < total ? __ldg(w + i) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int i = base + u * 256;
            if (i < total) {
                int kk = i / n, j = i - kk * n;
                w_s[(int64_t)j * k + kk] = (double)tmp[u];
            }
        }
    }
    __syncthreads();
    const int lane     = threadIdx.x & 31;
    const int64_t warp = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int64_t step = (int64_t)gridDim.x * 8;
    const bool vec     = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    for (int64_t row = warp; row < m; row += step) {
        const float *xr = x + row * k;
        double acc[N_MAX];
#pragma unroll
        for (int j = 0; j < N_MAX; ++j)
            acc[j] = 0.0;
        if (vec) {
            // eight 128-bit loads in flight per lane before any arithmetic: with few resident warps
            // the row would otherwise be one load-latency per 128 values of k
            constexpr int kChunk = 8;
            for (int64_t kk0 = (int64_t)lane * 4; kk0 < k; kk0 += 128 * kChunk) {
                float4 q[kChunk];
#pragma unroll
                for (int c = 0; c < kChunk; ++c) {
                    int64_t kk = kk0 + (int64_t)c * 128;
                    q[c]       = kk < k ? __ldcs(reinterpret_cast<const float4 *>(xr + kk)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int c = 0; c < kChunk; ++c) {
                    int64_t kk = kk0 + (int64_t)c * 128;
                    if (kk >= k)
                        break;
                    double x0 = (double)q[c].x, x1 = (double)q[c].y, x2 = (double)q[c].z, x3 = (double)q[c].w;
#pragma unroll
                    for (int j = 0; j < N_MAX; ++j)
                        if (j < n) {
                            const double2 *wp = reinterpret_cast<const double2 *>(w_s + (int64_t)j * k + kk);
                            double2 wa = wp[0], wb = wp[1];
                            acc[j] = __fma_rn(x0, wa.x, acc[j]);
                            acc[j] = __fma_rn(x1, wa.y, acc[j]);
                            acc[j] = __fma_rn(x2, wb.x, acc[j]);
                            acc[j] = __fma_rn(x3, wb.y, acc[j]);
                        }
                }
            }
        } else {
            for (int64_t kk = lane; kk < k; kk += 32) {
                double xd = (double)xr[kk];
#pragma unroll
                for (int j = 0; j < N_MAX; ++j)
                    if (j < n)
                        acc[j] = __fma_rn(xd, w_s[(int64_t)j * k + kk], acc[j]);
            }
        }
        skinny_finish_row<N_MAX>(acc, bias, row, n, act, lane, out, argmax);
    }
}

template <int N_MAX>
ct_status launch_skinny_smem(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k, int n,
    int act, float *out, int64_t *argmax) {
    size_t smem = (size_t)k * n * sizeof(double);
    if (smem > 48 * 1024)
        CT_CUDA(cudaFuncSetAttribute(
            gemm_skinny_smem_kernel<N_MAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    int64_t blocks = (m + 7) / 8;
    int64_t cap    = (int64_t)st->sm_count * (smem > 100 * 1024 ? 1 : 2);
    if (blocks > cap)
        blocks = cap;
    gemm_skinny_smem_kernel<N_MAX><<<(unsigned)blocks, 256, smem, stream()>>>(a, b, bias, m, k, n, act, out, argmax);
    CT_LAUNCH_CHECK("gemm_skinny_smem");
    return CT_OK;
}

// Few output columns (n <= 16), many rows: the classifier layer and its forward pass in training.  Lanes own
// values of k, registers own rows: a warp walks k in steps of 32 with R rows at a time, so the activations
// are read from global memory as they lie (128 contiguous bytes per row and step, any alignment, no staging),
// and a lane's weights - n doubles, read from shared memory where the whole matrix sits widened for the life
// of the block - feed R float64 FMAs each.  What bounds it: per step a warp takes 2 n shared-memory cycles and
// n R / 2 cycles of the SM's float64 pipe, so R = 8 leaves the pipe (and the read of x) as the bound; with rows
// on lanes and a broadcast weight per FMA, as before, shared memory took four times what the pipe did.
// 60000 x 785 x 10: 139 -> 74 us (the pipe alone 33, the read of x 29); the rest is issue, nearly two other instructions
// per FMA, of them the conversions to float64 at 16 per clock and SM.  (From eight columns on many rows take gemm_tall_kernel.)
// From eight columns on the weights come in whole lines, the first of them before the activations: 1024 x 10 at 4000 rows 13.6 -> 12.2 us,
// 1600 x 14 at 20000 84.9 -> 80.5; below, a thread takes rows of them, 200 x 5 at 20000 rows 11.2 us in whole lines and 10.6 so.
//
// The float64 sums of the lanes are added by exchanging rows first (each step halves the rows a lane keeps),
// then across what is left; every lane of a group of 32 / R then holds its row's n sums, adds the bias, rounds
// once and does the activation; softmax and argmax scan the columns in order like the reference.
constexpr int kFewWarps = 8;
constexpr int kFewRing  = 64; // activations in a lane's ring: 8 warps x 64 x 128 B = 64 KB an SM, 1 - R / 64 of it in flight
constexpr int kFewRingShort = 16; // where the weights leave room for no more

// Asynchronous 4-byte copies into a ring that only the copying lane reads: the depth of the prefetch is then in
// shared memory and in the hardware's group count, not in registers and their scoreboards - with register
// prefetch these kernels ran at one memory latency per step whatever its depth.  Zero where !ok.
__device__ __forceinline__ void copy_async_4(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_4(uint32_t dst, const float *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// Doubles between two k in shared memory: n rounded up to even, and an odd number of 16-byte units so that the
// 128-bit reads of consecutive lanes fall into distinct banks.
template <int NE> struct FewStride { static constexpr int value = (NE / 2) % 2 == 1 ? NE : NE + 2; };

template <int NE, int GROUP>
__device__ __forceinline__ void few_finish(
    const double (&sum)[NE], const float *__restrict__ bias, int64_t row, bool row_ok, int n, int act, int sub, float *__restrict__ out, int64_t *__restrict__ argmax) {
    float logit[NE];
#pragma unroll
    for (int j = 0; j < NE; ++j) {
        double v = sum[j];
        if (bias && j < n)
            v += (double)__ldg(bias + j); // the bias is the last term of the float64 sum
        logit[j] = (float)v;
        if (act == CT_ACT_RELU)
            logit[j] = __fmul_rn(logit[j], logit[j] > 0.0f ? 1.0f : 0.0f);
    }
    if (act == CT_ACT_SOFTMAX) {
        float best   = logit[0];
        int best_idx = 0;
#pragma unroll
        for (int j = 1; j < NE; ++j)
            if (j < n && logit[j] > best)
                best = logit[j], best_idx = j;
        if (argmax && sub == 0 && row_ok)
            argmax[row] = best_idx;
        // lane `sub` of the group has columns sub, sub + GROUP, ...: its exponentials, then everybody's in column order
        constexpr int OWN = (NE + GROUP - 1) / GROUP;
        float own[OWN];
#pragma unroll
        for (int u = 0; u < OWN; ++u) {
            float v = 0.0f;
#pragma unroll
            for (int q = 0; q < GROUP; ++q)
                if (u * GROUP + q < NE && q == sub)
                    v = logit[u * GROUP + q];
            own[u] = u * GROUP + sub < n ? exp_f32(__fsub_rn(v, best)) : 0.0f;
        }
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const float e = __shfl_sync(0xffffffffu, own[j / GROUP], j % GROUP, GROUP);
            if (j < n)
                s += (double)e;
        }
        const float d = (float)s;
#pragma unroll
        for (int u = 0; u < OWN; ++u)
            if (u * GROUP + sub < n && row_ok)
                out[row * n + u * GROUP + sub] = __fdiv_rn(own[u], d);
        return;
    }
#pragma unroll
    for (int j = 0; j < NE; ++j)
        if (j < n && j % GROUP == sub && row_ok)
            out[row * n + j] = logit[j];
}

// acc[r][j] of all lanes -> sum[j] of row `lane / (32 / R)` in every lane.
template <int R, int NE>
__device__ __forceinline__ void few_reduce(double (&acc)[R][NE], int lane, double (&sum)[NE]) {
#pragma unroll
    for (int half = R / 2, o = 16; half >= 1; half /= 2, o /= 2) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int r = 0; r < half; ++r)
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                const double give = upper ? acc[r][j] : acc[r + half][j];
                const double keep = upper ? acc[r + half][j] : acc[r][j];
                acc[r][j]         = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
    }
#pragma unroll
    for (int j = 0; j < NE; ++j) {
#pragma unroll
        for (int o = 16 / R; o >= 1; o /= 2)
            acc[0][j] += __shfl_xor_sync(0xffffffffu, acc[0][j], o);
        sum[j] = acc[0][j];
    }
}

template <int NE, int R, int RING>
__global__ void __launch_bounds__(32 * kFewWarps, 1) gemm_few_columns_kernel(
    const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias, int64_t m, int k, int n,
    int act, float *__restrict__ out, int64_t *__restrict__ argmax) {
    constexpr int S = FewStride<NE>::value, D = RING / R; // steps in the ring
    constexpr bool kLines = NE >= 8; // weights staged by whole lines
    extern __shared__ __align__(16) double w_few[]; // [k rounded up to 32][S], then the warps' rings [D][R][32] floats
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int steps = (k + 31) >> 5;
    griddep_launch_dependents();
    griddep_wait(); // activations (and possibly weights) come from the previous kernel
    // the walk of a warp: tiles of R rows, 32 values of k a step; the fetch runs D - 1 steps ahead of it, across tiles
    const int64_t tiles = (m + R - 1) / R, first = (int64_t)blockIdx.x + (int64_t)warp * gridDim.x;
    const int64_t stride = (int64_t)gridDim.x * kFewWarps;
    float *ring = reinterpret_cast<float *>(w_few + (size_t)steps * 32 * S) + warp * RING * 32 + lane;
    const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring);
    int64_t f_tile = first;
    int f_step = 0, f_slot = 0;
    const float *f_src = x + first * R * k + lane; // this lane's element of the first row
    auto fetch = [&]() {
        if (f_tile < tiles) {
            const uint32_t dst = ring_a + (uint32_t)(f_slot * R) * 128u;
            const int kk       = f_step * 32 + lane;
            if (f_tile * R + R <= m && f_step * 32 + 32 <= k) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    copy_async_4(dst + (uint32_t)r * 128u, f_src + (int64_t)r * k);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool ok = kk < k && f_tile * R + r < m;
                    copy_async_4(dst + (uint32_t)r * 128u, ok ? f_src + (int64_t)r * k : x, ok);
                }
            }
            f_src += 32;
            if (++f_step == steps) {
                f_step = 0, f_tile += stride;
                f_src = x + f_tile * R * k + lane;
            }
        }
        copy_async_commit();
        f_slot = f_slot + 1 == D ? 0 : f_slot + 1;
    };
    // the weights, widened once per block
    const int elements = k * n, e_rows = (32 * kFewWarps) / n, e_cols = (32 * kFewWarps) % n;
    int e_row = (int)threadIdx.x / n, e_col = (int)threadIdx.x % n;
    constexpr int kBatch = 16;
    float e_v[kLines ? kBatch : 1];
    auto ask = [&](int e) {
#pragma unroll
        for (int u = 0; kLines && u < kBatch; ++u)
            e_v[u] = e + u * 32 * kFewWarps < elements ? __ldg(w + e + u * 32 * kFewWarps) : 0.0f;
    };
    ask((int)threadIdx.x);
#pragma unroll 1
    for (int d = 0; d < D - 1; ++d)
        fetch();
    if (kLines) { // whole lines of w, the first of them asked for before the activations
        for (int e = (int)threadIdx.x; e < elements;) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                if (e + u * 32 * kFewWarps < elements)
                    w_few[e_row * S + e_col] = (double)e_v[kLines ? u : 0];
                e_row += e_rows, e_col += e_cols;
                if (e_col >= n)
                    e_col -= n, ++e_row;
            }
            e += kBatch * 32 * kFewWarps;
            if (e < elements)
                ask(e);
        }
        if (n < NE)
            for (int kk = threadIdx.x; kk < k; kk += 32 * kFewWarps)
                for (int j = n; j < NE; ++j)
                    w_few[kk * S + j] = 0.0;
        for (int e = k * S + (int)threadIdx.x; e < steps * 32 * S; e += 32 * kFewWarps)
            w_few[e] = 0.0;
    } else { // a thread takes rows of w
#pragma unroll 4
        for (int kk = threadIdx.x; kk < steps * 32; kk += 32 * kFewWarps) {
            float v[NE];
#pragma unroll
            for (int j = 0; j < NE; ++j)
                v[j] = (kk < k && j < n) ? __ldg(w + (int64_t)kk * n + j) : 0.0f;
#pragma unroll
            for (int j = 0; j < NE; j += 2)
                *reinterpret_cast<double2 *>(w_few + kk * S + j) = make_double2((double)v[j], (double)v[j + 1]);
        }
    }
    __syncthreads();
    int slot = 0;
    for (int64_t t = first; t < tiles; t += stride) {
        const int64_t row0 = t * R;
        double acc[R][NE];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int j = 0; j < NE; ++j)
                acc[r][j] = 0.0;
#pragma unroll 1
        for (int step = 0; step < steps; ++step) {
            copy_async_wait<D - 2>();
            double xv[R];
#pragma unroll
            for (int r = 0; r < R; ++r)
                xv[r] = (double)ring[(slot * R + r) * 32];
            slot = slot + 1 == D ? 0 : slot + 1;
            const double2 *wp = reinterpret_cast<const double2 *>(w_few + (step * 32 + lane) * S);
#pragma unroll
            for (int j = 0; j < NE / 2; ++j) {
                const double2 wv = wp[j];
                // float32 x float32 is exact in float64, so the fused form rounds like mul, add
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[r][2 * j]     = __fma_rn(xv[r], wv.x, acc[r][2 * j]);
                    acc[r][2 * j + 1] = __fma_rn(xv[r], wv.y, acc[r][2 * j + 1]);
                }
            }
            fetch(); // into the slot before this one, whose values have been used
        }
        double sum[NE];
        few_reduce<R, NE>(acc, lane, sum);
        constexpr int group = 32 / R;
        const int64_t row   = row0 + lane / group;
        few_finish<NE, group>(sum, bias, row, row < m, n, act, lane % group, out, argmax);
    }
}

// Eight columns and more, weights that leave room for the ring: the first eight columns (all, above twelve) by the float64 MMA, 8 rows
// x 8 columns x 4 values of k to an instruction, the others by multiply-adds.  The MMA is exact products and rounded
// additions like those, at the full rate of the float64 pipe (65 of 64 nominal per clock and SM against 52 of multiply-adds with
// operands from all over the register file), takes one issue slot for eight, and its sums lie in two registers a
// lane, so sixteen warps fit an SM and hardly anything is left to add up across lanes.
//
// A warp walks tiles of 8 T rows, 32 values of k a step, fed by its ring like the kernel above.  Lane 4 r + q has row r and the
// values 8 q .. 8 q + 7 of a step (which four values of k meet in an MMA is free), two 16-byte reads; rows are 36 floats
// apart, so eight lanes' reads cover all banks.  The weights lie as the lanes read them, 16 bytes each.
//
// 60000 x 785 x 10: 74.4 -> 55.7 us, x 8 62.5 -> 45.9, x 16 121 -> 80; 8192 x 785 x 10 16.2 -> 12.2.  The float64 pipe takes 31 of the 55.7, the
// read of x 29.  Warps wait for that pipe first (2.7 of 9 stalled per issue), then for dependences; the reads of shared memory, half of
// them for the columns beside the first eight, and the 4-byte copies keep its pipe at 0.57.
constexpr int kTallWarps = 16, kTallRow = 36, kTallRing = 48; // floats of a ring row; rows in a warp's ring
template <int NE> struct TallCfg {
    static constexpr int kTiles = NE > 12 ? 2 : 1, kExtra = NE > 12 ? 0 : NE - 8;
    static constexpr int kUnits = kTiles * 128 + kExtra * 16; // of 16 bytes, 32 values of k
    static constexpr size_t smem(int64_t k) { return (size_t)((k + 31) / 32) * kUnits * 16 + (size_t)kTallWarps * kTallRing * kTallRow * 4; }
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

template <int NE, int T>
__global__ void __launch_bounds__(32 * kTallWarps, 1) gemm_tall_kernel(
    const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias, int64_t m, int k, int n,
    int act, float *__restrict__ out, int64_t *__restrict__ argmax) {
    using C = TallCfg<NE>;
    constexpr int R = 8 * T, D = kTallRing / R, NT = C::kTiles, NX = C::kExtra;
    constexpr int CH = T == 1 ? 2 : 1; // chains of sums per tile of the result
    constexpr bool kAhead = T == 1;     // few warps have tiles: a step's activations are read while the one before is multiplied
    extern __shared__ __align__(16) double2 w_tall[]; // [steps][units], then the warps' rings [D][R][kTallRow] floats
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int steps = (k + 31) >> 5;
    griddep_launch_dependents();
    griddep_wait(); // activations (and possibly weights) come from the previous kernel
    const int64_t tiles = (m + R - 1) / R, first = (int64_t)blockIdx.x + (int64_t)warp * gridDim.x;
    const int64_t stride = (int64_t)gridDim.x * kTallWarps;
    float *ring = reinterpret_cast<float *>(w_tall + (size_t)steps * C::kUnits) + warp * kTallRing * kTallRow;
    const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring + lane);
    int64_t f_tile = first;
    int f_step = 0, f_slot = 0;
    bool f_whole = f_tile * R + R <= m;
    const float *f_src = x + first * R * k + lane; // this lane's element of the first row
    auto fetch = [&]() {
        if (f_tile < tiles) {
            const uint32_t dst = ring_a + (uint32_t)(f_slot * R * kTallRow) * 4u;
            const int kk       = f_step * 32 + lane;
            if (f_whole && f_step * 32 + 32 <= k) {
                const float *src = f_src;
#pragma unroll
                for (int r = 0; r < R; ++r, src += k)
                    copy_async_4(dst + (uint32_t)(r * kTallRow) * 4u, src);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool ok = kk < k && f_tile * R + r < m;
                    copy_async_4(dst + (uint32_t)(r * kTallRow) * 4u, ok ? f_src + (int64_t)r * k : x, ok);
                }
            }
            f_src += 32;
            if (++f_step == steps) {
                f_step = 0, f_tile += stride;
                f_whole = f_tile * R + R <= m;
                f_src   = x + f_tile * R * k + lane;
            }
        }
        copy_async_commit();
        f_slot = f_slot + 1 == D ? 0 : f_slot + 1;
    };
    // the weights, widened once per block and laid out by 16-byte units; the first of them are asked for before the activations
    constexpr int kBatch = 10;
    const int units = steps * C::kUnits;
    float v0[kBatch], v1[kBatch];
    auto weight = [&](int kk, int j) { return kk < k && j < n ? __ldg(w + (int64_t)kk * n + j) : 0.0f; };
    auto ask    = [&](int first_unit) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int at = first_unit + i * 32 * kTallWarps, block = at / C::kUnits, u = at - block * C::kUnits;
            if (at < units && u < NT * 128) { // [tile][pair of values of k][lane]
                const int kk = block * 32 + (u & 3) * 8 + ((u >> 5) & 3) * 2, j = (u >> 7) * 8 + ((u & 31) >> 2);
                v0[i] = weight(kk, j), v1[i] = weight(kk + 1, j);
            } else if (at < units) { // [value of k][pair of columns][q]
                const int e = u - NT * 128, pairs = NX / 2 > 0 ? NX / 2 : 1;
                const int kk = block * 32 + (e & 3) * 8 + (e >> 2) / pairs, j = 8 + (e >> 2) % pairs * 2;
                v0[i] = weight(kk, j), v1[i] = weight(kk, j + 1);
            }
        }
    };
    ask((int)threadIdx.x);
#pragma unroll 1
    for (int d = 0; d < D - 1; ++d)
        fetch();
    for (int at = (int)threadIdx.x; at < units;) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
            if (at + i * 32 * kTallWarps < units)
                w_tall[at + i * 32 * kTallWarps] = make_double2((double)v0[i], (double)v1[i]);
        at += kBatch * 32 * kTallWarps;
        if (at < units)
            ask(at);
    }
    __syncthreads();
    const float *mine = ring + (lane >> 2) * kTallRow + (lane & 3) * 8;
    int slot = 0;
    float4 xf[T][2];
    auto read = [&](float4 (&to)[T][2]) {
#pragma unroll
        for (int a = 0; a < T; ++a)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                to[a][h] = *reinterpret_cast<const float4 *>(mine + (slot * R + a * 8) * kTallRow + h * 4);
        slot = slot + 1 == D ? 0 : slot + 1;
    };
    if (kAhead) {
        copy_async_wait<D - 2>();
        __syncwarp();
        read(xf);
    }
    for (int64_t t = first; t < tiles; t += stride) {
        double acc[T][NT][CH][2], extra[T][CH][NX > 0 ? NX : 1];
#pragma unroll
        for (int a = 0; a < T; ++a) {
#pragma unroll
            for (int b = 0; b < NT * CH; ++b)
                acc[a][b / CH][b % CH][0] = acc[a][b / CH][b % CH][1] = 0.0;
#pragma unroll
            for (int j = 0; j < NX * CH; ++j)
                extra[a][NX > 0 ? j / NX : 0][NX > 0 ? j % NX : 0] = 0.0;
        }
        const double2 *wp = w_tall;
#pragma unroll 1
        for (int step = 0; step < steps; ++step, wp += C::kUnits) {
            // every lane's copies are there, and every lane has read the slot that is fetched next
            copy_async_wait<kAhead ? D - 3 : D - 2>();
            __syncwarp();
            float4 next[T][2];
            if (kAhead)
                read(next);
            else
                fetch(), read(xf);
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                double2 wv[NT];
#pragma unroll
                for (int b = 0; b < NT; ++b)
                    wv[b] = wp[(b * 4 + p) * 32 + lane];
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    double2 we[NX / 2 > 0 ? NX / 2 : 1];
#pragma unroll
                    for (int j = 0; j < NX / 2; ++j)
                        we[j] = wp[NT * 128 + ((2 * p + o) * (NX / 2) + j) * 4 + (lane & 3)];
#pragma unroll
                    for (int a = 0; a < T; ++a) {
                        const float4 q  = xf[a][p >> 1];
                        const double xv = (double)((p & 1) ? (o ? q.w : q.z) : (o ? q.y : q.x));
#pragma unroll
                        for (int b = 0; b < NT; ++b)
                            mma_f64(acc[a][b][o % CH], xv, o ? wv[b].y : wv[b].x);
                        // float32 x float32 is exact in float64, so the fused form rounds like mul, add
#pragma unroll
                        for (int j = 0; j < NX / 2; ++j) {
                            extra[a][o % CH][2 * j]     = __fma_rn(xv, we[j].x, extra[a][o % CH][2 * j]);
                            extra[a][o % CH][2 * j + 1] = __fma_rn(xv, we[j].y, extra[a][o % CH][2 * j + 1]);
                        }
                    }
                }
            }
            if (kAhead) {
                fetch();
#pragma unroll
                for (int h = 0; h < 2 * T; ++h)
                    xf[h / 2][h % 2] = next[h / 2][h % 2];
            }
        }
        // a lane has two columns of each tile: all of its row's sums to each of the row's four lanes
#pragma unroll
        for (int a = 0; a < T; ++a) {
            double sum[NE];
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                if (j < NT * 8) {
                    double c = acc[a][j / 8][0][j % 2];
                    if (CH == 2)
                        c += acc[a][j / 8][CH - 1][j % 2];
                    sum[j] = __shfl_sync(0xffffffffu, c, (lane & 28) | (j % 8) / 2);
                } else {
                    double c = extra[a][0][NX > 0 ? (j - 8) % NX : 0];
                    if (CH == 2)
                        c += extra[a][CH - 1][NX > 0 ? (j - 8) % NX : 0];
                    c += __shfl_xor_sync(0xffffffffu, c, 1);
                    sum[j] = c + __shfl_xor_sync(0xffffffffu, c, 2);
                }
            }
            const int64_t row = t * R + a * 8 + (lane >> 2);
            few_finish<NE, 4>(sum, bias, row, row < m, n, act, lane & 3, out, argmax);
        }
    }
}

// Few rows (a small request), or a weight matrix too long for shared memory: a block takes R rows, its eight
// warps an eighth of k each, weights straight from L2; the warps' sums meet in shared memory in warp order.
template <int NE, int R>
__global__ void __launch_bounds__(32 * kFewWarps) gemm_few_rows_kernel(
    const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias, int64_t m, int64_t k, int n,
    int act, float *__restrict__ out, int64_t *__restrict__ argmax) {
    __shared__ double part[kFewWarps][R][NE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    griddep_launch_dependents();
    griddep_wait();
    const int64_t row0 = (int64_t)blockIdx.x * R;
    const int rows     = m - row0 < R ? (int)(m - row0) : R;
    double acc[R][NE];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < NE; ++j)
            acc[r][j] = 0.0;
#pragma unroll 4
    for (int64_t kk = warp * 32 + lane; kk < k; kk += 32 * kFewWarps) {
        float q[R], wv[NE];
#pragma unroll
        for (int r = 0; r < R; ++r)
            q[r] = r < rows ? x[(row0 + r) * k + kk] : 0.0f;
#pragma unroll
        for (int j = 0; j < NE; ++j)
            wv[j] = j < n ? __ldg(w + kk * n + j) : 0.0f;
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const double wd = (double)wv[j];
#pragma unroll
            for (int r = 0; r < R; ++r)
                acc[r][j] = __fma_rn((double)q[r], wd, acc[r][j]);
        }
    }
    double sum[NE];
    few_reduce<R, NE>(acc, lane, sum);
    constexpr int group = 32 / R;
    if (lane % group == 0)
#pragma unroll
        for (int j = 0; j < NE; ++j)
            part[warp][lane / group][j] = sum[j];
    __syncthreads();
    if (warp == 0) {
        const int r = lane / group;
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            double v = part[0][r][j];
#pragma unroll
            for (int u = 1; u < kFewWarps; ++u)
                v += part[u][r][j];
            sum[j] = v;
        }
        few_finish<NE, group>(sum, bias, row0 + r, row0 + r < m, n, act, lane % group, out, argmax);
    }
}

// Blocks of gemm_few_rows_kernel that fit the machine at once.
template <int NE, int R> int few_rows_per_wave(const DeviceState *st) {
    static std::atomic<int> per_sm{0};
    int fit = per_sm.load(std::memory_order_relaxed);
    if (fit == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, gemm_few_rows_kernel<NE, R>, 32 * kFewWarps, 0) != cudaSuccess || fit < 1)
            fit = 1;
        per_sm.store(fit, std::memory_order_relaxed);
    }
    return fit * st->sm_count;
}

template <int NE>
ct_status launch_few(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k, int n, int act, float *out,
    int64_t *argmax) {
    constexpr size_t kMost = 220 * 1024;
    const size_t weights   = (size_t)((k + 31) / 32 * 32) * FewStride<NE>::value * sizeof(double);
    const bool longer      = weights + kFewWarps * kFewRing * 128 > kMost;
    const size_t smem      = weights + kFewWarps * (longer ? kFewRingShort : kFewRing) * 128;
    // What the two kernels take, in us.  Blocks of four (two) rows: a wave of them costs the same whatever k is beyond
    // 800, and there are few to a wave (one to an SM at ten columns).  Resident weights: staging them, then a cost
    // per activation and FMA.  Measured / by these (k x n at m): blocks 785 x 10 7.0 / 7.0 at 512 and 11.4 / 12.5 at 640,
    // 785 x 16 9.9 / 11.0 and 17.6 / 20.6, 300 x 10 6.3 / 6.7 at 640, 785 x 5 8.9 / 8.8 at 2047; resident 785 x 10
    // 9.3 / 9.7 at 640 and 11.2 / 13.2 at 4096, 785 x 16 13.7 / 13.2 at 640, 1500 x 10 14.6 / 15.2, 785 x 5 7.1 / 8.4 at 2047.
    const int64_t blocks = m <= 2 * st->sm_count ? (m + 1) / 2 : (m + 3) / 4;
    const int wave       = m <= 2 * st->sm_count ? few_rows_per_wave<NE, 2>(st) : few_rows_per_wave<NE, 4>(st);
    const double by_rows = 1.5 + (double)((blocks + wave - 1) / wave) * ((NE > 12 ? 2.0 : 0.8) + 6e-4 * NE * (double)std::min<int64_t>(k, 800));
    const double resident = 3.5 + 7e-4 * NE * (double)k + (double)m * (double)k * (6e-7 + 7e-8 * NE);
    if constexpr (NE >= 8) {
        // From where the kernel below walks a second time (32 rows to an SM; from half of that where no column is left to the
        // multiply-adds).  785 x 8 / 10 / 12 / 16 in us, there and here: 7.4 / 7.7 / 8.9 / 10.3 and 8.0 / 9.3 / 10.0 / 11.1 at 2000 rows, 8.9 / 9.5 /
        // 11.0 / 13.1 and 8.0 / 9.4 / 10.4 / 11.0 at 3000, 13.6 / 14.4 / 16.7 / 19.6 and 9.4 / 12.0 / 13.6 / 13.6 at 6000; 1024 x 10 at 4096
        // 11.4 and 12.2.
        const bool many = m > 32 * (int64_t)st->sm_count || (TallCfg<NE>::kExtra == 0 && m > 16 * (int64_t)st->sm_count);
        // sixteen rows to a warp where tiles of eight would be walked twice: 785 x 10 19.0 and 18.8 at 16000 rows, 26.3 and 24.2 at
        // 20000; 785 x 8 13.3 and 14.1, 19.5 and 16.7
        const bool deep = m > (int64_t)st->sm_count * kTallWarps * 8;
        // Rows that are no whole lines share a line between two steps, which has to stay in L1 meanwhile: 196 KB of shared memory leave that 60 KB,
        // more leave 28.  There the kernel is ahead for one pass only: 1400 x 8 30.4 us and above 41.9 at 16000 rows, 82.3 and 72.4 at
        // 40000 (1200 x 8, with 60 KB, 53.4 and 64.5), 1200 x 10 30.0 and 39.9, 80.7 and 72.0; whole lines, 1600 x 8, 39.1 and 50.3 at 20000.
        // Beyond twelve columns it is ahead all the same (785 x 16 64.2 and 80.8 at 40000 rows).
        const bool cached = NE > 12 || TallCfg<NE>::smem(k) <= 195 * 1024 || k % 32 == 0;
        if (many && TallCfg<NE>::smem(k) <= kMost && (cached || !deep) && resident < by_rows) {
            static bool tall_attr_set_dev[16] = {};
            if (!tall_attr_set_dev[st->device & 15]) {
                CT_CUDA(cudaFuncSetAttribute(gemm_tall_kernel<NE, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
                CT_CUDA(cudaFuncSetAttribute(gemm_tall_kernel<NE, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
                tall_attr_set_dev[st->device & 15] = true;
            }
            const int64_t tiles = deep ? (m + 15) / 16 : (m + 7) / 8;
            const unsigned grid = (unsigned)(tiles < st->sm_count ? tiles : st->sm_count);
            CT_CUDA(launch_dependent(deep ? gemm_tall_kernel<NE, 2> : gemm_tall_kernel<NE, 1>, dim3(grid), dim3(32 * kTallWarps), TallCfg<NE>::smem(k), stream(),
                a, b, bias, m, (int)k, n, act, out, argmax));
            CT_LAUNCH_CHECK("gemm_tall");
            return CT_OK;
        }
    }
    if (smem <= kMost && resident < by_rows) {
        // eight rows per warp where there are rows enough for two such tiles each and the sums stay in registers
        const bool deep = NE <= 12 && !longer && m >= (int64_t)st->sm_count * kFewWarps * 8 * 2;
        constexpr int kDeep     = NE <= 12 ? 8 : 4;
        static bool attr_set_dev[16] = {};
        if (!attr_set_dev[st->device & 15]) {
            CT_CUDA(cudaFuncSetAttribute(gemm_few_columns_kernel<NE, kDeep, kFewRing>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
            CT_CUDA(cudaFuncSetAttribute(gemm_few_columns_kernel<NE, 4, kFewRing>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
            CT_CUDA(cudaFuncSetAttribute(gemm_few_columns_kernel<NE, 4, kFewRingShort>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
            attr_set_dev[st->device & 15] = true;
        }
        const int rows      = deep ? kDeep : 4;
        const int64_t tiles = (m + rows - 1) / rows;
        const unsigned grid = (unsigned)(tiles < st->sm_count ? tiles : st->sm_count);
        auto kernel         = longer ? gemm_few_columns_kernel<NE, 4, kFewRingShort>
                                     : (deep ? gemm_few_columns_kernel<NE, kDeep, kFewRing> : gemm_few_columns_kernel<NE, 4, kFewRing>);
        // One block comes to an SM.  Where two would fit, they crowd on the SMs that are free first, and shared memory is set aside for both, so that L1,
        // which has to keep the lines that two steps share, gets the little that is left: 785 x 3 at 60000 rows 62 us, so 50, and an update
        // with such a product 170 and 112.
        const size_t alone = std::max<size_t>(smem, smem > 80 * 1024 ? 115 * 1024 : 0);
        CT_CUDA(launch_dependent(kernel, dim3(grid), dim3(32 * kFewWarps), alone, stream(), a, b, bias, m, (int)k, n, act, out, argmax));
        CT_LAUNCH_CHECK("gemm_few_columns");
        return CT_OK;
    }
    // weights that fit shared memory only without padding and ring: 1500 x 16 121 against 153 us at 8192 rows, 751 against
    // 1255 at 60000, 76 both ways at 4096; up to eight columns the blocks of rows are faster (3000 x 8: 189 against 228)
    if (smem > kMost && NE > 8 && m >= 4096 && (size_t)k * n * sizeof(double) <= 200 * 1024)
        return launch_skinny_smem<16>(st, a, b, bias, m, k, n, act, out, argmax);
    if (m <= 2 * st->sm_count)
        CT_CUDA(launch_dependent(gemm_few_rows_kernel<NE, 2>, dim3((unsigned)blocks), dim3(32 * kFewWarps), 0, stream(), a, b, bias, m, k, n,
                                 act, out, argmax));
    else
        CT_CUDA(launch_dependent(gemm_few_rows_kernel<NE, 4>, dim3((unsigned)blocks), dim3(32 * kFewWarps), 0, stream(), a, b, bias, m, k, n,
                                 act, out, argmax));
    CT_LAUNCH_CHECK("gemm_few_rows");
    return CT_OK;
}

} // namespace

ct_status matmul_generic(
    int adt, const void *a, int bdt, const void *b, int64_t m, int64_t k, int64_t n, void *out) {
    if (m == 0 || n == 0)
        return CT_OK;
    int odt = ct_result_dtype(CT_ADD, (ct_dtype)adt, (ct_dtype)bdt);
    if ((m + 15) / 16 > 65535)
        return fail(CT_ERR_TOO_LARGE, "matmul: too many rows for the generic kernel");
    dim3 grid((unsigned)((n + 15) / 16), (unsigned)((m + 15) / 16));
    matmul_generic_kernel<<<grid, 256, 0, stream()>>>(adt, a, bdt, b, m, k, n, odt, out);
    CT_LAUNCH_CHECK("matmul_generic");
    return CT_OK;
}

// ---- transposed left operand, few output columns --------------------------------------------
//
// out[i][j] = sum_k a_km[k][i] * b[k][j], n <= 32: the gradient of a classifier,
// `transpose(X) @ (probs - y)` (test/run/nn/mnist.cml:39; k = samples, m = features, n = classes).
// Both operands are read in their own row-major order, X exactly once: a thread owns R output rows
// (columns of X, so a warp's loads are contiguous), the rows of b are widened to float64 in shared
// memory once per block and read as broadcasts, and every product is an exact float64 FMA as in
// the reference (operators.cpp:757-766).  The long dimension is cut into slices over the grid;
// the slices' float64 sums are added in slice order by gemm_tn_skinny_finish_kernel, so the result
// does not depend on scheduling.  Bound by the float64 pipe and the read of X, which are about
// equal at n = 10.
//
// R and the warps of a block are chosen so that the block's warps cover the output rows evenly: with blocks of
// 4 x 128 rows, 785 features made every other block a quarter full.  785 x 60000 x 10: 94 -> 90 us (eight columns and more have the
// kernel behind this one now).
constexpr int kTnMinThreads = 64, kTnMaxThreads = 160; // two blocks to an SM at 168 registers
constexpr int kTnChunk   = 32; // rows of b staged per step
constexpr int kTnGroup   = 2;  // k steps fetched together
constexpr int kTnGroups  = 6;  // groups in a warp's ring, all but one in flight

__device__ __forceinline__ void tn_block_barrier() {
    // a named barrier counts arriving threads, wherever in the code they arrive from: the warps of a
    // block run differently specialised copies of the loop below
    asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x) : "memory");
}

template <int NMAX, int R>
__global__ void __launch_bounds__(kTnMaxThreads, 2) gemm_tn_skinny_kernel(
    const float *__restrict__ a_km, const float *__restrict__ b, int64_t m, int64_t k, int n, int64_t k_per_slice,
    double *__restrict__ partial) {
    griddep_wait();
    griddep_launch_dependents();
    constexpr int G  = kTnGroup;
    constexpr int BL = (kTnChunk * NMAX + kTnMinThreads - 1) / kTnMinThreads; // staged b values per thread
    __shared__ __align__(16) double bs[2][kTnChunk][NMAX];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int threads      = (int)blockDim.x;
    const int64_t warp_row = ((int64_t)blockIdx.x * (threads / 32) + warp) * (32 * R);
    const int64_t row0     = warp_row + lane;
    const int64_t k0   = (int64_t)blockIdx.y * k_per_slice;
    const int64_t k1   = k0 + k_per_slice < k ? k0 + k_per_slice : k;

    float bnext[BL];
    auto fetch_b = [&](int64_t kc) {
#pragma unroll
        for (int u = 0; u < BL; ++u) {
            const int idx = threadIdx.x + u * threads;
            if (u * threads >= kTnChunk * NMAX)
                break;
            const int kk = idx / NMAX, j = idx - kk * NMAX;
            bnext[u] = (idx < kTnChunk * NMAX && kc + kk < k1 && j < n) ? __ldg(b + (kc + kk) * n + j) : 0.0f;
        }
    };
    auto store_b = [&](int buf) {
#pragma unroll
        for (int u = 0; u < BL; ++u) {
            const int idx = threadIdx.x + u * threads;
            if (u * threads >= kTnChunk * NMAX)
                break;
            if (idx < kTnChunk * NMAX)
                (&bs[buf][0][0])[idx] = (double)bnext[u];
        }
    };

    double acc[R][NMAX];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < NMAX; ++j)
            acc[r][j] = 0.0;
    // the operand arrives G k steps at a time in a ring of its own for each lane
    __shared__ float ring_s[kTnMaxThreads / 32][kTnGroups][G][R][32];
    float(*ring)[G][R][32] = ring_s[warp];
    const float *pa        = a_km + k0 * m + row0; // row `next` of the operand, this lane's first column
    int64_t next           = k0;
    int put = 0, get = 0;
    const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(&ring[0][0][0][lane]);
    const bool full       = warp_row + 32 * R <= m;
    auto fetch_a = [&]() {
        const uint32_t dst = ring_a + (uint32_t)put * (G * R * 128u);
        if (full && next + G <= k1) {
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const float *src = pa + u * m;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    copy_async_4(dst + (uint32_t)(u * R + r) * 128u, src + 32 * r);
            }
        } else {
#pragma unroll
            for (int u = 0; u < G; ++u)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool ok = next + u < k1 && row0 + 32 * r < m;
                    copy_async_4(dst + (uint32_t)(u * R + r) * 128u, ok ? pa + u * m + 32 * r : a_km, ok);
                }
        }
        copy_async_commit();
        pa += G * m;
        next += G;
        put = put + 1 == kTnGroups ? 0 : put + 1;
    };
    auto compute = [&](int buf, int g) {
        copy_async_wait<kTnGroups - 2>();
#pragma unroll
        for (int u = 0; u < G; ++u) {
            double av[R];
#pragma unroll
            for (int r = 0; r < R; ++r)
                av[r] = (double)ring[get][u][r][lane];
#pragma unroll
            for (int j = 0; j < NMAX; j += 2) {
                const double2 bj = *reinterpret_cast<const double2 *>(&bs[buf][g + u][j]);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[r][j]     = fma(av[r], bj.x, acc[r][j]);
                    acc[r][j + 1] = fma(av[r], bj.y, acc[r][j + 1]);
                }
            }
        }
        get = get + 1 == kTnGroups ? 0 : get + 1;
    };
    fetch_b(k0);
#pragma unroll 1
    for (int d = 0; d < kTnGroups - 1; ++d)
        fetch_a();
    store_b(0);
    tn_block_barrier();
    int buf = 0;
    for (int64_t kc = k0; kc < k1; kc += kTnChunk, buf ^= 1) {
        const bool more = kc + kTnChunk < k1;
        if (more)
            fetch_b(kc + kTnChunk);
#pragma unroll 1
        for (int g = 0; g < kTnChunk; g += G) {
            compute(buf, g);
            fetch_a(); // may already belong to the next chunk; zeros past the slice
        }
        if (more)
            store_b(buf ^ 1); // nobody reads that buffer any more: all warps passed the last barrier
        tn_block_barrier();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (row0 + 32 * r < m) {
            double *dst = partial + ((int64_t)blockIdx.y * m + row0 + 32 * r) * n;
#pragma unroll
            for (int j = 0; j < NMAX; ++j)
                if (j < n)
                    dst[j] = acc[r][j];
        }
    }
}

// Eight to sixteen columns: the first eight (all, above ten) by the float64 MMA, 8 rows of the result x 8 columns x 4 values of k
// to an instruction, as in gemm_tall_kernel, with the grid, slices and staging of b of the kernel above.  A ring holds four
// values of k at a time; lane 4 f + q has the q-th of them and the 4 R rows of the result from 4 R f on, which its 16-byte reads take
// in turn as row f of 4 R tiles, and one weight of b serves them all.
//
// At 785 x 60000 x 10 the float64 pipe takes 32 us, the read of X 29, the shared-memory pipe is at 0.57: they overlap as far as there are
// warps (what they wait for: dependences 1.9, the chunks' barrier 1.5, copies 1.1, the float64 pipe 1.1 per issue), so few rows to a warp are
// best: 88.4 us by multiply-adds, with R = 5 / 4 / 3 / 2 spills / 97 / 75.4 / 71.9; x 8 76.3 -> 59.7, x 16 145 -> 95; 300 x 5000 x 10
// 14.9 -> 11.6.
template <int NMAX, int R>
__global__ void __launch_bounds__(kTnMaxThreads, 3) gemm_tn_tall_kernel(
    const float *__restrict__ a_km, const float *__restrict__ b, int64_t m, int64_t k, int n, int64_t k_per_slice,
    double *__restrict__ partial) {
    griddep_wait();
    griddep_launch_dependents();
    constexpr int G = 4, GROUPS = 3, NT = NMAX > 10 ? 2 : 1, NX = NMAX == 10 ? 2 : 0;
    constexpr int NB = NT * 8 + NX;                       // columns of b staged
    constexpr int ROW = 32 * R + 4;                       // floats of a ring row
    constexpr int BL  = (kTnChunk * NB + kTnMinThreads - 1) / kTnMinThreads; // staged b values per thread
    __shared__ __align__(16) double bs[2][kTnChunk][NB];
    __shared__ __align__(16) float ring_s[kTnMaxThreads / 32][GROUPS][G][ROW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, threads = (int)blockDim.x;
    const int64_t warp_row = ((int64_t)blockIdx.x * (threads / 32) + warp) * (32 * R);
    const int64_t row0     = warp_row + lane;
    const int64_t k0       = (int64_t)blockIdx.y * k_per_slice;
    const int64_t k1       = k0 + k_per_slice < k ? k0 + k_per_slice : k;

    float bnext[BL];
    auto fetch_b = [&](int64_t kc) {
#pragma unroll
        for (int u = 0; u < BL; ++u) {
            const int idx = threadIdx.x + u * threads;
            if (u * threads >= kTnChunk * NB)
                break;
            const int kk = idx / NB, j = idx - kk * NB;
            bnext[u] = (idx < kTnChunk * NB && kc + kk < k1 && j < n) ? __ldg(b + (kc + kk) * n + j) : 0.0f;
        }
    };
    auto store_b = [&](int buf) {
#pragma unroll
        for (int u = 0; u < BL; ++u) {
            const int idx = threadIdx.x + u * threads;
            if (u * threads >= kTnChunk * NB)
                break;
            if (idx < kTnChunk * NB)
                (&bs[buf][0][0])[idx] = (double)bnext[u];
        }
    };

    double acc[4 * R][NT][2], extra[4 * R][NX > 0 ? NX : 1];
#pragma unroll
    for (int t = 0; t < 4 * R; ++t) {
#pragma unroll
        for (int u = 0; u < NT; ++u)
            acc[t][u][0] = acc[t][u][1] = 0.0;
#pragma unroll
        for (int j = 0; j < NX; ++j)
            extra[t][j] = 0.0;
    }
    float(*ring)[G][ROW] = ring_s[warp];
    const float *pa      = a_km + k0 * m + row0; // row `next` of the operand, this lane's first column
    int64_t next         = k0;
    int put = 0, get = 0;
    const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(&ring[0][0][lane]);
    const bool full       = warp_row + 32 * R <= m;
    auto fetch_a = [&]() {
        const uint32_t dst = ring_a + (uint32_t)put * (G * ROW * 4u);
        const bool whole   = full && next + G <= k1;
        const float *src   = pa;
#pragma unroll
        for (int u = 0; u < G; ++u, src += m)
            if (whole) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    copy_async_4(dst + (uint32_t)(u * ROW + 32 * r) * 4u, src + 32 * r);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool ok = next + u < k1 && row0 + 32 * r < m;
                    copy_async_4(dst + (uint32_t)(u * ROW + 32 * r) * 4u, ok ? src + 32 * r : a_km, ok);
                }
            }
        copy_async_commit();
        pa += G * m;
        next += G;
        put = put + 1 == GROUPS ? 0 : put + 1;
    };
    auto compute = [&](int buf, int g) {
        copy_async_wait<GROUPS - 2>();
        __syncwarp(); // every lane's copies are there, and every lane has read the group before
        double bv[NT];
#pragma unroll
        for (int u = 0; u < NT; ++u)
            bv[u] = bs[buf][g + (lane & 3)][u * 8 + (lane >> 2)];
        double2 be = make_double2(0.0, 0.0);
        if (NX > 0)
            be = *reinterpret_cast<const double2 *>(&bs[buf][g + (lane & 3)][NB - 2]);
        const float *mine = &ring[get][lane & 3][(lane >> 2) * (4 * R)];
#pragma unroll
        for (int h = 0; h < R; ++h) {
            const float4 q   = *reinterpret_cast<const float4 *>(mine + 4 * h);
            const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double av = (double)v[e];
#pragma unroll
                for (int u = 0; u < NT; ++u)
                    mma_f64(acc[4 * h + e][u], av, bv[u]);
                if (NX > 0) { // float32 x float32 is exact in float64
                    extra[4 * h + e][0]               = __fma_rn(av, be.x, extra[4 * h + e][0]);
                    extra[4 * h + e][NX > 0 ? NX - 1 : 0] = __fma_rn(av, be.y, extra[4 * h + e][NX > 0 ? NX - 1 : 0]);
                }
            }
        }
        get = get + 1 == GROUPS ? 0 : get + 1;
    };
    fetch_b(k0);
    const bool has_rows = warp_row < m; // a block's last warps may have none
#pragma unroll 1
    for (int d = 0; has_rows && d < GROUPS - 1; ++d)
        fetch_a();
    store_b(0);
    __syncthreads();
    int buf = 0;
    for (int64_t kc = k0; kc < k1; kc += kTnChunk, buf ^= 1) {
        const bool more = kc + kTnChunk < k1;
        if (more)
            fetch_b(kc + kTnChunk);
#pragma unroll 1
        for (int g = 0; has_rows && g < kTnChunk; g += G) {
            compute(buf, g);
            fetch_a(); // may already belong to the next chunk; zeros past the slice
        }
        if (more)
            store_b(buf ^ 1); // nobody reads that buffer any more: all warps passed the last barrier
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < 4 * R; ++t) {
        const int64_t row = warp_row + (lane >> 2) * (4 * R) + t;
        double *dst       = partial + ((int64_t)blockIdx.y * m + row) * n;
#pragma unroll
        for (int u = 0; u < NT; ++u)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int j = u * 8 + (lane & 3) * 2 + i;
                if (row < m && j < n)
                    dst[j] = acc[t][u][i];
            }
#pragma unroll
        for (int x = 0; x < NX; ++x) {
            double c = extra[t][x];
            c += __shfl_xor_sync(0xffffffffu, c, 1);
            c += __shfl_xor_sync(0xffffffffu, c, 2);
            if (row < m && (lane & 3) == x && NT * 8 + x < n)
                dst[NT * 8 + x] = c;
        }
    }
}

// One warp per output element: lane l adds the slices l, l + 32, ... in that order, then the lanes'
// sums are added in a fixed butterfly - the same order on every run.
__global__ void __launch_bounds__(256) gemm_tn_skinny_finish_kernel(
    const double *__restrict__ partial, int64_t mn, int slices, float *__restrict__ out) {
    griddep_wait();
    griddep_launch_dependents();
    const int lane  = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5;
    if (i >= mn)
        return;
    double sum = 0.0;
    for (int s = lane; s < slices; s += 32)
        sum += partial[(int64_t)s * mn + i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0)
        out[i] = (float)sum;
}

template <int NMAX, int R>
static ct_status launch_tn_skinny(
    DeviceState *st, const float *a_km, const float *b, int64_t m, int64_t k, int n, float *out) {
    constexpr bool kTall = NMAX >= 8 && NMAX <= 16;
    auto choose         = [] {
        if constexpr (kTall)
            return gemm_tn_tall_kernel<NMAX, R>;
        else
            return gemm_tn_skinny_kernel<NMAX, R>;
    };
    const auto kernel = choose();
    const int64_t warps   = (m + 32 * R - 1) / (32 * R);
    const int64_t mblocks = (warps + kTnMaxThreads / 32 - 1) / (kTnMaxThreads / 32);
    const int threads     = (int)std::max<int64_t>(kTnMinThreads, (warps + mblocks - 1) / mblocks * 32);
    // one wave of blocks; rounding the slice length up only takes blocks away
    static std::atomic<int> per_sm[kTnMaxThreads / 32 + 1];
    int fit = per_sm[threads / 32].load(std::memory_order_relaxed);
    if (fit == 0) {
        CT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, 0));
        fit = fit < 1 ? 1 : fit;
        per_sm[threads / 32].store(fit, std::memory_order_relaxed);
    }
    int64_t slices     = fit * (int64_t)st->sm_count / mblocks;
    // a warp takes about a fifth of a microsecond per k whatever the size, so a short k is cut down to single chunks
    const int64_t most = (k + kTnChunk - 1) / kTnChunk;
    if (slices > most)
        slices = most;
    if (slices < 1)
        slices = 1;
    if (slices > 65535)
        slices = 65535;
    int64_t k_per_slice = (k + slices - 1) / slices;
    k_per_slice         = (k_per_slice + kTnChunk - 1) / kTnChunk * kTnChunk;
    if (k_per_slice < kTnChunk)
        k_per_slice = kTnChunk;
    // Small blocks with a chunk or two each that nearly fill the machine leave the kernels before and behind them no registers to start with, and
    // more sums to add up than the chunk saved: one chunk more to each then (one product behind another, 100 x 33000 x 13 60 us, 1032
    // blocks in 1184 places, and 21, 256 x 17000 x 8 26.3 and 16.6, 192 x 45000 x 8 35 and 18; at 0.63 of the places 12.0 and 14.9 for 40 x 17000 x
    // 13; blocks of five warps lose, 600 x 12000 x 13 25.7 and 30.1).
    if (kTall && threads < kTnMaxThreads && k_per_slice <= 2 * kTnChunk && mblocks * ((k + k_per_slice - 1) / k_per_slice) * 5 > 4 * fit * (int64_t)st->sm_count)
        k_per_slice += kTnChunk;
    slices = k > 0 ? (k + k_per_slice - 1) / k_per_slice : 1;
    CT_TRY(ensure_ws(&st->splitk_ws, &st->splitk_ws_bytes, (size_t)slices * m * n * sizeof(double)));
    auto *partial = static_cast<double *>(st->splitk_ws);
    dim3 grid((unsigned)mblocks, (unsigned)slices);
    // Both start while their predecessor ends (9018 x 1088 x 10 62.5 -> 60.3 us with what precedes and follows it, 878 x 854 x 8
    // 23.8 -> 21.5), but for many small blocks with several chunks each: those crowd on the SMs that are free first (one update
    // of 96854 x 191 x 16 178, started on an idle machine 169; 33930 x 76 x 4 38 and 33).
    if (threads > kTnMinThreads || k_per_slice == kTnChunk)
        (void)launch_dependent(kernel, grid, dim3(threads), 0, stream(), a_km, b, m, k, n, k_per_slice, partial);
    else
        kernel<<<grid, threads, 0, stream()>>>(a_km, b, m, k, n, k_per_slice, partial);
    CT_LAUNCH_CHECK("gemm_tn_skinny");
    const int64_t mn = m * n;
    (void)launch_dependent(gemm_tn_skinny_finish_kernel, dim3((unsigned)((mn * 32 + 255) / 256)), dim3(256), 0, stream(), partial, mn, (int)slices, out);
    CT_LAUNCH_CHECK("gemm_tn_skinny_finish");
    return CT_OK;
}

ct_status gemm_f32_tn_skinny(
    DeviceState *st, const float *a_km, const float *b, int64_t m, int64_t k, int64_t n, float *out) {
    if (m == 0 || n == 0)
        return CT_OK;
    if (n > 32 || m > 0x7fffffffll * 64)
        return fail(CT_ERR_INVALID, "transposed skinny GEMM takes at most 32 output columns");
    ProfScope prof("gemm_skinny");
    // Rows per lane: up to four cost the reads of b in shared memory (2 n cycles per warp and k), more cost
    // float64 FMAs (R n / 2); take what covers the m / 32 row groups with the least of it.
    const int64_t groups = (m + 31) / 32;
    auto cost            = [&](int64_t r) { return (groups + r - 1) / r * (r > 4 ? r : 4); };
    const bool five      = cost(5) < cost(4);
#define CT_TN(NMAX)                                                                 \
    return five ? launch_tn_skinny<NMAX, 5>(st, a_km, b, m, k, (int)n, out) \
                : launch_tn_skinny<NMAX, 4>(st, a_km, b, m, k, (int)n, out)
    switch ((n + 1) / 2) {
    case 1: CT_TN(2);
    case 2: CT_TN(4);
    case 3: CT_TN(6);
    case 4: return launch_tn_skinny<8, 2>(st, a_km, b, m, k, (int)n, out);
    case 5: return launch_tn_skinny<10, 2>(st, a_km, b, m, k, (int)n, out);
    case 6: return launch_tn_skinny<12, 2>(st, a_km, b, m, k, (int)n, out);
    case 7: return launch_tn_skinny<14, 2>(st, a_km, b, m, k, (int)n, out);
    case 8: return launch_tn_skinny<16, 2>(st, a_km, b, m, k, (int)n, out);
    default: break;
    }
#undef CT_TN
    if (n <= 24)
        return launch_tn_skinny<24, 1>(st, a_km, b, m, k, (int)n, out);
    return launch_tn_skinny<32, 1>(st, a_km, b, m, k, (int)n, out);
}

ct_status gemm_f32_skinny(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k,
    int64_t n, int act, float *out, int64_t *argmax) {
    if (m == 0 || n == 0)
        return CT_OK;
    if (n > 32)
        return fail(CT_ERR_INVALID, "skinny GEMM takes at most 32 output columns");
    unsigned blocks = (unsigned)((m + 7) / 8);
    ProfScope prof("gemm_skinny");
    if (n <= 16 && m <= 0x7fffffffll && k <= 0x7fffffffll) {
        switch ((n + 1) / 2) {
        case 1: return launch_few<2>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 2: return launch_few<4>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 3: return launch_few<6>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 4: return launch_few<8>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 5: return launch_few<10>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 6: return launch_few<12>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        case 7: return launch_few<14>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        default: return launch_few<16>(st, a, b, bias, m, k, (int)n, act, out, argmax);
        }
    }
    if ((size_t)k * n * sizeof(double) <= 200 * 1024 && k > 0) {
        return launch_skinny_smem<32>(st, a, b, bias, m, k, (int)n, act, out, argmax);
    }
    gemm_skinny_kernel<32><<<blocks, 256, 0, stream()>>>(a, b, bias, m, k, (int)n, act, out, argmax);
    CT_LAUNCH_CHECK("gemm_skinny");
    return CT_OK;
}

} // namespace ct
