// Shared host/device plumbing of libcamel_tensor_b200.so: per-thread error text, the current
// device/stream, the launch counter, the device-side error words and cached workspaces.
#pragma once

#include "camel_tensor_b200.h"

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <utility>

namespace ct {

// Device-side error words, read back by the entry points that must report them.
//   words 0-1  data-dependent exceptions of one call: cleared by the entry point that checks them,
//              read back (with a synchronisation) before it returns.
//   word 2     sticky: written by a contraction kernel whose bounded wait ran out and by nothing
//              else; only ct_check() (or a *_host entry point that reports it) clears it.  While it
//              is set every later contraction kernel returns at once, so that a failed launch is
//              not followed by products of its undefined output; no entry point clears it on the
//              way in, and the failure is therefore still there when the host next looks.
enum FlagWord : int {
    FLAG_DIV_ZERO   = 0, // a divisor was 0 (reference: "Division by zero")
    FLAG_LOG_DOMAIN = 1, // an input of log was <= 0
    FLAG_TIMEOUT    = 2, // a bounded in-kernel wait ran out (value = 1 + the block that gave up)
    FLAG_EXCEPTION_READERS = 4, // CTAs of a product that have read the exceptions of its operands (half_split.cuh)
    FLAG_PANEL      = 5, // a panel product (gemm_panel.cu) left its operands to the kernels behind it
    FLAG_COUNT      = 8
};

struct HalfExceptions;
struct DeviceState {
    bool ready           = false;
    int device           = -1;
    int sm_count         = 0;
    uint32_t *flags_dev  = nullptr; // FLAG_COUNT words
    uint32_t *flags_host = nullptr; // pinned mirror
    struct HalfExceptions *exceptions_dev = nullptr; // of the operands of the product being prepared
    void *reduce_ws      = nullptr; // partials of the two-pass reductions
    size_t reduce_ws_bytes = 0;
    void *gemm_ws        = nullptr; // split operand planes of the tensor-core GEMM
    size_t gemm_ws_bytes = 0;
    void *splitk_ws      = nullptr; // partial outputs of the split-K GEMM
    size_t splitk_ws_bytes = 0;
    void *stage_ws[3]    = {nullptr, nullptr, nullptr}; // device staging of the *_host forms
    size_t stage_ws_bytes[3] = {0, 0, 0};
};

void set_error(const char *fmt, ...);
ct_status fail(ct_status code, const char *fmt, ...);
ct_status cuda_fail(cudaError_t e, const char *what);

// The reference's Taskflow scheduler calls operators from up to 32 threads at once
// (src/passes/sched/taskflow/taskflow.h:79-80).  An entry point may enqueue several kernels that
// share a cached workspace or the device error words; those sequences must not interleave on the
// stream, so every compute entry point holds this lock (recursive: entry points call each other)
// while it enqueues.  Device work itself stays asynchronous.
class OpLock {
  public:
    OpLock();
    ~OpLock();
    OpLock(const OpLock &)            = delete;
    OpLock &operator=(const OpLock &) = delete;
};

// Current device state (initialised on first use) and stream of the calling process.
ct_status current(DeviceState **out);
cudaStream_t stream();
void count_launch(unsigned n = 1);

// Grows a cached workspace (never shrinks); contents are undefined after the call.
ct_status ensure_ws(void **ptr, size_t *cap, size_t bytes);

// Clears the per-call error words (FLAG_DIV_ZERO, FLAG_LOG_DOMAIN) on the stream; the sticky
// FLAG_TIMEOUT word is left alone.
ct_status clear_data_flags(DeviceState *st);
// Synchronises the stream and copies the error words to st->flags_host.
ct_status fetch_flags(DeviceState *st);
// After fetch_flags: reports (and clears) a recorded kernel timeout; CT_OK if there is none.
ct_status report_timeout(DeviceState *st, const char *what);

#define CT_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t e__ = (call);                                                                  \
        if (e__ != cudaSuccess)                                                                    \
            return ::ct::cuda_fail(e__, #call);                                                    \
    } while (0)

#define CT_TRY(call)                                                                               \
    do {                                                                                           \
        ct_status s__ = (call);                                                                    \
        if (s__ != CT_OK)                                                                          \
            return s__;                                                                            \
    } while (0)

#define CT_LAUNCH_CHECK(name)                                                                      \
    do {                                                                                           \
        ::ct::count_launch();                                                                      \
        cudaError_t e__ = cudaGetLastError();                                                      \
        if (e__ != cudaSuccess)                                                                    \
            return ::ct::cuda_fail(e__, name);                                                     \
    } while (0)

// Programmatic dependent launch.  A chain of short kernels (the layers of an MLP: 8-40 us each)
// otherwise pays, at every boundary, the drain of one grid, the launch of the next and its set-up.
// A kernel launched with launch_dependent() may be scheduled while its predecessor in the stream
// is still running; it must execute griddep_wait() before it touches any global memory (the wait
// returns once the predecessor grid has completed and its writes are visible), so only its set-up
// (barrier initialisation, TMEM allocation, descriptor prefetch, index arithmetic) overlaps.  A
// kernel lets its successor start early with griddep_launch_dependents(); without that call the
// successor starts when the grid ends, as usual.  A kernel of a few microseconds calls it behind its own wait: before it,
// the successor of its successor would come up while its predecessor still runs, and take the slots that are free then instead
// of spreading over the SMs (a training step of 5493 x 279 x 16 47 us, and 39 so).  CAMEL_TENSOR_NO_PDL=1 turns the attribute off.
// While per-kernel event brackets are on (ct_profile_enable) kernels are launched the ordinary way,
// so that a bracket times one kernel alone and not its overlap with the neighbours.
bool profiling_enabled();

#ifdef __CUDACC__
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent_cluster(
    void (*kernel)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
    static const bool enabled = getenv("CAMEL_TENSOR_NO_PDL") == nullptr;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = grid;
    cfg.blockDim         = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs    = attr;
    cfg.numAttrs = 0;
    if (cluster > 1) {
        attr[cfg.numAttrs].id               = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)cluster;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    if (enabled && !profiling_enabled()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        ++cfg.numAttrs;
    }
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(
    void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
    return launch_dependent_cluster(kernel, 1, grid, block, smem, s, std::forward<Args>(args)...);
}
#endif

// When profiling is on (ct_profile_enable), brackets the launches made in its scope with CUDA
// events on the launching stream, filed under `name` (a string literal).
class ProfScope {
  public:
    explicit ProfScope(const char *name);
    ~ProfScope();
    ProfScope(const ProfScope &)            = delete;
    ProfScope &operator=(const ProfScope &) = delete;

  private:
    const char *name_;
    cudaEvent_t e0_, e1_;
};

inline size_t dtype_size(int dt) { return dt == CT_F32 ? 4 : (dt == CT_I64 ? 8 : 1); }
inline bool valid_dtype(int dt) { return dt == CT_F32 || dt == CT_I64 || dt == CT_BOOL; }

// Entry points of the other translation units used across files.
// The B operand of a float32 GEMM already in the layout the tensor-core kernel reads: transposed
// [n][kp] hi/lo planes (tf32, and scaled float16 pairs where the matrix fits them) or one bf16 plane, built
// once from a [k][n] weight matrix.
struct PackedWeights {
    uint32_t magic;
    int mode;
    int device;
    int64_t k, n, kp;
    const float *src; // the matrix the planes were built from
    void *base;       // one device allocation holding the planes
    void *hi, *lo;
    void *hi16, *lo16; // float16 planes and inverse column scales; null: the matrix needs tf32
    float *scale;
    HalfExceptions *exceptions; // of the float16 planes
};
constexpr uint32_t kPackedMagic = 0x43545057u; // "CTPW"

ct_status gemm_f32_tc(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k,
    int64_t n, int act, float *out, const PackedWeights *packed = nullptr, bool a_is_km = false);
// Products of a few tiles in one launch (gemm_direct.cu).
bool gemm_direct_applicable(const DeviceState *st, int64_t m, int64_t k, int64_t n);
ct_status gemm_direct(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k, int64_t n, int act, float *out);
// One operand of gemm_half (gemm_half.cu): K-major planes [rows][kp] of float16 pairs with an inverse scale
// per row, and of tf32 terms, which are read instead where the exceptions say so (or the caller forces it).
struct HalfOperand {
    const void *hi16, *lo16;
    const float *scale;
    const void *hi32, *lo32;
    HalfExceptions *exceptions;
    int operand; // 0 left, 1 right: whose exceptions in the list are this one's
    int64_t rows;
    int64_t line0 = 0; // the exceptions' line of row 0 (a row range of a packed operand)
};
// Row bands of one launch, see ct_matmul_packed_bands.
struct HalfBands {
    int bands = 0;
    int first[9];
    int64_t out_off[8];
    uint32_t *done = nullptr;
};
// out[z][m][n] = act(A . B[z]^T + bias) over prepared planes, B holding `batch` operands of b.rows / batch rows.
// Exceptions that are the device state's are cleared by the launch for the next product.  only_if: a device word; zero: the
// launch returns at once, else it is cleared with them.
ct_status gemm_half(
    DeviceState *st, const HalfOperand &a, const HalfOperand &b, int64_t kp, const float *bias, int act, float *out,
    bool force_wide, bool allow_splitk, const HalfBands *bands, int batch = 1, bool bias_per_row = false, uint32_t *only_if = nullptr);
// Tall products of at most 128 columns whose k is sliced (gemm_panel.cu), from A as it is and B's planes; sets FLAG_PANEL
// where the operands need the product from planes.
bool gemm_panel_applicable(const DeviceState *st, int64_t m, int64_t k, int64_t n);
ct_status gemm_panel(
    DeviceState *st, const float *a, const HalfOperand &b, int64_t kp, const float *bias, int64_t m, int64_t k, int64_t n, int act, float *out);
int gemm_tile_columns(const DeviceState *st, int64_t m, int64_t n, int64_t batch = 1); // of gemm_half and gemm_planes
// Pre-passes: rows of a row-major matrix, columns of one (transposed planes); both record exceptions.  `zero`
// words are cleared on the way (scales and col_max of a following half_split_cols, which needs them at zero).
// both_forms: the tf32 planes are written as well (no half_wide_planes needed).
ct_status half_split_rows(
    DeviceState *st, const float *in, int64_t k, int64_t kp, const HalfOperand &o, bool both_forms, uint32_t *zero,
    int64_t zero_count, const uint32_t *only_if = nullptr);
bool half_cols_is_short(int64_t kp); // one pass, which needs no col_max
ct_status half_split_cols(
    DeviceState *st, const float *in, int64_t k, int64_t kp, const HalfOperand &o, bool both_forms, uint32_t *col_max);
ct_status half_split_both(
    DeviceState *st, const float *a, const HalfOperand &oa, const float *b, const HalfOperand &ob, int64_t k, int64_t kp,
    bool both_forms, bool *done);
// tf32 planes of both operands where either needs them (n == 0 / m == 0: that operand has them already).
ct_status half_wide_planes(
    DeviceState *st, const HalfExceptions *ea, const HalfExceptions *eb, const float *a, int64_t m, bool a_is_km, void *a_hi, void *a_lo, const float *b,
    int64_t n, void *b_hi, void *b_lo, int64_t k, int64_t kp);
ct_status half_widen_rows(DeviceState *st, const HalfOperand &o, int64_t kp);
// Geometry of a stride-1 convolution run as an implicit GEMM over NHWC input planes.
struct ConvGeom {
    int c_pad;  // channels rounded up to the k-block
    int h, w;   // input height / width
    int ho, wo; // output height / width
    int kh, kw, pad;
    int th;     // output rows per tile (th * wo <= 256, multiple of 16)
    int pool = 0; // 2: store the 2x2 max-pool of the activated output (pixels-on-rows kernel only)
};

// mode: 0 = 3xTF32 (float32 hi/lo planes), 1 = bf16 (one plane).  With conv != nullptr the B
// planes are NHWC input planes [batch][h][w][c_pad] and n = ho*wo output pixels per image.
ct_status gemm_planes(
    DeviceState *st, int mode, const void *a_hi, const void *a_lo, const void *b_hi,
    const void *b_lo, int64_t m, int64_t n, int64_t kp, const float *bias, int act, float *out,
    int batch, int64_t out_batch_stride, int bias_per_row, const ConvGeom *conv = nullptr);
// x [batch][c][h*w] float32 -> NHWC planes [batch][h*w][c_pad] (transpose + split per image)
ct_status nhwc_planes(
    DeviceState *st, int mode, const float *x, int64_t batch, int64_t c, int64_t hw, int64_t c_pad,
    void *hi, void *lo);
ct_status split_rows_planes(
    DeviceState *st, int mode, const float *in, int64_t rows, int64_t k, int64_t kp, void *hi,
    void *lo);
ct_status gemm_f32_skinny(
    DeviceState *st, const float *a, const float *b, const float *bias, int64_t m, int64_t k,
    int64_t n, int act, float *out, int64_t *argmax);
// out[m][n] = A^T . B with A stored [k][m], n <= 32 (float64 accumulation, two launches)
ct_status gemm_f32_tn_skinny(
    DeviceState *st, const float *a_km, const float *b, int64_t m, int64_t k, int64_t n, float *out);
ct_status matmul_generic(
    int adt, const void *a, int bdt, const void *b, int64_t m, int64_t k, int64_t n, void *out);

} // namespace ct
