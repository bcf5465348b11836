// Error reporting, argument validation and the hqm_linear entry point.
#include <stdarg.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "gemm_grouped.cuh"
#include "kernels.cuh"

namespace hqm {

static thread_local char g_error[512] = "";
static std::atomic<long long> g_launches{0};

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long launches() { return g_launches.load(std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

int check_weight(const hqm_weight* w, int* G, int* C) {
    HQM_CHECK_ARG(w != nullptr, "weight descriptor is null");
    HQM_CHECK_ARG(w->nbits == 2 || w->nbits == 3 || w->nbits == 4, "nbits == %d isn't supported (2, 3 or 4)", w->nbits);
    HQM_CHECK_ARG(w->N > 0 && w->K > 0, "weight shape (%d, %d) must be positive", w->N, w->K);
    HQM_CHECK_ARG(w->group_size > 0 && w->N % w->group_size == 0, "N = %d is not a multiple of group_size = %d", w->N,
                  w->group_size);
    if (w->nbits != 3)
        HQM_CHECK_ARG(w->N % codes_per_word(w->nbits) == 0, "N = %d is not a multiple of %d codes per byte", w->N,
                      codes_per_word(w->nbits));
    const int64_t g = w->N / w->group_size;
    const int64_t L = g * (int64_t)w->K;
    HQM_CHECK_ARG(w->meta_group > 0 && L % w->meta_group == 0,
                  "scale/zero length %lld is not a multiple of meta_group = %d", (long long)L, w->meta_group);
    HQM_CHECK_ARG(L / w->meta_group <= INT32_MAX, "scale/zero vector too long");
    HQM_CHECK_ARG(w->meta_group_zero >= 0 && (w->meta_group_zero == 0 || L % w->meta_group_zero == 0),
                  "zero length %lld is not a multiple of meta_group_zero = %d", (long long)L, w->meta_group_zero);
    HQM_CHECK_ARG(w->W_q && w->scale_q && w->zero_q && w->ms_scale && w->mz_scale && w->ms_zero && w->mz_zero,
                  "weight descriptor holds a null tensor pointer");
    *G = (int)g;
    *C = (int)(L / w->meta_group);
    return HQM_OK;
}

// HQM_FORCE_GENERIC=1 in the environment routes every linear through the shape-agnostic
// kernel (used by the tests to check the two paths against each other).
bool force_generic() {
    static const bool on = [] {
        const char* v = getenv("HQM_FORCE_GENERIC");
        return v && v[0] == '1';
    }();
    return on;
}

static std::atomic<int> g_overlap{-1};
bool overlap_enabled() {
    int v = g_overlap.load(std::memory_order_relaxed);
    if (v < 0) {
        const char* e = getenv("HQM_NO_OVERLAP");
        v = (e && e[0] == '1') ? 0 : 1;
        g_overlap.store(v, std::memory_order_relaxed);
    }
    return v != 0;
}
int set_overlap(int on) {
    const int prev = overlap_enabled() ? 1 : 0;
    g_overlap.store(on ? 1 : 0, std::memory_order_relaxed);
    return prev;
}

// Rows from which a layer goes to the tensor-core kernel (gemm_grouped.cu); below, the streaming kernels,
// whose work per weight grows with the rows, are faster (figures at GG_MIN_ROWS).
// (3 bit: from two on, as the streaming kernel takes one row per launch: 14336 x 4096 21 us each, here 29 up to 16 rows.)
// fp16 rows go there in every format that it can read: the alternative rounds the rows and the result to bf16 (2.3e-3 from 64
// bits, 6e-4 there).
static bool use_gg(const hqm_weight* w, int G, int C, int64_t M, bool f16 = false) {
    return M >= (w->nbits == 3 ? 2 : GG_MIN_ROWS) && M <= (1 << 22) && (f16 ? gg_supported(w, G, C) : gg_takes(w, G, C, M));
}

// Large 2-bit layers with groups of 16, 2 to 5 rows, where the workspace holds the partial rows of a CTA per SM (the streaming and
// the tensor-core kernel, which take them otherwise, make do with less).  us, those / gemv_rows.cu:
//   rows             2            3            4            5            8
//   14336 x 4096     15.1 / 13.6  17.9 / 13.8  18.2 / 15.2  19.1 / 16.2  19.1 / 19.3
//   4096 x 14336     17.6 / 17.4  20.3 / 17.4  20.5 / 17.9  20.7 / 19.9  20.7 / 19.8
//   8192 x 8192      16.3 / 14.8  19.5 / 15.6  19.5 / 15.6  20.8 / 17.4  20.9 / 18.2
//   14336 x 14336     295 / 24.3  48.1 / 25.0  48.3 / 25.8  48.6 / 32.1  50.6 / 36.0  (two rows: the general kernel)
// and below three steps for every SM (448 and more above):
//   12288 x 4096     13.0 / 11.6  16.0 / 12.2  16.1 / 12.3  18.3 / 13.5  18.4 / 15.1  (384 steps)
//   8192 x 5120      15.0 / 12.8  15.2 / 13.9  15.2 / 14.8  15.8 / 15.5  15.9 / 16.6  (320)
//   6144 x 6144      14.9 / 12.5  13.5 / 12.8  13.5 / 13.9  17.0 / 14.1  17.2 / 15.5  (288)
//   4096 x 4096       9.9 / 10.4   9.4 / 10.5  10.1 / 11.6  10.9 / 12.5  (128)
//   3072 x 5120       9.4 / 10.6   9.5 / 11.3   9.9 / 11.8  11.1 / 12.3  (120)
// The line is on the safe side of where the two meet, somewhere between 130 and 290 steps.
static bool use_rows(int64_t M, const hqm_weight* w, StreamPlan* plan, size_t* bytes) {
    const hqm_weight* one[1] = {w};
    if (M < 2 || M > 5 || force_generic() || !gemv_rows_plan(one, 1, M, plan) || plan->rho0[1] * plan->PT < 3 * plan->grid) return false;
    *bytes = (gemv_stream_scratch_bytes(*plan, M) + 255) / 256 * 256;
    return true;
}

// The kernels beside gemm_grouped.cu: what the one that takes the call needs.
static size_t other_scratch_bytes(int64_t M, const hqm_weight* w, int G, int C) {
    if (gemm_tc3_supported(w, G, C, M)) return gemm_tc3_scratch_bytes(w, G, M);
    Stream3Plan plan3;
    if (gemv_stream3_plan(w, G, C, M, &plan3)) return gemv_stream3_scratch_bytes(plan3, M, w->N);
    StreamPlan plan;
    const hqm_weight* one[1] = {w};
    if (!gemv_stream_plan(one, 1, M, &plan, /*chained=*/false)) return 0;
    return (gemv_stream_scratch_bytes(plan, M) + 255) / 256 * 256;
}

// The least is a contract with callers whose memory plan is fixed: the fp32 sums of the call, or what the streaming and
// 3-bit kernels leave behind for as few rows as they take.  The tensor-core kernel makes do with that (linear_gg); it only
// wants room for 16 rows at a time on a third of the SMs.
size_t linear_scratch_bytes(int64_t M, const hqm_weight* w, bool preferred) {
    int G, C;
    if (M <= 0 || check_weight(w, &G, &C) != HQM_OK || force_generic()) return 0;
    if (preferred) {
        StreamPlan plan;
        size_t bytes;
        if (use_rows(M, w, &plan, &bytes)) return std::max(bytes, linear_scratch_bytes(M, w));
    }
    if (!use_gg(w, G, C, M)) return other_scratch_bytes(M, w, G, C);
    const size_t sums = w->nbits != 3 && M > STREAM_MAX_ROWS ? (size_t)M * w->N * sizeof(float) : other_scratch_bytes(M, w, G, C);
    const size_t least = std::max(gg_least_bytes(w->K), (sums + 255) / 256 * 256);
    if (!preferred) return least;
    const GgRows rows = gg_linear_layout(M, &w, 1).rows;
    return std::max(least, gg_stage_bytes(rows.padded(), w->K, true) + gg_scratch_bytes(rows.n));
}

static int need_scratch(void* scratch, size_t have, size_t need) {
    if (scratch == nullptr || have < need) {
        set_error("linear: scratch of %zu bytes given, %zu needed", have, need);
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 15u) == 0, "linear: scratch must be 16-byte aligned");
    return HQM_OK;
}

// Layers of one K and format over the same rows: the rows staged once, one launch over all tiles.  With less scratch than
// that wants, narrower chunks and fewer CTAs, or the rows in several passes, by the cost that gg_linear_layout gives.
static int linear_gg(uint16_t* const* y, const hqm_weight* const* ws, const uint16_t* const* bias, int count, const uint16_t* x,
                     const int32_t* x_idx, int64_t M, uint32_t* counters, void* scratch, size_t scratch_bytes, cudaStream_t st,
                     int f16 = 0) {
    const int K = ws[0]->K;
    int rc = need_scratch(scratch, scratch_bytes, gg_least_bytes(K));
    if (rc != HQM_OK) return rc;
    GgLayout layout = gg_linear_layout(M, ws, count, scratch_bytes);
    int64_t rows = M;
    if (layout.grid == 0 || gg_stage_bytes(layout.rows.padded(), K, true) + gg_scratch_bytes(layout.rows.n) > scratch_bytes) {
        rc = need_scratch(scratch, scratch_bytes, linear_scratch_bytes(M, ws[0]));
        if (rc != HQM_OK) return rc;
        constexpr int64_t PASS = 10000;          // cycles of two more launches
        int64_t best = layout.grid ? layout.cost : INT64_MAX;
        const int64_t most = (M + 15) / 16;
        for (int64_t passes = 2; passes <= most; passes = passes == most ? most + 1 : std::min(most, passes + 1 + passes / 4)) {
            const int64_t r = ((M + passes - 1) / passes + 15) / 16 * 16;
            const GgLayout l = gg_linear_layout(r, ws, count, scratch_bytes);
            if (l.grid && passes * (l.cost + PASS) < best) {
                best = passes * (l.cost + PASS);
                layout = l;
                rows = r;
            }
        }
    }
    for (int64_t r0 = 0; r0 < M; r0 += rows) {
        const int64_t m = std::min(rows, M - r0);
        if (r0 > 0 && m < rows) layout = gg_linear_layout(m, ws, count, scratch_bytes);
        const int64_t xt_rows = layout.rows.padded();
        const size_t staged = gg_stage_bytes(xt_rows, K, true);
        const GgStaged xs = gg_staged(scratch, xt_rows, K, true);
        rc = launch_gg_stage(xs, x_idx ? x : x + r0 * K, f16, x_idx ? x_idx + r0 : nullptr, nullptr, 1, m, K, ws[0]->nbits, st);
        if (rc != HQM_OK) return rc;
        GgJob job{};
        job.problems = count;
        job.rows = (int)m;
        job.layout = layout;
        job.x = xs;
        job.mode = GG_LINEAR;
        job.y_f16 = f16;
        for (int i = 0; i < count; ++i) {
            job.w0[i] = ws[i];
            job.y[i] = y[i] + r0 * ws[i]->N;
            job.bias[i] = bias ? bias[i] : nullptr;
        }
        rc = launch_gg(job, counters, (uint8_t*)scratch + staged, scratch_bytes - staged, st);
        if (rc != HQM_OK) return rc;
    }
    return HQM_OK;
}

int launch_linear(uint16_t* y, const uint16_t* x, const int32_t* x_idx, int64_t M, const hqm_weight* w,
                  const uint16_t* bias, uint32_t* counters, void* scratch, size_t scratch_bytes, cudaStream_t st) {
    int G, C;
    int rc = check_weight(w, &G, &C);
    if (rc != HQM_OK) return rc;
    if (M == 0) return HQM_OK;
    StreamPlan plan;
    const bool x_ok = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    if (!x_ok || force_generic()) return launch_linear_generic(y, x, x_idx, M, w, G, C, bias, st);
    size_t rows_bytes;
    if (scratch != nullptr && (reinterpret_cast<uintptr_t>(scratch) & 15u) == 0 && use_rows(M, w, &plan, &rows_bytes) && scratch_bytes >= rows_bytes) {
        StreamJob job{};
        job.w[0] = w;
        job.counters = counters;
        rc = launch_gemv_stream((float*)scratch, x, x_idx, M, job, plan, st);
        return rc != HQM_OK ? rc : launch_finalize_linear(y, (const float*)scratch, bias, M, plan, st);
    }
    if (use_gg(w, G, C, M)) {
        return linear_gg(&y, &w, &bias, 1, x, x_idx, M, counters, scratch, scratch_bytes, st);
    }
    if (gemm_tc3_supported(w, G, C, M)) {
        rc = need_scratch(scratch, scratch_bytes, gemm_tc3_scratch_bytes(w, G, M));
        return rc != HQM_OK ? rc : launch_gemm_tc3(y, scratch, x, x_idx, M, w, bias, G, C, st);
    }
    Stream3Plan plan3;
    if (gemv_stream3_plan(w, G, C, M, &plan3)) {
        rc = need_scratch(scratch, scratch_bytes, gemv_stream3_scratch_bytes(plan3, M, w->N));
        return rc != HQM_OK ? rc : launch_gemv_stream3(y, (float*)scratch, x, x_idx, M, w, bias, G, C, plan3, st);
    }
    const hqm_weight* one[1] = {w};
    if (gemv_stream_plan(one, 1, M, &plan, /*chained=*/false)) {
        rc = need_scratch(scratch, scratch_bytes, gemv_stream_scratch_bytes(plan, M));
        if (rc != HQM_OK) return rc;
        StreamJob job{};
        job.w[0] = w;
        job.counters = counters;
        if (plan.kind == STREAM_TMA) {                      // the launch finishes the row itself: bf16, bias added
            job.y_out = y;
            job.bias = bias;
            return launch_gemv_stream((float*)scratch, x, x_idx, M, job, plan, st);
        }
        rc = launch_gemv_stream((float*)scratch, x, x_idx, M, job, plan, st);
        if (rc != HQM_OK) return rc;
        return launch_finalize_linear(y, (const float*)scratch, bias, M, plan, st);
    }
    return launch_linear_generic(y, x, x_idx, M, w, G, C, bias, st);
}

// Workspace, header included, of a launch over several layers; 0 where the tensor-core kernel does not take them.
static size_t group_scratch_bytes(int64_t M, const hqm_weight* const* w, int count, bool f16) {
    if (M <= 0 || count < 1 || count > 4 || w == nullptr || force_generic()) return 0;
    for (int i = 0; i < count; ++i) {
        int G, C;
        if (check_weight(w[i], &G, &C) != HQM_OK || !use_gg(w[i], G, C, M, f16)) return 0;
        if (w[i]->K != w[0]->K || w[i]->nbits != w[0]->nbits || w[i]->group_size != w[0]->group_size) return 0;
    }
    const GgRows rows = gg_linear_layout(M, w, count).rows;
    return SCRATCH_HEADER + gg_stage_bytes(rows.padded(), w[0]->K, true) + gg_scratch_bytes(rows.n);
}

}  // namespace hqm

extern "C" {

const char* hqm_last_error(void) { return hqm::g_error; }
int hqm_version(void) { return 1; }
int64_t hqm_launch_count(void) { return (int64_t)hqm::launches(); }
int hqm_set_overlap(int on) { return hqm::set_overlap(on); }

size_t hqm_scratch_header_bytes(void) { return hqm::SCRATCH_HEADER; }

int hqm_scratch_init(void* scratch, void* stream) {
    using namespace hqm;
    HQM_CHECK_ARG(scratch != nullptr, "scratch_init: null pointer");
    HQM_CUDA(cudaMemsetAsync(scratch, 0, SCRATCH_HEADER, (cudaStream_t)stream));
    return HQM_OK;
}

size_t hqm_linear_scratch_bytes(int64_t M, const hqm_weight* w) {
    const size_t inner = hqm::linear_scratch_bytes(M, w);
    return inner ? inner + hqm::SCRATCH_HEADER : 0;
}

size_t hqm_linear_scratch_preferred(int64_t M, const hqm_weight* w) {
    const size_t inner = hqm::linear_scratch_bytes(M, w, /*preferred=*/true);
    return inner ? inner + hqm::SCRATCH_HEADER : 0;
}

size_t hqm_linear_f16_scratch_bytes(int64_t M, const hqm_weight* w) { return hqm::group_scratch_bytes(M, &w, 1, /*f16=*/true); }

int hqm_linear_f16(uint16_t* y, const uint16_t* x, int64_t M, const hqm_weight* w, const uint16_t* bias, void* scratch,
                   size_t scratch_bytes, void* stream) {
    using namespace hqm;
    const size_t need = hqm_linear_f16_scratch_bytes(M, w);
    HQM_CHECK_ARG(need != 0, "linear_f16: rows and a layer that the tensor-core kernel takes are needed");
    HQM_CHECK_ARG(y && x && (reinterpret_cast<uintptr_t>(x) & 15u) == 0, "linear_f16: null or unaligned activation pointer");
    if (scratch == nullptr || scratch_bytes < need) {
        set_error("linear_f16: scratch of %zu bytes given, %zu needed", scratch_bytes, need);
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "linear_f16: scratch must be 256-byte aligned");
    return linear_gg(&y, &w, &bias, 1, x, nullptr, M, (uint32_t*)scratch, (uint8_t*)scratch + SCRATCH_HEADER,
                     scratch_bytes - SCRATCH_HEADER, (cudaStream_t)stream, 1);
}

size_t hqm_linear_group_scratch_bytes(int64_t M, const hqm_weight* const* w, int32_t count) {
    return hqm::group_scratch_bytes(M, w, count, /*f16=*/false);
}

int hqm_linear_group(uint16_t* const* y, const uint16_t* x, int64_t M, const hqm_weight* const* w, const uint16_t* const* bias,
                     int32_t count, void* scratch, size_t scratch_bytes, void* stream) {
    using namespace hqm;
    const size_t need = hqm_linear_group_scratch_bytes(M, w, count);
    HQM_CHECK_ARG(need != 0, "linear_group: layers of one K and format, and rows that the tensor-core kernel takes, are needed");
    HQM_CHECK_ARG(y && x && (reinterpret_cast<uintptr_t>(x) & 15u) == 0, "linear_group: null or unaligned activation pointer");
    for (int i = 0; i < count; ++i) HQM_CHECK_ARG(y[i] != nullptr, "linear_group: null output %d", i);
    if (scratch == nullptr || scratch_bytes < need) {
        set_error("linear_group: scratch of %zu bytes given, %zu needed", scratch_bytes, need);
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "linear_group: scratch must be 256-byte aligned");
    return linear_gg(y, w, bias, count, x, nullptr, M, (uint32_t*)scratch, (uint8_t*)scratch + SCRATCH_HEADER,
                     scratch_bytes - SCRATCH_HEADER, (cudaStream_t)stream);
}

int hqm_linear(uint16_t* y, const uint16_t* x, int64_t M, const hqm_weight* w, const uint16_t* bias, void* scratch,
               size_t scratch_bytes, void* stream) {
    using namespace hqm;
    HQM_CHECK_ARG(M >= 0 && M <= INT32_MAX, "linear: bad row count %lld", (long long)M);
    HQM_CHECK_ARG(M == 0 || (y && x), "linear: null activation pointer");
    if (scratch == nullptr || scratch_bytes <= SCRATCH_HEADER)
        return launch_linear(y, x, nullptr, M, w, bias, nullptr, nullptr, 0, (cudaStream_t)stream);
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "linear: scratch must be 256-byte aligned");
    return launch_linear(y, x, nullptr, M, w, bias, (uint32_t*)scratch, (uint8_t*)scratch + SCRATCH_HEADER,
                         scratch_bytes - SCRATCH_HEADER, (cudaStream_t)stream);
}

}  // extern "C"
