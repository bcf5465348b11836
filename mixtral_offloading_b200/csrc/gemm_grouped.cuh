// Quantized GEMM on the 5th-generation tensor cores for several weights and row lists at once (gemm_grouped.cu).
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace hqm {

constexpr int GG_MAX_PROBLEMS = 32;
constexpr int GG_MAX_ROWS = 256;          // rows of x per pass over a weight (the MMA's N)
// The scratch that a call asks for at the least lets 16 rows at a time run on this many SMs, a third of them.  (4096 x 14336
// 2-bit, 17 rows: 81 us in that, 53 in 2 MiB, 23 with a CTA on every SM.)
constexpr int GG_LEAST_CTAS = 48;
constexpr int GG_F16_ROWS = 16;           // up to here h of an expert is staged as fp16, beyond it as bf16 (gemm_grouped.cu)

// How a launch's rows are laid out in the staged copy of x ("tiles": [K / 64][row][64], see gemm_grouped.cu): a row
// list of `cnt` rows is cut into equal chunks of at most GG_MAX_ROWS rows, padded to a multiple of 16.
struct GgRows {
    int chunks, n;                        // n = rows per chunk
    __host__ __device__ static GgRows of(int cnt, int cap = GG_MAX_ROWS) {
        GgRows r;
        r.chunks = (cnt + cap - 1) / cap;
        r.n = r.chunks == 0 ? 0 : ((cnt + r.chunks - 1) / r.chunks + 15) / 16 * 16;
        return r;
    }
    __host__ __device__ int padded() const { return chunks * n; }
};
struct GgLayout {                         // of a launch whose row count the host knows
    GgRows rows;
    int grid;
    int share;                            // units of a CTA, the last one may have fewer (0: shares of equal cost)
    int64_t cost;                         // cycles, by the rule of gg_linear_layout
};
// Upper bound of the padded rows of `rows` rows spread over `lists` lists.
inline int64_t gg_padded_rows(int64_t rows, int lists) {
    return (rows + 16 * ((int64_t)lists + rows / GG_MAX_ROWS + 1) + 15) / 16 * 16;
}

// A staged copy of x or h.
struct GgStaged {
    void* data;                           // [K / 64][rows][64]
    float* scale;                         // power-of-two factor of every row (null: 1)
    int64_t rows;
};
inline size_t gg_align(size_t v) { return (v + 1023) / 1024 * 1024; }
inline size_t gg_stage_bytes(int64_t rows, int K, bool scaled) {
    return gg_align((size_t)rows * (size_t)K * 2) + (scaled ? gg_align((size_t)rows * 4) : 0);
}
inline GgStaged gg_staged(void* at, int64_t rows, int K, bool scaled) {
    return GgStaged{at, scaled ? (float*)((uint8_t*)at + gg_align((size_t)rows * (size_t)K * 2)) : nullptr, rows};
}

// What happens to a finished sum.
enum GgMode {
    GG_LINEAR = 0,       // y[row, n] = sum (+ bias[n])
    GG_UP = 1,           // h = silu(gate) * up, staged as the next launch's x
    GG_DOWN = 2,         // out[row] (+)= weight * sum
};

struct GgJob {
    int problems;                         // weights (GG_LINEAR, one expert) or experts of the table
    const hqm_weight* w0[4];              // host descriptors of the problems (no table), GG_UP: w1
    const hqm_weight* w1[4];              // GG_UP: w3
    const StreamEntry* table;             // device table, entries 3 * e + which; shape[] then only gives the shapes
    const hqm_weight* shape;
    int which0, which1;
    const int32_t* counts;                // device: rows of every problem; null: `rows` rows, shared by all problems
    int few;                              // (counts) lists of up to `few` rows are left out
    int rows;                             // rows (counts == null), or the most all lists hold together
    GgLayout layout;                      // (counts == null)
    GgStaged x;                           // the staged rows
    GgMode mode;
    // GG_LINEAR
    void* y[4];                           // (rows, N) of each problem
    const uint16_t* bias[4];
    int y_f16;                            // y is fp16 instead of bf16
    // GG_UP
    void* ht;                             // staged h
    // GG_DOWN
    void* out;                            // (*, H)
    const int32_t* out_idx;               // row of `out` of list entry i (null: i)
    const float* row_w;                   // weight of list entry i (null: 1)
    int accumulate;
};

bool gg_supported(const hqm_weight* w, int G, int C);
// Is M rows of the layer a call for 16-bit factors?  (gemm_grouped.cu)
bool gg_takes(const hqm_weight* w, int G, int C, int64_t M);
// Layers of one K and format over M rows, with `bytes` of scratch for the staged rows and the partial tiles (grid 0: too few).
GgLayout gg_linear_layout(int64_t M, const hqm_weight* const* ws, int count, size_t bytes = SIZE_MAX);
GgLayout gg_expert_layout(int64_t M);
size_t gg_scratch_bytes(int n);           // partial tiles of a launch with up to n rows per chunk and a CTA on every SM
// Scratch with which 16 rows at a time can be multiplied on GG_LEAST_CTAS SMs, whatever the layer's size.
inline size_t gg_least_bytes(int K) { return gg_stage_bytes(16, K, true) + (size_t)GG_LEAST_CTAS * 2 * 16 * 128 * sizeof(float); }
int launch_gg(const GgJob& job, uint32_t* counters, void* scratch, size_t scratch_bytes, cudaStream_t st);

// Where gg_stage puts the rows of short lists (gemv_lists.cu); most = 0: there are none.
struct GgFew {
    int most;
    unsigned char* data;
    float* scale;                         // of list entry i
    uint32_t* largest;                    // of list entry i, cleared: [2 i] and [2 i + 1], the largest |gate| and |up| of any piece
};

// Stages rows of x (bf16 or fp16) for layers of `nbits`.  counts == null: one list of `rows` rows, else `lists` lists of together at most `rows`;
// idx: row of x of list entry i (null: i).
int launch_gg_stage(const GgStaged& to, const void* x, int x_f16, const int32_t* idx, const int32_t* counts, int lists, int64_t rows,
                    int K, int nbits, cudaStream_t st, const GgFew& few = GgFew{});

}  // namespace hqm
