// Internal launchers shared between the translation units of the library.
#pragma once
#include "common.cuh"

namespace hqm {

// linear_generic.cu — any shape check_weight() accepts.
int launch_linear_generic(uint16_t* y, const uint16_t* x, const int32_t* x_idx, int64_t M, const hqm_weight* w, int G,
                          int C, const uint16_t* bias, cudaStream_t st);

// gemv_stream.cu — the weight-streaming path for small row counts.
constexpr int STREAM_MAX_LAYERS = 4;
constexpr int STREAM_MAX_ROWS = 16;
// What one launch multiplies: up to four layers of the same K, bit width and group size (N may differ).
// Layer l reads rows x_idx?[m] + xrow[l] of x.  With `table` set, layer l's descriptor is read on the
// device: table[3 * *sel[l] + which[l]] (3 entries per expert: w1, w2, w3), and w[l] only gives the shape.
// One entry of the device-side expert table (hqm_expert_table_build): the layer's descriptor and the tensor maps (packed
// codes, scale bytes, zero bytes) that the kernels copy their tiles with: a storage-row residue at a time, and 16 of them.
struct alignas(128) StreamEntry {
    hqm_weight w;
    unsigned char pad[128 - sizeof(hqm_weight)];
    unsigned char maps[3][128];
    unsigned char rows_maps[3][128];
};
static_assert(sizeof(StreamEntry) == 896, "table entries are 896 bytes");

struct StreamJob {
    const hqm_weight* w[STREAM_MAX_LAYERS];
    int xrow[STREAM_MAX_LAYERS];
    const StreamEntry* table;
    int experts;                        // that the table holds (0: not known)
    const int32_t* sel[STREAM_MAX_LAYERS];
    int which[STREAM_MAX_LAYERS];
    // Set only when the kernel launched in front of this one lets its successor start after everything
    // before it has completed (launch_finalize_silu_mul(..., late_trigger = true)) and the indices behind
    // `sel` are older than that: the launch then reads them, and starts on the weights, without waiting.
    int sel_settled;
    // STREAM_TMA launches only.  counters: the zeroed header of the caller's scratch buffer (arrival
    // counters of units split over several CTAs; left zero again).  y_out: when set, the launch writes the finished
    // row as bf16 (+ bias) there itself, and no finalize launch follows.
    uint32_t* counters;
    uint16_t* y_out;
    const uint16_t* bias;
};
// Every scratch buffer handed to the library starts with this many bytes of library state, zero when the buffer is
// first used (hqm_scratch_init) and zero again after every call.
constexpr size_t SCRATCH_HEADER = 64 * 1024;
enum StreamKind {
    STREAM_WARPS,   // gemv_stream.cu: the passes are split over warps
    STREAM_TMA,     // gemv_tma.cu: units are (residue, block of 16 members), rho0 counts those units, and `warps` counts CTAs
    STREAM_ROWS,    // gemv_rows.cu: units are 16 storage-row residues, rho0 counts those units, and `warps` counts CTAs
};
struct StreamPlan {
    int count;                          // layers in the launch
    int nbits, nb;                      // bit width, group size / 16
    int G[STREAM_MAX_LAYERS], C[STREAM_MAX_LAYERS];
    int rho0[STREAM_MAX_LAYERS + 1];    // first storage-row residue of each layer; [count] = all of them
    int col0[STREAM_MAX_LAYERS + 1];    // first column of each layer in a partial row; [count] = row length
    int PT;      // passes per residue (K / pass width)
    int grid;    // CTAs of the single-wave persistent grid
    int warps;   // warps of that grid: the units the passes are split over
    int toks;    // rows of x decoded per launch
    int slots;   // upper bound on the warps contributing to one residue: fp32 partials [slots][M][row length]
    StreamKind kind;
};
// 2- and 4-bit layers of the streaming kernels' formats and shapes.
bool gemv_stream_shape_ok(const hqm_weight* w, int G, int C);
// False when the layers / row count are outside what the streaming kernels cover.  `chained`: the launch is a
// link of the decode step's launch chain (its consumers read the sums); false for a linear that stands alone.
bool gemv_stream_plan(const hqm_weight* const* ws, int count, int64_t M, StreamPlan* plan, bool chained = true);
size_t gemv_stream_scratch_bytes(const StreamPlan& plan, int64_t M);
int launch_gemv_stream(float* partial, const uint16_t* x, const int32_t* x_idx, int64_t M, const StreamJob& job,
                       const StreamPlan& plan, cudaStream_t st);
// y (M, row length) = bf16(sums + bias)
int launch_finalize_linear(uint16_t* y, const float* partial, const uint16_t* bias, int64_t M, const StreamPlan& plan,
                           cudaStream_t st);
// h[p] (M, F) = silu(layer 2p) * layer 2p+1 for each pair of layers of the launch
int launch_finalize_silu_mul(uint16_t* h, const float* partial, int64_t M, const StreamPlan& plan, cudaStream_t st,
                             bool late_trigger = false);
// out[token_idx[m]] (+)= sum over the launch's layers l of route_w[l * M + m] * layer l
int launch_finalize_scatter(uint16_t* out, const float* partial, const int32_t* token_idx, const float* route_w,
                            int accumulate, int64_t M, const StreamPlan& plan, cudaStream_t st);
bool force_generic();
// gemv_tma.cu — the same for ONE row of x, tiles staged by TMA.
bool gemv_tma_plan(const hqm_weight* const* ws, int count, bool chained, StreamPlan* plan);
int tma_mode();
int launch_gemv_tma(float* partial, const uint16_t* x, const int32_t* x_idx, int64_t M, const StreamJob& job,
                    const StreamPlan& plan, cudaStream_t st);

// gemv_rows.cu — 2-bit layers with groups of 16, up to 8 rows.
constexpr int STREAM_ROWS_MAX = 8;
bool gemv_rows_shape_ok(const hqm_weight* w, int G, int C);
bool gemv_rows_plan(const hqm_weight* const* ws, int count, int64_t M, StreamPlan* plan);
int launch_gemv_rows(float* partial, const uint16_t* x, const int32_t* x_idx, int64_t M, const StreamJob& job,
                     const StreamPlan& plan, cudaStream_t st);
bool rows_cached_maps(const hqm_weight* w, int G, void* out3);        // gemv_tma.cu

// gemv_lists.cu — the experts of a MoE block whose lists are short (2-bit layers with groups of 16).
constexpr int FEW_ROWS = 8;              // rows of a short list at most
constexpr int FEW_MAX_LISTS = 32;
// Whether it is asked: what decides is how long the lists are, 2 T / E entries on average.  Where many are longer than FEW_ROWS both
// kernels run, one after the other; with two experts every list has all T tokens.  A block of 4096 -> 14336 -> 4096, us, without / with:
//    2 experts   2 tokens  96 /  74   8  98 /  83  12  98 / 104  24 106 / 114
//    4           4 tokens 130 /  92  12 164 / 130  16 164 / 160  24 164 / 172
//    8           8 tokens 262 / 160  16 295 / 205  36 295 / 282  48 296 / 319
//   16          16 tokens 505 / 307  36 545 / 374  64 593 / 514  96 638 / 605  128 677 / 695
//   32          16 tokens 740 / 425  36 1044 / 602  96 1176 / 863  128 1193 / 1025
// (33 to 36 tokens and 8 experts: 282 against 295; 17 and 18 tokens and 4: 174 against 165.)
inline bool few_tokens_ok(int64_t T, int E) { return 2 * T <= (E <= 4 ? 8 : 9) * (int64_t)E; }
struct FewPlan {
    size_t x_bytes, scale_bytes, h_bytes, part_bytes;
    size_t total() const { return x_bytes + scale_bytes + h_bytes + part_bytes; }
};
struct FewJob {
    const StreamEntry* table;
    const int32_t* counts;               // device: entries of every list
    int lists;
    const hqm_weight *w1, *w2;           // the shapes
};
bool few_plan(int64_t T, int E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, FewPlan* fp);
// Where columns k .. k + 7 (k a multiple of 8) of row m lie in a staged list of `cap` rows.
__host__ __device__ inline size_t few_staged_at(int k, int m, int cap) {
    const int c = (k >> 3) & 15;
    return (size_t)(k >> 7) * cap * 256 + (size_t)((2 * ((c >> 1) & 1) + (c & 1)) * cap + m) * 64 + (c >> 2) * 16;
}
// Gate and up projections where `largest` (GgFew) is given, else the down projections.
int launch_few_projection(const FewJob& job, const unsigned char* xt, float* partial, uint32_t* largest, cudaStream_t st);
int launch_few_silu(const FewJob& job, unsigned char* ht, const float* partial, const float* row_scale, const uint32_t* largest, float* h_scale,
                    int64_t T, cudaStream_t st);
int launch_few_combine(const FewJob& job, uint16_t* out, const float* partial, const uint16_t* y, const int32_t* entry_of, const float* token_w,
                       const float* h_scale, int64_t T, cudaStream_t st);

// router.cu — logits, top-2 indices and weights of M tokens (no per-expert lists).
int launch_router_top2(uint16_t* router_logits, float* topk_w, int32_t* topk_idx, const uint16_t* x,
                       const uint16_t* gate_w, int64_t M, int64_t K, int32_t E, cudaStream_t st);

// Per-expert row lists of routed tokens; entry_of (may be null): the list entries of token t at [2t], [2t + 1].
int launch_router_lists(int32_t* counts, int32_t* offsets, int32_t* token_idx, float* token_w, int32_t* entry_of,
                        const float* topk_w, const int32_t* topk_idx, int64_t M, int32_t E, cudaStream_t st);

// How the storage rows of a 3-bit layer repeat: row rho + i * P3 holds the same ten residues in the same slots for every
// member i; `full` whole members and `left` rows of one more.
struct Members3 {
    int P3, full, left;
    static Members3 of(const hqm_weight* w, int G) {
        int a = G, b = 10;
        while (b) { const int t = a % b; a = b; b = t; }
        const int rows = (w->N + 9) / 10, P3 = G / a;
        return Members3{P3, rows / P3, rows % P3};
    }
};
// gemv_tma.cu — 2- and 4-bit layers whose tensor maps can be encoded: what every kernel that copies tiles of them has to ask.
bool tensor_maps_ok(const hqm_weight* w, int G);
bool stream_cached_maps3(const hqm_weight* w, int G, const Members3& m, void* out4);      // words, scales, zeros, left-over words
// gemv_stream3.cu — the weight-streaming path for 3-bit layers.
constexpr int STREAM3_ROWS = 4;      // beyond it the tensor-core kernels
struct Stream3Plan {
    int P3;      // storage-row classes (rows R and R + P3 hold the same residues in the same slots)
    int PT;      // 64-column passes per class
    int rows;    // storage rows, ceil(N / 10)
    int grid, warps, slots;
};
bool gemv_stream3_plan(const hqm_weight* w, int G, int C, int64_t M, Stream3Plan* plan);
size_t gemv_stream3_scratch_bytes(const Stream3Plan& plan, int64_t M, int N);
int launch_gemv_stream3(uint16_t* y, float* partial, const uint16_t* x, const int32_t* x_idx, int64_t M,
                        const hqm_weight* w, const uint16_t* bias, int G, int C, const Stream3Plan& plan,
                        cudaStream_t st);

int* tc_error_ptr();                  // device flag the bounded waits set when they give up (device_state.cu)
void* tma_encode_entry();             // cuTensorMapEncodeTiled of the installed driver, or null
// y (M, N) = bf16(sums + bias)
int launch_rows_from_sums(uint16_t* y, const float* sums, const uint16_t* bias, int64_t M, int N, cudaStream_t st);
// Rows from which 2- and 4-bit layers go to gemm_grouped.cu.  The streaming kernels decode up to 4 rows in one
// instantiation, 5 to 8 in the next one up, and more rows in more passes over the weight.  us, streaming / here:
//   rows                      3            4            5            8           16
//   2 bit 14336 x 4096   18.0 / 19.2  18.3 / 19.1  27.4 / 19.1  29.1 / 19.1  53.7 / 19.4
//   4 bit 4096 x 4096    11.3 / 11.1  12.3 / 11.2  14.0 / 11.2  15.5 / 11.3  24.4 / 11.5
// Experts whose layers gemv_rows.cu takes (2 bit, groups of 16) come here from 9 rows on (gemv_rows.cu / here: 3 rows 36.9 / 53.6, 8 rows 48.6 / 54.4).
// 2-bit layers of three steps and more per SM leave the line to api.cu, use_rows().
constexpr int64_t GG_MIN_ROWS = 5;

// gemm_tc3.cu — tcgen05 / TMEM path for the 3-bit layers that gemm_grouped.cu does not take, from five rows on.
bool gemm_tc3_supported(const hqm_weight* w, int G, int C, int64_t M);
size_t gemm_tc3_scratch_bytes(const hqm_weight* w, int G, int64_t M);
int launch_gemm_tc3(uint16_t* y, void* scratch, const uint16_t* x, const int32_t* x_idx, int64_t M,
                    const hqm_weight* w, const uint16_t* bias, int G, int C, cudaStream_t st);

// ffn.cu — launches of the single-token MoE block: [w1; w3] of both chosen experts (4 layers), then both w2.
struct MoeDecodePlan {
    StreamPlan up, down;
    size_t router_bytes, up_bytes, h_bytes, down_bytes;
};
bool moe_decode_plan(int E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, MoeDecodePlan* mp);
// `slots` (1 or 2) experts per launch instead of the two routed ones (an expert-parallel rank's share).
bool moe_decode_plan_slots(int E, int slots, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3,
                           MoeDecodePlan* mp);

// Dispatcher used by hqm_linear and by the expert FFN: picks the streaming
// kernel when the layer's shape allows it, the generic one otherwise.
// (scratch excludes the header; counters points at it)
// `preferred`: what the fastest launch wants instead of the least that works.
size_t linear_scratch_bytes(int64_t M, const hqm_weight* w, bool preferred = false);
int launch_linear(uint16_t* y, const uint16_t* x, const int32_t* x_idx, int64_t M, const hqm_weight* w,
                  const uint16_t* bias, uint32_t* counters, void* scratch, size_t scratch_bytes, cudaStream_t st);

}  // namespace hqm
