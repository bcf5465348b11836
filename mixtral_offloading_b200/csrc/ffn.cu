// Expert FFN: w2( silu(w1 x) * w3 x ), with the gather of the routed rows in
// front and the routing-weight scale + accumulate into the MoE output behind
// (MixtralBLockSparseTop2MLP_HQQ.forward and the per-expert body of
// SparseMoeWrapper.forward in the reference's custom_layers.py).
#include <algorithm>

#include "common.cuh"
#include "gemm_grouped.cuh"
#include "kernels.cuh"

namespace hqm {

// h = silu(a) * b, in place in a.  Both operands are the bf16 outputs of the
// w1 / w3 linears, the product is rounded to bf16 as the reference rounds to fp16.
__global__ void silu_mul_kernel(uint16_t* __restrict__ a, const uint16_t* __restrict__ b, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float av = bf16_bits_to_float(a[i]), bv = bf16_bits_to_float(b[i]);
        const float act = round_bf16(av / (1.f + __expf(-av)));
        a[i] = float_to_bf16_bits(act * bv);
    }
}

// out[t] = (accumulate ? out[t] : 0) + w_i * y[i]; one expert touches a token at
// most once, so plain read-modify-write is race free.
__global__ void scale_scatter_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ y,
                                     const int32_t* __restrict__ token_idx, const float* __restrict__ route_w,
                                     int64_t M, int H, int accumulate) {
    const int64_t total = M * H;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / H;
        const int h = (int)(i % H);
        const int64_t t = token_idx ? token_idx[m] : m;
        const float wgt = route_w ? route_w[m] : 1.f;
        const float v = round_bf16(bf16_bits_to_float(y[i]) * wgt);
        uint16_t* dst = out + t * H + h;
        *dst = float_to_bf16_bits(accumulate ? bf16_bits_to_float(*dst) + v : v);
    }
}

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static bool same_format(const hqm_weight* a, const hqm_weight* b) {
    return a->N == b->N && a->K == b->K && a->nbits == b->nbits && a->group_size == b->group_size &&
           a->meta_group == b->meta_group;
}

// The tensor-core path: x staged, [w1; w3] with the gate fused into its epilogue (h staged for the next launch), w2.
// One expert (hqm_expert_ffn) or all experts of a block (hqm_moe_forward: `rows` = tokens, two list entries each).
struct GgPlan {
    int64_t xt_rows;
    size_t x_bytes, h_bytes, part_bytes;
    size_t total() const { return x_bytes + h_bytes + part_bytes; }
};
static bool gg_plan(int64_t entries, int lists, int64_t most, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3,
                    GgPlan* gp) {
    int G1, C1, G2, C2;
    if (force_generic() || !same_format(w1, w3) || entries > (1 << 22)) return false;
    if (check_weight(w1, &G1, &C1) != HQM_OK || check_weight(w3, &G1, &C1) != HQM_OK || check_weight(w2, &G2, &C2) != HQM_OK)
        return false;
    for (int64_t rows : {most, lists > 1 ? (int64_t)1 : most})       // (lists of any length up to the most)
        if (!gg_takes(w1, G1, C1, rows) || !gg_takes(w3, G1, C1, rows) || !gg_takes(w2, G2, C2, rows)) return false;
    if (w1->nbits != 2 || w1->group_size != 16 || w2->nbits != 2 || w2->group_size != 16) return false;   // tiles of two parts
    gp->xt_rows = gg_padded_rows(entries, lists);
    gp->x_bytes = gg_stage_bytes(gp->xt_rows, w1->K, true);
    gp->h_bytes = gg_stage_bytes(gp->xt_rows, w1->N, false);
    gp->part_bytes = gg_scratch_bytes((int)(most > GG_MAX_ROWS ? GG_MAX_ROWS : (most + 15) / 16 * 16));
    return true;
}

// The streaming path for a whole expert: w1 and w3 in one launch, then w2.
struct FusedPlan {
    StreamPlan up, down;
    int G1, C1, G2, C2;
    size_t up_bytes, h_bytes, down_bytes;
};
static bool fused_plan(int64_t M, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, const void* x,
                       FusedPlan* fp) {
    if (force_generic() || !same_format(w1, w3)) return false;
    if (check_weight(w1, &fp->G1, &fp->C1) != HQM_OK || check_weight(w3, &fp->G1, &fp->C1) != HQM_OK ||
        check_weight(w2, &fp->G2, &fp->C2) != HQM_OK)
        return false;
    if (x && (reinterpret_cast<uintptr_t>(x) & 15u) != 0) return false;
    const hqm_weight* up[2] = {w1, w3};
    const hqm_weight* down[1] = {w2};
    if (!gemv_stream_plan(up, 2, M, &fp->up) || !gemv_stream_plan(down, 1, M, &fp->down)) return false;
    fp->up_bytes = align_up(gemv_stream_scratch_bytes(fp->up, M), 256);
    fp->h_bytes = align_up((size_t)M * w1->N * 2, 256);
    fp->down_bytes = align_up(gemv_stream_scratch_bytes(fp->down, M), 256);
    return true;
}

// Rows from which an expert goes to the tensor-core kernel: where gemv_rows.cu takes its layers, those that it does not.
static bool expert_uses_gg(int64_t M, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, GgPlan* gp) {
    FusedPlan fp;
    if (M < GG_MIN_ROWS || !gg_plan(M, 1, M, w1, w2, w3, gp)) return false;
    return !(fused_plan(M, w1, w2, w3, nullptr, &fp) && fp.up.kind == STREAM_ROWS && fp.down.kind == STREAM_ROWS);
}

// The three layers one after the other: their outputs, and what a single layer's launch needs.
static size_t separate_bytes(int64_t M, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3) {
    size_t lin = 0, rows = 0;
    for (const hqm_weight* w : {w1, w3, w2}) {
        lin = std::max(lin, linear_scratch_bytes(M, w));
        rows += align_up((size_t)M * (size_t)w->N * 2, 256);
    }
    return rows + lin;
}

}  // namespace hqm

extern "C" {

size_t hqm_expert_ffn_scratch_bytes(int64_t M, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3) {
    using namespace hqm;
    if (!w1 || !w2 || !w3 || M <= 0) return 0;
    // (whatever the shapes allow, rows of x that are not 16-byte aligned take the layers one after the other)
    size_t bytes = separate_bytes(M, w1, w2, w3);
    GgPlan gp;
    FusedPlan fp;
    if (expert_uses_gg(M, w1, w2, w3, &gp)) bytes = std::max(bytes, gp.total());
    else if (fused_plan(M, w1, w2, w3, nullptr, &fp)) bytes = std::max(bytes, fp.up_bytes + fp.h_bytes + fp.down_bytes);
    return SCRATCH_HEADER + bytes;
}

int hqm_expert_ffn(uint16_t* out, const uint16_t* x, int64_t M, const int32_t* token_idx, const float* route_w,
                   int accumulate, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, void* scratch,
                   size_t scratch_bytes, void* stream) {
    using namespace hqm;
    HQM_CHECK_ARG(M >= 0 && M <= INT32_MAX, "expert_ffn: bad row count %lld", (long long)M);
    if (M == 0) return HQM_OK;
    HQM_CHECK_ARG(out && x && w1 && w2 && w3, "expert_ffn: null pointer");
    HQM_CHECK_ARG(w1->N == w3->N && w1->K == w3->K, "expert_ffn: w1 (%d,%d) and w3 (%d,%d) differ", w1->N, w1->K,
                  w3->N, w3->K);
    HQM_CHECK_ARG(w2->K == w1->N && w2->N == w1->K, "expert_ffn: w2 (%d,%d) does not map (%d) back to (%d)", w2->N,
                  w2->K, w1->N, w1->K);
    const size_t need = hqm_expert_ffn_scratch_bytes(M, w1, w2, w3);
    if (scratch == nullptr || scratch_bytes < need) {
        set_error("expert_ffn: scratch of %zu bytes given, %zu needed", scratch_bytes, need);
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "expert_ffn: scratch must be 256-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const int F = w1->N, H = w2->N;
    uint32_t* counters = (uint32_t*)scratch;
    uint8_t* p = (uint8_t*)scratch + SCRATCH_HEADER;
    GgPlan gp;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0 && expert_uses_gg(M, w1, w2, w3, &gp)) {
        // 3 launches: x staged -> h = silu(w1 x) * w3 x, staged -> w2 h, weighted, into out
        uint8_t *xt = p, *ht = p + gp.x_bytes, *parts = ht + gp.h_bytes;
        const GgStaged xs = gg_staged(xt, gp.xt_rows, w1->K, true), hs = gg_staged(ht, gp.xt_rows, w1->N, false);
        int rc = launch_gg_stage(xs, x, 0, token_idx, nullptr, 1, M, w1->K, w1->nbits, st);
        if (rc != HQM_OK) return rc;
        GgJob up{}, down{};
        up.problems = down.problems = 1;
        up.rows = down.rows = (int)M;
        up.layout = down.layout = gg_expert_layout(M);
        up.mode = GG_UP;
        up.w0[0] = w1;
        up.w1[0] = w3;
        up.x = xs;
        up.ht = ht;
        rc = launch_gg(up, counters, parts, gp.part_bytes, st);
        if (rc != HQM_OK) return rc;
        down.mode = GG_DOWN;
        down.w0[0] = w2;
        down.x = hs;
        down.out = out;
        down.out_idx = token_idx;
        down.row_w = route_w;
        down.accumulate = accumulate;
        return launch_gg(down, counters, parts, gp.part_bytes, st);
    }
    FusedPlan fp;
    if (fused_plan(M, w1, w2, w3, x, &fp)) {
        // 4 launches: [w1;w3] partials -> h = silu(a) * b -> w2 partials -> scale / accumulate into out
        float* up = (float*)p;
        uint16_t* h = (uint16_t*)(p + fp.up_bytes);
        float* down = (float*)(p + fp.up_bytes + fp.h_bytes);
        StreamJob gate_up{}, down_proj{};
        gate_up.w[0] = w1;
        gate_up.w[1] = w3;
        down_proj.w[0] = w2;
        gate_up.counters = down_proj.counters = counters;
        int rc = launch_gemv_stream(up, x, token_idx, M, gate_up, fp.up, st);
        if (rc != HQM_OK) return rc;
        rc = launch_finalize_silu_mul(h, up, M, fp.up, st);
        if (rc != HQM_OK) return rc;
        rc = launch_gemv_stream(down, h, nullptr, M, down_proj, fp.down, st);
        if (rc != HQM_OK) return rc;
        return launch_finalize_scatter(out, down, token_idx, route_w, accumulate, M, fp.down, st);
    }
    uint16_t* a = (uint16_t*)p;
    p += align_up((size_t)M * F * 2, 256);
    uint16_t* b = (uint16_t*)p;
    p += align_up((size_t)M * F * 2, 256);
    uint16_t* c = (uint16_t*)p;
    p += align_up((size_t)M * H * 2, 256);
    void* lin = p;
    const size_t lin_bytes = scratch_bytes - (size_t)(p - (uint8_t*)scratch);

    int rc = launch_linear(a, x, token_idx, M, w1, nullptr, counters, lin, lin_bytes, st);
    if (rc != HQM_OK) return rc;
    rc = launch_linear(b, x, token_idx, M, w3, nullptr, counters, lin, lin_bytes, st);
    if (rc != HQM_OK) return rc;
    const int64_t nf = M * F;
    silu_mul_kernel<<<(int)((nf + 255) / 256 > 148 * 8 ? 148 * 8 : (nf + 255) / 256), 256, 0, st>>>(a, b, nf);
    HQM_LAUNCH_CHECK();
    rc = launch_linear(c, a, nullptr, M, w2, nullptr, counters, lin, lin_bytes, st);
    if (rc != HQM_OK) return rc;
    const int64_t nh = M * H;
    scale_scatter_kernel<<<(int)((nh + 255) / 256 > 148 * 8 ? 148 * 8 : (nh + 255) / 256), 256, 0, st>>>(
        out, c, token_idx, route_w, M, H, accumulate);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

// ---- MoE block of many tokens with every expert resident: no host read-back, six to nine launches --------------------------
}  // extern "C"

namespace hqm {
// out[t] = bf16(y[i] + y[j]) of the two list entries of token t (each already weighted and rounded to bf16).
__global__ void __launch_bounds__(256) moe_combine_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ y,
                                                          const int32_t* __restrict__ entry_of, int64_t tokens, int H8) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int64_t total = tokens * H8;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / H8;
        const int c = (int)(i - t * H8);
        const uint4 a = reinterpret_cast<const uint4*>(y)[(int64_t)entry_of[2 * t] * H8 + c];
        const uint4 b = reinterpret_cast<const uint4*>(y)[(int64_t)entry_of[2 * t + 1] * H8 + c];
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float lo = __uint_as_float(av[j] << 16) + __uint_as_float(bv[j] << 16);
            const float hi = __uint_as_float(av[j] & 0xffff0000u) + __uint_as_float(bv[j] & 0xffff0000u);
            o[j] = (uint32_t)float_to_bf16_bits(lo) | ((uint32_t)float_to_bf16_bits(hi) << 16);
        }
        reinterpret_cast<uint4*>(out)[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

struct MoePlan {
    GgPlan gg;
    FewPlan few;
    bool short_lists, long_lists;             // what the lists can be: up to FEW_ROWS entries (gemv_lists.cu), more (gemm_grouped.cu)
    size_t route_bytes, y_bytes;
    size_t total() const { return route_bytes + (long_lists ? gg.total() : 0) + (short_lists ? few.total() : 0) + y_bytes; }
};
static bool moe_plan(int64_t T, int E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, MoePlan* mp) {
    if (T < 1 || T > (1 << 20) || E < 2 || E > GG_MAX_PROBLEMS || w2->N % 8 != 0 || w2->N != w1->K || w2->K != w1->N) return false;
    if (!gg_plan(2 * T, E, T, w1, w2, w3, &mp->gg)) return false;
    mp->short_lists = few_plan(T, E, w1, w2, w3, &mp->few);
    mp->long_lists = !mp->short_lists || T > FEW_ROWS;                // (a token is in a list at most once)
    mp->route_bytes = align_up((size_t)T * 2 * 4 * 5 + (size_t)(2 * E + 1) * 4, 1024);
    mp->y_bytes = align_up((size_t)T * 2 * w2->N * 2, 1024);
    return true;
}
}  // namespace hqm

extern "C" {

size_t hqm_moe_forward_scratch_bytes(int64_t T, int32_t E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3) {
    if (!w1 || !w2 || !w3) return 0;
    hqm::MoePlan mp;
    return hqm::moe_plan(T, E, w1, w2, w3, &mp) ? hqm::SCRATCH_HEADER + mp.total() : 0;
}

int hqm_moe_forward(uint16_t* out, uint16_t* router_logits, const uint16_t* x, const uint16_t* gate_w, int64_t T, int32_t E,
                    const void* table, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, void* scratch,
                    size_t scratch_bytes, void* stream) {
    using namespace hqm;
    HQM_CHECK_ARG(out && router_logits && x && gate_w && table && w1 && w2 && w3, "moe_forward: null pointer");
    HQM_CHECK_ARG(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0, "moe_forward: x and out must be 16-byte aligned");
    MoePlan mp;
    HQM_CHECK_ARG(moe_plan(T, E, w1, w2, w3, &mp), "moe_forward: %lld tokens, %d experts of these shapes are not supported", (long long)T, E);
    if (scratch == nullptr || scratch_bytes < SCRATCH_HEADER + mp.total()) {
        set_error("moe_forward: scratch of %zu bytes given, %zu needed", scratch_bytes, SCRATCH_HEADER + mp.total());
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "moe_forward: scratch must be 256-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* counters = (uint32_t*)scratch;
    uint8_t* p = (uint8_t*)scratch + SCRATCH_HEADER;
    float* topk_w = (float*)p;                                        // [T][2]
    int32_t* topk_idx = (int32_t*)(topk_w + 2 * T);                   // [T][2]
    int32_t* entry_of = topk_idx + 2 * T;                             // [T][2]: list entries of a token
    int32_t* token_idx = entry_of + 2 * T;                            // [2T]
    float* token_w = (float*)(token_idx + 2 * T);                     // [2T]
    int32_t* counts = (int32_t*)(token_w + 2 * T);                    // [E]
    int32_t* offsets = counts + E;                                    // [E + 1]
    uint16_t* y = (uint16_t*)(p + mp.route_bytes);
    uint8_t* xt = p + mp.route_bytes + mp.y_bytes;
    uint8_t* ht = xt + mp.gg.x_bytes;
    uint8_t* parts = ht + mp.gg.h_bytes;
    GgFew few{};
    uint8_t* few_ht = nullptr;
    float* few_part = nullptr;
    if (mp.short_lists) {
        uint8_t* f = mp.long_lists ? parts + mp.gg.part_bytes : xt;
        float* scales = (float*)(f + mp.few.x_bytes);                // [2T] of x, [2T] of h, [2T][2] largest pieces
        few = GgFew{FEW_ROWS, f, scales, (uint32_t*)(scales + 4 * T)};
        few_ht = f + mp.few.x_bytes + mp.few.scale_bytes;
        few_part = (float*)(few_ht + mp.few.h_bytes);
    }
    const FewJob fj{static_cast<const StreamEntry*>(table), counts, E, w1, w2};
    int rc = launch_router_top2(router_logits, topk_w, topk_idx, x, gate_w, T, w1->K, E, st);
    if (rc != HQM_OK) return rc;
    rc = launch_router_lists(counts, offsets, token_idx, token_w, entry_of, topk_w, topk_idx, T, E, st);
    if (rc != HQM_OK) return rc;
    const GgStaged xs = gg_staged(xt, mp.gg.xt_rows, w1->K, true), hs = gg_staged(ht, mp.gg.xt_rows, w1->N, false);
    rc = launch_gg_stage(xs, x, 0, token_idx, counts, E, 2 * T, w1->K, w1->nbits, st, few);
    if (rc != HQM_OK) return rc;
    GgJob up{}, down{};
    up.problems = down.problems = E;
    up.table = down.table = static_cast<const StreamEntry*>(table);
    up.counts = down.counts = counts;
    up.rows = down.rows = (int)T;
    up.few = down.few = few.most;
    up.mode = GG_UP;
    up.shape = w1;
    up.which0 = 0;
    up.which1 = 2;
    up.x = xs;
    up.ht = ht;
    if (mp.short_lists) {
        rc = launch_few_projection(fj, few.data, few_part, few.largest, st);
        if (rc != HQM_OK) return rc;
        rc = launch_few_silu(fj, few_ht, few_part, few.scale, few.largest, few.scale + 2 * T, T, st);
        if (rc != HQM_OK) return rc;
    }
    if (mp.long_lists) {
        rc = launch_gg(up, counters, parts, mp.gg.part_bytes, st);
        if (rc != HQM_OK) return rc;
    }
    down.mode = GG_DOWN;
    down.shape = w2;
    down.which0 = down.which1 = 1;
    down.x = hs;
    down.out = y;
    down.row_w = token_w;
    if (mp.long_lists) {
        rc = launch_gg(down, counters, parts, mp.gg.part_bytes, st);
        if (rc != HQM_OK) return rc;
    }
    if (mp.short_lists) {
        rc = launch_few_projection(fj, few_ht, few_part, nullptr, st);
        if (rc != HQM_OK) return rc;
        return launch_few_combine(fj, out, few_part, y, entry_of, token_w, few.scale + 2 * T, T, st);
    }
    const int64_t work = T * (w2->N / 8);
    launch_overlapped(moe_combine_kernel, (int)((work + 255) / 256 > 148 * 8 ? 148 * 8 : (work + 255) / 256), 256, 0, st, out,
                      (const uint16_t*)y, (const int32_t*)entry_of, T, (int)(w2->N / 8));
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

// ---- single-token MoE block with every expert resident: the host never learns the routing ----------
// Both experts of the token share every launch: [w1; w3] of expert A and of expert B in one streaming
// launch (4 layers), one silu-mul over both, the two w2 in one launch (2 layers, each reading its own h
// row), one weighted sum.
}  // extern "C"

namespace hqm {
bool moe_decode_plan(int E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, MoeDecodePlan* mp) {
    return moe_decode_plan_slots(E, 2, w1, w2, w3, mp);
}
bool moe_decode_plan_slots(int E, int slots, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3,
                           MoeDecodePlan* mp) {
    const hqm_weight* up[4] = {w1, w3, w1, w3};
    const hqm_weight* down[2] = {w2, w2};
    if (slots < 1 || slots > 2) return false;
    if (!same_format(w1, w3) || !gemv_stream_plan(up, 2 * slots, 1, &mp->up) || !gemv_stream_plan(down, slots, 1, &mp->down))
        return false;
    mp->router_bytes = align_up((size_t)(4 + 4 + 2 * E + 1 + 4) * 4, 256);
    mp->up_bytes = align_up(gemv_stream_scratch_bytes(mp->up, 1), 256);
    mp->h_bytes = align_up((size_t)slots * w1->N * 2, 256);
    mp->down_bytes = align_up(gemv_stream_scratch_bytes(mp->down, 1), 256);
    return true;
}
}  // namespace hqm

extern "C" {

size_t hqm_moe_decode_scratch_bytes(int32_t E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3) {
    if (!w1 || !w2 || !w3 || E < 2) return 0;
    hqm::MoeDecodePlan mp;
    if (!hqm::moe_decode_plan(E, w1, w2, w3, &mp)) return 0;
    return hqm::SCRATCH_HEADER + mp.router_bytes + mp.up_bytes + mp.h_bytes + mp.down_bytes;
}

int hqm_moe_decode(uint16_t* out, uint16_t* router_logits, const uint16_t* x, const uint16_t* gate_w, int32_t E,
                   const void* table, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3,
                   void* scratch, size_t scratch_bytes, void* stream) {
    using namespace hqm;
    HQM_CHECK_ARG(out && router_logits && x && gate_w && table && w1 && w2 && w3, "moe_decode: null pointer");
    HQM_CHECK_ARG(E >= 2 && E <= 32, "moe_decode: %d experts not supported (2..32)", E);
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15u) == 0, "moe_decode: x must be 16-byte aligned");
    MoeDecodePlan mp;
    HQM_CHECK_ARG(moe_decode_plan(E, w1, w2, w3, &mp), "moe_decode: these expert shapes are outside the streaming path");
    const size_t need = SCRATCH_HEADER + mp.router_bytes + mp.up_bytes + mp.h_bytes + mp.down_bytes;
    if (scratch == nullptr || scratch_bytes < need) {
        set_error("moe_decode: scratch of %zu bytes given, %zu needed", scratch_bytes, need);
        return HQM_ERR_SCRATCH;
    }
    HQM_CHECK_ARG((reinterpret_cast<uintptr_t>(scratch) & 255u) == 0, "moe_decode: scratch must be 256-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    // router outputs live at the head of the scratch buffer (behind the library's header)
    uint32_t* counters = (uint32_t*)scratch;
    scratch = (uint8_t*)scratch + SCRATCH_HEADER;
    float* topk_w = (float*)scratch;                    // [2] (+2 pad)
    int32_t* topk_idx = (int32_t*)(topk_w + 4);         // [2] (+2 pad)
    int rc = launch_router_top2(router_logits, topk_w, topk_idx, x, gate_w, 1, w1->K, E, st);
    if (rc != HQM_OK) return rc;
    uint8_t* p = (uint8_t*)scratch + mp.router_bytes;
    float* up = (float*)p;
    uint16_t* h = (uint16_t*)(p + mp.up_bytes);         // [2][F]: one row per chosen expert
    float* down = (float*)(p + mp.up_bytes + mp.h_bytes);
    // the experts are whatever the router wrote to topk_idx[0..1]; their descriptors come from the table
    StreamJob gate_up{}, down_proj{};
    gate_up.table = down_proj.table = static_cast<const StreamEntry*>(table);
    gate_up.experts = down_proj.experts = E;
    gate_up.counters = down_proj.counters = counters;
    for (int slot = 0; slot < 2; ++slot) {
        gate_up.w[2 * slot] = w1;
        gate_up.w[2 * slot + 1] = w3;
        gate_up.sel[2 * slot] = gate_up.sel[2 * slot + 1] = topk_idx + slot;
        gate_up.which[2 * slot] = 0;
        gate_up.which[2 * slot + 1] = 2;
        down_proj.w[slot] = w2;
        down_proj.sel[slot] = topk_idx + slot;
        down_proj.which[slot] = 1;
        down_proj.xrow[slot] = slot;
    }
    // the down projections may read the router's choice and start on their weights while the silu kernel runs:
    // that kernel releases its successor only after the gate / up launch (and so the router) has completed
    down_proj.sel_settled = 1;
    rc = launch_gemv_stream(up, x, nullptr, 1, gate_up, mp.up, st);
    if (rc != HQM_OK) return rc;
    rc = launch_finalize_silu_mul(h, up, 1, mp.up, st, /*late_trigger=*/true);
    if (rc != HQM_OK) return rc;
    rc = launch_gemv_stream(down, h, nullptr, 1, down_proj, mp.down, st);
    if (rc != HQM_OK) return rc;
    return launch_finalize_scatter(out, down, nullptr, topk_w, /*accumulate=*/0, 1, mp.down, st);
}

}  // extern "C"
