// The experts of a MoE block with few rows each (up to FEW_ROWS), all of them in one launch per projection; how long their row
// lists are only the device knows.  Replaces the per-expert loop of the reference (custom_layers.py:243-256, 295-312) for a small
// batch of sequences or a short prompt.  Lists with more rows are left to gemm_grouped.cu.
//
// The arithmetic, the stage and what bounds them are gemv_rows.cu's.  Here every list is a problem: units of (16 storage-row
// residues, all of K) of its one or two layers, in steps of 128 columns whose cost depends on the list's length (up to 4 rows: 4,
// up to 8: 5; measured 2.0 and 2.4 us per step in a launch of 36).  The steps of all lists follow each other and every CTA takes an equal share of
// their cost.  A CTA leaves one fp32 partial row-set per unit that it touched; the kernels behind add them in CTA order.  Since
// the share depends on the lists' lengths, every kernel computes the split anew (ListSplit, a warp's prefix sums).
//
// The rows of a list are staged by gg_stage_kernel, h by few_silu_kernel: fp16 in the order in which a step reads them,
// [step][half][16-byte piece][row][thread column], with a power of two per row.
//
// Measured on B200, 8 experts 4096 -> 14336 -> 4096, 8 tokens, up + gate / down: 202 / 98 us through the tensor-core kernel (whose
// dequantisation takes 1345 warp instructions for 8192 codes), 95 / 49 here: 565 warp instructions, 60 % of the issue slots and 59 % of
// shared memory's cycles in use; the copies alone take 56 / 30.
#include <algorithm>

#include "gemv_rows.cuh"

namespace hqm {

namespace rows {

constexpr uint32_t COST_4 = 4, COST_8 = 5;
// How a launch's steps are split; computed by a warp.
struct ListSplit {
    int n[FEW_MAX_LISTS], list0[FEW_MAX_LISTS + 1];                 // rows of a list, its first entry among those of all lists
    int row0[FEW_MAX_LISTS + 1], xrow0[FEW_MAX_LISTS + 1];          // of the short lists: first partial row, first staged row
    uint32_t step0[FEW_MAX_LISTS + 1], cost0[FEW_MAX_LISTS + 1];    // steps and their cost in front of a list
    int lists, grid, R;                                             // CTAs that have steps; rows of all short lists

    __host__ __device__ static int cap(int n) { return n == 0 || n > FEW_ROWS ? 0 : (n <= 4 ? 4 : 8); }     // staged rows
    __device__ __forceinline__ uint32_t cost(int e) const { return n[e] <= 4 ? COST_4 : COST_8; }
    __device__ void make(const int32_t* counts, int E, uint32_t steps, int ctas) {
        const int lane = threadIdx.x & 31;
        const int c = lane < E ? __ldcg(counts + lane) : 0;
        const int few = c <= FEW_ROWS ? c : 0, k = cap(c);
        int list = c, row = few, xrow = k;
        uint32_t st = k ? steps : 0u, co = st * (c <= 4 ? COST_4 : COST_8);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, list, o), b = __shfl_up_sync(0xffffffffu, row, o), d = __shfl_up_sync(0xffffffffu, xrow, o);
            const uint32_t s = __shfl_up_sync(0xffffffffu, st, o), t = __shfl_up_sync(0xffffffffu, co, o);
            if (lane >= o) {
                list += a;
                row += b;
                xrow += d;
                st += s;
                co += t;
            }
        }
        if (lane < E) {
            n[lane] = c;
            list0[lane + 1] = list;
            row0[lane + 1] = row;
            xrow0[lane + 1] = xrow;
            step0[lane + 1] = st;
            cost0[lane + 1] = co;
        }
        if (lane == 0) list0[0] = row0[0] = xrow0[0] = 0, step0[0] = cost0[0] = 0u, lists = E;
        if (lane == E - 1) {
            R = row;
            // (a share of at least the dearest step: every CTA up to `grid` has one)
            grid = max(1, min(ctas, (int)(co / COST_8)));
        }
    }
    // First step of CTA c's share.
    __device__ uint32_t begin(int c) const {
        if (c >= grid) return step0[lists];
        const uint32_t at = (uint32_t)((uint64_t)cost0[lists] * (uint32_t)c / (uint32_t)grid);
        int e = 0;
        while (e < lists - 1 && at >= cost0[e + 1]) ++e;
        return step0[e] + (at - cost0[e] + cost(e) - 1) / cost(e);
    }
    // The CTA whose share holds step s of list e: the last one that begins at or before it.
    __device__ __forceinline__ int owner(int e, uint32_t s) const {
        const uint64_t at = cost0[e] + (uint64_t)s * cost(e) + 1;
        return (int)((at * (uint32_t)grid + cost0[lists] - 1) / cost0[lists]) - 1;
    }
    __device__ __forceinline__ int list_of(int entry) const {
        int e = 0;
        while (e < lists - 1 && entry >= list0[e + 1]) ++e;
        return e;
    }
};

struct ListParams {
    const StreamEntry* table;
    const int32_t* counts;
    int lists, layers, which0, which1;                  // layers of an expert in this launch, and their table entries
    int K, PT, N, G, C, units, period, stages, stage_bytes, x_off;      // units: of a layer
    const unsigned char* xt;
    float* partial;
    uint32_t* largest;                                  // (two layers) see GgFew
    int* error_flag;
};

// A run of steps of one unit: list, unit of the list, steps [pa, pb) of it.
struct Run {
    int e, unit, pa, pb;
    // That of step u; the caller's steps end at ue, and list `from` does not lie behind the step's.
    __device__ __forceinline__ static Run at(const ListSplit& sp, int PT, uint32_t ue, uint32_t u, int from) {
        Run r;
        r.e = from;
        while (u >= sp.step0[r.e + 1]) ++r.e;
        const uint32_t rel = u - sp.step0[r.e];
        r.unit = (int)(rel / (uint32_t)PT);
        r.pa = (int)(rel - (uint32_t)r.unit * (uint32_t)PT);
        r.pb = (int)min((uint32_t)PT, (uint32_t)r.pa + (ue - u));
        return r;
    }
};

// sum_again() for the runs of this warp in the steps [u, ue).
__device__ __noinline__ void lists_again(const ListParams& prm, const ListSplit& sp, uint32_t u, uint32_t ue) {
    const int warp = threadIdx.x >> 5, K = prm.K, row_len = prm.layers * prm.N;
    while (u < ue) {
        const Run r = Run::at(sp, prm.PT, ue, u, 0);
        u += (uint32_t)(r.pb - r.pa);
        const int layer = r.unit / prm.units, rho = (r.unit - layer * prm.units) * CW + warp;
        if (rho * PER >= prm.G) continue;
        const int piece = r.pa ? (int)blockIdx.x - sp.owner(r.e, (uint32_t)(r.unit * prm.PT)) : 0;
        Again a{};
        a.layer(prm.table[3 * r.e + (layer ? prm.which1 : prm.which0)].w);
        a.K = K;
        a.G = prm.G;
        a.C = prm.C;
        a.rho = rho;
        a.k0 = r.pa * KC;
        a.k1 = r.pb * KC;
        a.staged = prm.xt + (size_t)sp.xrow0[r.e] * K * 2;
        a.cap = ListSplit::cap(sp.n[r.e]);
        for (a.m = 0; a.m < sp.n[r.e]; ++a.m) {
            const float v = sum_again(a, prm.partial + ((size_t)piece * sp.R + sp.row0[r.e] + a.m) * row_len + layer * prm.N + PER * rho, 1.f);
            if (prm.layers == 2 && v > 0.f && (threadIdx.x & 31) == 0) atomicMax(prm.largest + 2 * (sp.list0[r.e] + a.m) + layer, __float_as_uint(v));
        }
    }
}

__global__ void __launch_bounds__(THREADS, 1) gemv_lists_kernel(const __grid_constant__ ListParams prm) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ ListSplit sp;
    __shared__ uint32_t s_begin[2];
    __shared__ int s_failed, s_again;
    __shared__ uint32_t s_largest[FEW_MAX_LISTS * 2 * FEW_ROWS];        // of [list][layer][row], this CTA's
    __shared__ int s_largest_at[CW];                                    // of each computing warp's run
    __shared__ __align__(8) uint64_t s_bars[2 * MAX_STAGES];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t exch = ring + prm.stages * prm.stage_bytes;
    const uint32_t full = smem_u32(s_bars), empty = full + 8 * MAX_STAGES;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int K = prm.K, PT = prm.PT, cta = (int)blockIdx.x;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        init_barriers(full, empty, prm.stages);
        s_failed = s_again = 0;
    }
    for (int i = threadIdx.x; i < FEW_MAX_LISTS * 2 * FEW_ROWS; i += THREADS) s_largest[i] = 0u;
    // the table's entries in L2 by the time the lists are known
    for (int i = threadIdx.x; i < 4 * prm.layers * prm.lists; i += THREADS) {
        const StreamEntry* en = prm.table + 3 * ((i >> 2) / prm.layers) + ((i >> 2) % prm.layers ? prm.which1 : prm.which0);
        prefetch_l2((i & 3) == 0 ? reinterpret_cast<const void*>(&en->w) : en->rows_maps[(i & 3) - 1]);
    }
    grid_dependency_wait();
    if (warp == 0) {
        sp.make(prm.counts, prm.lists, (uint32_t)(prm.layers * prm.units * PT), (int)gridDim.x);
        __syncwarp();
        if (lane < 2) s_begin[lane] = sp.begin(cta + lane);
    }
    __syncthreads();
    const uint32_t ub = s_begin[0], ue = s_begin[1];

    auto run_at = [&](uint32_t u, int from) { return Run::at(sp, PT, ue, u, from); };

    if (warp == CW) {
        // =========================== copies ===========================
        const uint32_t C = (uint32_t)prm.C;
        const StepCopy copy{prm.period, lane, C, (uint32_t)K % C, elect_one()};
        const int hi = lane >> 4;
        int st = 0, fenced = -1, e = 0;
        uint32_t par = 1;
        bool ok = true;
        for (uint32_t u = ub; u < ue && ok;) {
            const Run r = run_at(u, e);
            u += (uint32_t)(r.pb - r.pa);
            e = r.e;
            const int layer = r.unit / prm.units;
            const StreamEntry* en = prm.table + 3 * e + (layer ? prm.which1 : prm.which0);
            const CUtensorMap* maps = reinterpret_cast<const CUtensorMap*>(en->rows_maps);
            const uint16_t *src0 = hi ? en->w.mz_scale : en->w.ms_scale, *src1 = hi ? en->w.mz_zero : en->w.ms_zero;
            if (fenced != 2 * e + layer) {
                fenced = 2 * e + layer;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(maps + i) : "memory");
            }
            const int rho = (r.unit - layer * prm.units) * CW;
            const uint32_t x_bytes = (uint32_t)ListSplit::cap(sp.n[e]) * (KC * 2);
            const unsigned char* xs = prm.xt + (size_t)sp.xrow0[e] * K * 2 + (size_t)r.pa * x_bytes;
            uint32_t col = (uint32_t)(r.pa * KC) % C;
            for (int p = r.pa; p < r.pb; ++p) {
                if (!wait(empty + 8 * st, par)) {
                    ok = false;
                    break;
                }
                const uint32_t dst = ring + st * prm.stage_bytes, bar = full + 8 * st;
                copy(dst, bar, maps, p * KC, rho, src0, src1, col, x_bytes);
                if (copy.elected)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(dst + prm.x_off), "l"(xs), "r"(x_bytes), "r"(bar)
                                 : "memory");
                xs += x_bytes;
                col += KC;
                col = col >= C ? col - C : col;
                if (++st == prm.stages) {
                    st = 0;
                    par ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");        // (no lane leaves with copies on their way)
        if (!ok) s_failed = 1;
    } else {
        // =========================== computing warps ===========================
        int st = 0, e = 0;
        uint32_t par = 0;
        bool ok = true;
        const int row_len = prm.layers * prm.N;
        for (uint32_t u = ub; u < ue && ok;) {
            const Run r = run_at(u, e);
            u += (uint32_t)(r.pb - r.pa);
            e = r.e;
            const int layer = r.unit / prm.units;
            const int rho = (r.unit - layer * prm.units) * CW + warp;
            const int piece = r.pa ? cta - sp.owner(e, (uint32_t)(r.unit * PT)) : 0;
            const Segment sg{ring, full, empty, exch + warp * EXCH_BYTES, prm.stage_bytes, prm.stages, prm.period,
                             (PER * rho + (lane >> 3)) % prm.period, sp.n[e], prm.G, row_len, rho * PER < prm.G};
            float* dst = prm.partial + ((size_t)piece * sp.R + sp.row0[e]) * row_len + layer * prm.N + PER * rho;
            const auto one = [](int) { return 1.f; };
            uint32_t* largest = prm.layers == 2 ? s_largest : nullptr;
            __syncwarp();                               // (the last run's has been read)
            if (lane == 0) s_largest_at[warp] = (2 * e + layer) * FEW_ROWS;
            __syncwarp();
            if (sg.M <= 4) ok = rows_segment<4, true>(sg, r.pb - r.pa, st, par, (uint32_t)prm.x_off, 0u, dst, one, s_again, largest, s_largest_at + warp);
            else ok = rows_segment<8, true>(sg, r.pb - r.pa, st, par, (uint32_t)prm.x_off, 0u, dst, one, s_again, largest, s_largest_at + warp);
        }
        if (!ok) s_failed = 1;
    }
    __syncthreads();
    if (prm.layers == 2)
        for (int i = threadIdx.x; i < FEW_MAX_LISTS * 2 * FEW_ROWS; i += THREADS)
            if (const uint32_t v = s_largest[i])
                atomicMax(prm.largest + 2 * (sp.list0[i / (2 * FEW_ROWS)] + i % FEW_ROWS) + i / FEW_ROWS % 2, v);
    if (s_again && !s_failed && warp < CW) lists_again(prm, sp, s_begin[0], s_begin[1]);
    // ---- a wait ran out: copies may still be on their way to this CTA's shared memory
    if (s_failed) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        if (threadIdx.x == 0 && prm.error_flag) atomicExch(prm.error_flag, 1);
    }
}

// Sum of the pieces of four neighbouring columns of a row.
__device__ __forceinline__ float4 sum_pieces(const ListSplit& sp, const float* partial, int e, int m, int unit, int PT, int col, int row_len) {
    const int cnt = sp.owner(e, (uint32_t)(unit * PT + PT - 1)) - sp.owner(e, (uint32_t)(unit * PT)) + 1;
    const float* at = partial + (size_t)(sp.row0[e] + m) * row_len + col;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 0; i < cnt; ++i) {
        const float4 p = *reinterpret_cast<const float4*>(at + (size_t)i * sp.R * row_len);
        v.x += p.x;
        v.y += p.y;
        v.z += p.z;
        v.w += p.w;
    }
    return v;
}

// h = bf16(bf16(silu(bf16(gate))) * bf16(up)) of the short lists, staged for the down projections as fp16 with a power of two per
// row: h of 1e-6 times a scale of 0.02 would be a denormal in fp16 (a block of weights of 1e-4: 0.24 from 64 bits without the factor).
// What decides the factor is a bound of |h| that no CTA has to wait for: the pieces of a sum times the largest of them, of gate and of
// up (the launch in front leaves both; |silu(a)| <= |a|).  The bound comes into [2^11, 2^12): h lies some 2^5 below it, typically
// between 1 and 100, far from either end of fp16.  (Blocks of 8 experts with 2 / 8 / 24 / 36 tokens, us, without
// a factor 107.3 / 158.8 / 243.8 / 281.7, so 108.6 / 159.9 / 247.3 / 283.0, and with a row's true maximum, by a cluster of CTAs per row, 108.8 /
// 160.6 / 252.8 / 288.3.)
// A thread: four columns of list entry blockIdx.y.
__global__ void __launch_bounds__(256) few_silu_kernel(unsigned char* __restrict__ ht, const float* __restrict__ partial,
                                                       const int32_t* __restrict__ counts, const float* __restrict__ row_scale,
                                                       const uint32_t* __restrict__ largest, float* __restrict__ h_scale, int lists, int ctas,
                                                       int units, int PT, int F, int G) {
    __shared__ ListSplit sp;
    grid_launch_dependents();
    grid_dependency_wait();
    if (threadIdx.x < 32) sp.make(counts, lists, (uint32_t)(2 * units * PT), ctas);
    __syncthreads();
    const int entry = blockIdx.y, f = 4 * (blockIdx.x * 256 + threadIdx.x);
    const int e = sp.list_of(entry), m = entry - sp.list0[e], cap = ListSplit::cap(sp.n[e]);
    if (cap == 0 || m >= sp.n[e] || f >= F) return;
    const int unit = f % G / PER / CW;
    const float scale = __ldcg(row_scale + entry);
    const float pieces = (float)((uint32_t)PT * sp.cost(e) / (sp.cost0[sp.lists] / (uint32_t)sp.grid) + 2u) * scale;
    const float most = (pieces * __uint_as_float(__ldcg(largest + 2 * entry))) * (pieces * __uint_as_float(__ldcg(largest + 2 * entry + 1)));
    const int ex = min(max((int)(__float_as_uint(most) >> 23), 30), 250) - 11;      // biased
    const float down = __uint_as_float((uint32_t)(254 - ex) << 23);
    if (f == 0) h_scale[entry] = __uint_as_float((uint32_t)ex << 23);
    const float4 a = sum_pieces(sp, partial, e, m, unit, PT, f, 2 * F), b = sum_pieces(sp, partial, e, m, units + unit, PT, F + f, 2 * F);
    auto act = [scale, down](float x, float y) {
        const float g = round_bf16(x * scale);
        return round_bf16(round_bf16(g / (1.f + __expf(-g))) * round_bf16(y * scale)) * down;
    };
    const uint32_t lo = h2_of(act(a.x, b.x), act(a.z, b.z)), hi = h2_of(act(a.y, b.y), act(a.w, b.w));
    *reinterpret_cast<uint2*>(ht + (size_t)sp.xrow0[e] * F * 2 + few_staged_at(f, m, cap) + ((f >> 2) & 1) * 8) = make_uint2(lo, hi);
}

// out[t] = bf16(bf16(w_i * y_i) + bf16(w_j * y_j)) of the two list entries of token t: sums of pieces where the list is short, else
// the finished rows `y` of the tensor-core kernel.  A thread: four columns of token blockIdx.y.
__global__ void __launch_bounds__(256) few_combine_kernel(uint16_t* __restrict__ out, const float* __restrict__ partial,
                                                          const uint16_t* __restrict__ y, const int32_t* __restrict__ counts,
                                                          const int32_t* __restrict__ entry_of, const float* __restrict__ token_w,
                                                          const float* __restrict__ h_scale, int lists, int ctas, int units, int PT, int H, int G) {
    __shared__ ListSplit sp;
    grid_launch_dependents();
    grid_dependency_wait();
    if (threadIdx.x < 32) sp.make(counts, lists, (uint32_t)(units * PT), ctas);
    __syncthreads();
    const int t = blockIdx.y, c = 4 * (blockIdx.x * 256 + threadIdx.x);
    if (c >= H) return;
    float v[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int entry = __ldcg(entry_of + 2 * t + j), e = sp.list_of(entry);
        if (sp.n[e] <= FEW_ROWS) {
            const float w = __ldcg(token_w + entry), up = __ldcg(h_scale + entry);
            const float4 s = sum_pieces(sp, partial, e, entry - sp.list0[e], c % G / PER / CW, PT, c, H);
            v[j][0] = round_bf16(round_bf16(s.x * up) * w);
            v[j][1] = round_bf16(round_bf16(s.y * up) * w);
            v[j][2] = round_bf16(round_bf16(s.z * up) * w);
            v[j][3] = round_bf16(round_bf16(s.w * up) * w);
        } else {
            const uint2 r = *reinterpret_cast<const uint2*>(y + (size_t)entry * H + c);
            v[j][0] = __uint_as_float(r.x << 16);
            v[j][1] = __uint_as_float(r.x & 0xffff0000u);
            v[j][2] = __uint_as_float(r.y << 16);
            v[j][3] = __uint_as_float(r.y & 0xffff0000u);
        }
    }
    auto two = [&](int i) {
        return (uint32_t)float_to_bf16_bits(v[0][i] + v[1][i]) | ((uint32_t)float_to_bf16_bits(v[0][i + 1] + v[1][i + 1]) << 16);
    };
    *reinterpret_cast<uint2*>(out + (size_t)t * H + c) = make_uint2(two(0), two(2));
}

static int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}
static size_t lists_smem(int period, int stages) { return 1024 + (size_t)stages * (meta_end(period) + FEW_ROWS * KC * 2) + (size_t)CW * EXCH_BYTES; }
static int lists_stages(int period) {
    for (int s = MAX_STAGES; s >= 2; --s)
        if (lists_smem(period, s) <= 224 * 1024) return s;
    return 0;
}
// Bytes of the partial row-sets of a launch, whatever the lists' lengths: A short lists have at most min(8 A, 2 T) rows, and a unit
// at most as many pieces as the smallest share of A lists makes.
static size_t partial_bytes(int64_t T, int E, int64_t units, int64_t PT, int64_t cols, int sms) {
    int64_t most = 0;
    for (int64_t A = 1; A <= E; ++A) {
        const int64_t cost = A * units * PT * COST_4, grid = std::max<int64_t>(1, std::min<int64_t>(sms, cost / COST_8));
        const int64_t share = std::max<int64_t>(1, cost / grid), pieces = (PT * COST_8 + share - 1) / share + 1;
        most = std::max(most, std::min<int64_t>(FEW_ROWS * A, 2 * T) * pieces);
    }
    return (size_t)(most * cols) * sizeof(float);
}

}  // namespace rows

bool few_plan(int64_t T, int E, const hqm_weight* w1, const hqm_weight* w2, const hqm_weight* w3, FewPlan* fp) {
    using namespace rows;
    if (T < 1 || E < 2 || !few_tokens_ok(T, E) || E > FEW_MAX_LISTS || force_generic() || tma_encode_entry() == nullptr) return false;
    const hqm_weight* ws[3] = {w1, w3, w2};
    for (const hqm_weight* w : ws) {
        int G, C;
        if (check_weight(w, &G, &C) != HQM_OK || !gemv_rows_shape_ok(w, G, C) || w->N % 4 != 0) return false;
        if (period_of(w->K, C) == 0 || lists_stages(period_of(w->K, C)) == 0) return false;
        if ((int64_t)((G / PER + CW - 1) / CW) * (w->K / KC) * 2 * E * COST_8 >= ((int64_t)1 << 31)) return false;
    }
    if (w1->N != w3->N || w1->K != w3->K || w1->meta_group != w3->meta_group || w2->K != w1->N || w2->N != w1->K) return false;
    const int sms = sm_count();
    const size_t staged_rows = (size_t)std::min<int64_t>(8 * E, 8 * T);              // (a list of one row takes four)
    const int64_t u1 = (w1->N / 16 / PER + CW - 1) / CW, u2 = (w2->N / 16 / PER + CW - 1) / CW;
    auto align = [](size_t v) { return (v + 1023) / 1024 * 1024; };
    fp->x_bytes = align(staged_rows * w1->K * 2);
    fp->scale_bytes = align((size_t)8 * T * sizeof(float));                          // factors of x and of h, GgFew::largest
    fp->h_bytes = align(staged_rows * w1->N * 2);
    fp->part_bytes = align(std::max(partial_bytes(T, E, 2 * u1, w1->K / KC, 2 * (int64_t)w1->N, sms), partial_bytes(T, E, u2, w2->K / KC, w2->N, sms)));
    return true;
}

int launch_few_projection(const FewJob& job, const unsigned char* xt, float* partial, uint32_t* largest, cudaStream_t st) {
    const bool up = largest != nullptr;
    using namespace rows;
    const hqm_weight* w = up ? job.w1 : job.w2;
    ListParams p{};
    int C;
    const int rc = check_weight(w, &p.G, &C);
    if (rc != HQM_OK) return rc;
    p.table = job.table;
    p.counts = job.counts;
    p.lists = job.lists;
    p.layers = up ? 2 : 1;
    p.which0 = up ? 0 : 1;
    p.which1 = up ? 2 : 1;
    p.K = w->K;
    p.PT = w->K / KC;
    p.N = w->N;
    p.C = C;
    p.units = (p.G / PER + CW - 1) / CW;
    p.period = period_of(w->K, C);
    p.stages = lists_stages(p.period);
    p.x_off = meta_end(p.period);
    p.stage_bytes = p.x_off + FEW_ROWS * KC * 2;
    p.xt = xt;
    p.partial = partial;
    p.largest = largest;
    p.error_flag = tc_error_ptr();
    static bool done[MAX_DEVICES];
    bool& d = done[current_device_slot()];
    if (!d) {
        HQM_CUDA(cudaFuncSetAttribute(gemv_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
        d = true;
    }
    launch_overlapped(gemv_lists_kernel, sm_count(), THREADS, lists_smem(p.period, p.stages), st, p);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

int launch_few_silu(const FewJob& job, unsigned char* ht, const float* partial, const float* row_scale, const uint32_t* largest, float* h_scale,
                    int64_t T, cudaStream_t st) {
    using namespace rows;
    const int F = job.w1->N, G = F / 16, units = (G / PER + CW - 1) / CW;
    launch_overlapped(few_silu_kernel, dim3((F / 4 + 255) / 256, (unsigned)(2 * T)), 256, 0, st, ht, partial, job.counts, row_scale, largest, h_scale,
                      job.lists, sm_count(), units, job.w1->K / KC, F, G);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

int launch_few_combine(const FewJob& job, uint16_t* out, const float* partial, const uint16_t* y, const int32_t* entry_of, const float* token_w,
                       const float* h_scale, int64_t T, cudaStream_t st) {
    using namespace rows;
    const int H = job.w2->N, G = H / 16, units = (G / PER + CW - 1) / CW;
    launch_overlapped(few_combine_kernel, dim3((H / 4 + 255) / 256, (unsigned)T), 256, 0, st, out, partial, y, job.counts, entry_of, token_w,
                      h_scale, job.lists, sm_count(), units, job.w2->K / KC, H, G);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

}  // namespace hqm
