// Quantized linear of 2-bit layers with groups of 16 for up to 8 rows of x: the experts of a decode step, of a small batch
// and of short row lists.  Replaces triton_matmul2_transpose of the reference (triton_kernels.py:321-380) and the two
// Quantizer.dequantize launches in front of it (custom_layers.py:62-66) there.
//
// Algebra.  With r = n % G the residue of output row n and j = n / G its position inside the quantisation group,
//     y[m, jG + r] = sum_k (x[m,k] s[r,k]) q[jG + r, k]  -  sum_k (x[m,k] s[r,k]) z[r,k]:
// scale and zero are decoded once per (r, k), the scale is folded into the activation, and of the weights only the bit
// fields are left.  mma.sync.m16n8k16 adds over k: its 16 rows are the 16 members of a group, its columns tokens.
//
// What bounds such a kernel is the number of instructions it issues per weight: at the HBM rate an SM receives 3 KB (8192
// codes with their scales and zeros) every 130 cycles, that is 520 issue slots.  Hence
//   * whole tiles by TMA, no copy instructions in the computing warps: a stage is 16 members x 16 storage-row residues x 128
//     columns of codes (32 KB) and the scale and zero bytes of the 64 residues (16 KB), three tiled copies by one warp; 16
//     computing warps take a storage-row residue each.
//   * a field is read where it stands: code << p in the low bits of a half IS the fp16 denormal code * 2^(p - 24), which the
//     tensor core multiplies exactly, so a pair of weights costs one AND (and a quarter of a shift); the slot's power of two is
//     taken out of the sums at the end.  No offsets, nothing to correct for.
//   * pairs are the columns (k, k+2) and (k+1, k+3) of a word, which need no byte permutation; x is staged in that order and
//     the scales are brought into it, 16 weights at a time.
//   * the fp16 values that decode scales and zeros repeat with the residue (7 different rows of them for 4096 -> 14336, one for
//     14336 -> 4096): the copying warp brings the rows of a step's columns into the stage once for 16 warps.  Read by every warp
//     for itself they are 4 KB for 3 KB of weights (out of L2), or take half of the time of a step (out of L1, 16 lines to a load).
//   * the sum of z: MMAs whose A are the scaled activations, in the registers in which they are B of the weights' MMAs, and whose B
//     are the zeros; from five rows on as fp16 and what is left of them beside it, so that z enters with 22 bits.
//
// Split: units of (16 residues, all of K) follow each other, layer after layer; a CTA (one per SM) takes an equal contiguous
// share of their 128-column steps and leaves one fp32 partial row-set per unit it touched, as the streaming kernel's warps do
// (stream_split.cuh); the consumers add them in order.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "stream_split.cuh"

namespace hqm {

namespace rows {

constexpr int CW = 16;                                  // computing warps: storage-row residues of a unit
constexpr int THREADS = (CW + 1) * 32;                  // and the copying warp
constexpr int KC = 128;                                 // columns of a step
constexpr int MEMBERS = 16, PER = 4;                    // members of a group; residues in a byte
constexpr int CODE_BYTES = CW * MEMBERS * KC, SZ_BYTES = CW * PER * KC;
constexpr int META_OFF = CODE_BYTES + 2 * SZ_BYTES;     // of a stage: tiles, then 4 x `period` rows of 128 fp16 values
constexpr int META_ROW = KC * 2 + 64;                   // (padded: the rows of neighbouring residues fall into different banks)
constexpr int MAX_PERIOD = 8;
constexpr int MAX_STAGES = 4;
constexpr int EXCH_BYTES = 4 * 128 + 8 * 128;           // of a warp: scales of 4 slots, zeros (8 rows)
constexpr uint32_t WAIT_POLLS = 1u << 18;

struct LayerParams {
    const uint16_t* meta[4];                            // ms_scale, mz_scale, ms_zero, mz_zero
    CUtensorMap maps[3];
};
struct Params {
    LayerParams ly[STREAM_MAX_LAYERS];
    int count, K, PT, stages, stage_bytes;
    int period;                                         // residues until the fp16 values of scales and zeros repeat
    int unit0[STREAM_MAX_LAYERS + 1], col0[STREAM_MAX_LAYERS + 1];
    int G[STREAM_MAX_LAYERS], C[STREAM_MAX_LAYERS], xrow[STREAM_MAX_LAYERS];
    const StreamEntry* table;
    const int32_t* sel[STREAM_MAX_LAYERS];
    int which[STREAM_MAX_LAYERS];
    int sel_settled, experts;
    int M;
    int* error_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    v = *reinterpret_cast<const uint4*>(__cvta_shared_to_generic(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    v = *reinterpret_cast<const uint2*>(__cvta_shared_to_generic(a));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint32_t perm(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t h2_of(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// half `hi` of a times the same of b, plus c in fp32
__device__ __forceinline__ float fma_half(uint32_t a, uint32_t b, float c, int hi) {
    float d;
    if (hi) asm("{\n\t.reg .b16 l, x, y;\n\tmov.b32 {l, x}, %1;\n\tmov.b32 {l, y}, %2;\n\tfma.rn.f32.f16 %0, x, y, %3;\n\t}" : "=f"(d) : "r"(a), "r"(b), "f"(c));
    else asm("{\n\t.reg .b16 h, x, y;\n\tmov.b32 {x, h}, %1;\n\tmov.b32 {y, h}, %2;\n\tfma.rn.f32.f16 %0, x, y, %3;\n\t}" : "=f"(d) : "r"(a), "r"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < WAIT_POLLS; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// Eight neighbouring bf16 of a row of x, times f, -> fp16, in their order or as (0, 2), (1, 3), (4, 6), (5, 7).
template <bool PAIRED>
__device__ __forceinline__ uint4 stage8(uint4 v, float f) {
    auto lo = [f](uint32_t a) { return __uint_as_float(a << 16) * f; };
    auto hi = [f](uint32_t a) { return __uint_as_float(a & 0xffff0000u) * f; };
    if (!PAIRED) return make_uint4(h2_of(lo(v.x), hi(v.x)), h2_of(lo(v.y), hi(v.y)), h2_of(lo(v.z), hi(v.z)), h2_of(lo(v.w), hi(v.w)));
    return make_uint4(h2_of(lo(v.x), lo(v.y)), h2_of(hi(v.x), hi(v.y)), h2_of(lo(v.z), lo(v.w)), h2_of(hi(v.z), hi(v.w)));
}

// TOKS: rows of x computed together.  1: the four slots of a byte are B columns 0-3.  4: a B fragment holds two slots of four
// rows; 8: one slot of eight.
template <int TOKS>
struct Shape {
    static constexpr int SPB = TOKS == 4 ? 2 : 1;                   // slots in a B fragment (TOKS > 1)
    static constexpr int PAIRS = TOKS == 4 ? 1 : 2;                 // pairs of B fragments
    static constexpr bool FINE_Z = TOKS > 4;                        // zeros with 22 bits (up to 4 rows 11, as the streaming kernels)
    // Rows with a power of two each, that their largest value of this CTA's columns lies in [16, 32): any bf16 row then fits fp16
    // (as in the tensor-core kernel, which took these row counts before; up to 4 rows as the streaming kernels, |x| < 65504).
    static constexpr bool SCALED = TOKS > 4;
    static constexpr int X_STEP = TOKS * KC * 2;                    // staged bytes of x per step
};

template <int TOKS>
__global__ void __launch_bounds__(THREADS, 1)
gemv_rows_kernel(float* __restrict__ partial, const uint16_t* __restrict__ x, const int32_t* __restrict__ x_idx, int M_total,
                 const __grid_constant__ Params prm, Split sp) {
    using S = Shape<TOKS>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ int s_absent[STREAM_MAX_LAYERS];
    __shared__ int s_failed;
    __shared__ uint32_t s_max[8];                       // largest |x| of a row's columns, as bf16
    __shared__ __align__(8) uint64_t s_bars[2 * MAX_STAGES];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int stages = prm.stages, stage_bytes = prm.stage_bytes, period = prm.period;
    const uint32_t exch = ring + stages * prm.stage_bytes;                            // (of TOKS > 1) a corner per warp
    const uint32_t x_area = exch + (TOKS > 1 ? CW * EXCH_BYTES : 0);
    const uint32_t full = smem_u32(s_bars), empty = full + 8 * MAX_STAGES;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int K = prm.K, PT = prm.PT;

    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(full + 8 * i));      // the tiles, and 32 lanes' copies
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8 * i), "n"(CW));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        s_failed = 0;
    }
    if (threadIdx.x < 8) s_max[threadIdx.x] = 0u;
    __syncthreads();
    // this CTA's steps: from step pa0 of unit0 on; how many CTAs hold a piece of that unit in front of this one
    const uint32_t L0 = sp.begin(blockIdx.x), L1 = sp.begin(blockIdx.x + 1);
    const int unit0 = (int)(L0 / (uint32_t)PT), pa0 = (int)(L0 - (uint32_t)unit0 * (uint32_t)PT), n_steps = (int)(L1 - L0);
    const int slot0 = (int)blockIdx.x - sp.owner((uint32_t)unit0 * (uint32_t)PT);
    auto layer_of = [&](int unit) {
        int l = 0;
#pragma unroll
        for (int i = 1; i < STREAM_MAX_LAYERS; ++i) l += (i < prm.count && unit >= prm.unit0[i]) ? 1 : 0;
        return l;
    };

    auto row_exponent = [&](int m) { return min(max((int)(s_max[m] >> 7), 30), 250) - 4; };     // of the factor, biased

    if (warp == CW) {
        // =========================== copies ===========================
        // (the weights are never written by a kernel of the chain: unless the experts are chosen by a kernel in front, the copies
        // start while that kernel is still running)
        // A step's fp16 values: rows (array, class) of 16 pieces of 16 bytes; this lane copies piece lane % 16 of the arrays
        // lane / 16 and 2 + lane / 16.  Piece 4 t + 2 u + h is put where (u, h, t) says.
        const int c16 = lane & 15, hi = lane >> 4;
        const uint32_t C0 = (uint32_t)prm.C[0], pa_col = (uint32_t)pa0 * KC % C0, k_col = (uint32_t)K % C0;
        uint32_t elected;
        asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(elected));
        int idx = 0;
        if (prm.table) {
            if (!prm.sel_settled) {
                // the entries of all experts in L2 by the time the choice is known
                const int last = layer_of(unit0 + (pa0 + n_steps - 1) / PT);
                for (int l = layer_of(unit0); l <= last; ++l)
                    for (int i = lane; i < 4 * prm.experts; i += 32) {
                        const StreamEntry* en = prm.table + 3 * (i >> 2) + prm.which[l];
                        prefetch_l2((i & 3) == 0 ? reinterpret_cast<const void*>(&en->w) : en->rows_maps[(i & 3) - 1]);
                    }
                grid_dependency_wait();
            }
            if (lane < prm.count) idx = __ldcg(prm.sel[lane]);
            // the chosen experts' other entries, for the launches that follow
            if (blockIdx.x == gridDim.x - 1 && !prm.sel_settled && lane < prm.count && idx >= 0)
                for (int i = 0; i < 3 * (int)sizeof(StreamEntry); i += 128)
                    prefetch_l2(reinterpret_cast<const unsigned char*>(prm.table + 3 * idx) + i);
        }
        int st = 0, fenced = -1;
        uint32_t par = 1;
        bool ok = true;
        for (int unit = unit0, pa = pa0, left = n_steps; left > 0 && ok; ++unit, pa = 0) {
            const int pb = min(PT, pa + left);
            left -= pb - pa;
            const int l = layer_of(unit);
            const int e = __shfl_sync(0xffffffffu, idx, l);
            if (e < 0) continue;
            const CUtensorMap* maps = prm.ly[l].maps;
            const uint16_t *src0 = prm.ly[l].meta[hi], *src1 = prm.ly[l].meta[2 + hi];
            if (prm.table) {
                const StreamEntry* en = prm.table + 3 * e + prm.which[l];
                maps = reinterpret_cast<const CUtensorMap*>(en->rows_maps);
                if (fenced != l && lane < 3) prefetch_l2(maps + lane);
                src0 = hi ? en->w.mz_scale : en->w.ms_scale;
                src1 = hi ? en->w.mz_zero : en->w.ms_zero;
                if (fenced != l) {
                    fenced = l;
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(maps + i) : "memory");
                }
            }
            const int rho = (unit - prm.unit0[l]) * CW;
            src0 += 8 * c16;
            src1 += 8 * c16;
            uint32_t col = pa ? pa_col : 0u;                  // of class 0
            for (int p = pa; p < pb; ++p) {
                if (!wait(empty + 8 * st, par)) {
                    ok = false;
                    break;
                }
                const uint32_t bar = full + 8 * st, dst = ring + st * stage_bytes;
                if (elected) {
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)META_OFF) : "memory");
                    tma_3d(dst, maps, p * KC, 0, rho, bar);
                    tma_3d(dst + CODE_BYTES, maps + 1, p * KC, PER * rho, 0, bar);
                    tma_3d(dst + CODE_BYTES + SZ_BYTES, maps + 2, p * KC, PER * rho, 0, bar);
                }
                uint32_t to = dst + (uint32_t)(META_OFF + hi * period * META_ROW + (c16 & 3) * 64 + (c16 >> 2) * 16), at = col;
                for (int cls = 0; cls < period; ++cls) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src0 + at) : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 2 * period * META_ROW), "l"(src1 + at) : "memory");
                    to += META_ROW;
                    at += k_col;
                    at = at >= C0 ? at - C0 : at;
                }
                col += KC;
                col = col >= C0 ? col - C0 : col;
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
                if (++st == stages) {
                    st = 0;
                    par ^= 1;
                }
            }
        }
        // (no lane leaves with copies on their way)
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) s_failed = 1;
    } else {
        // =========================== computing warps ===========================
        const int M = prm.M;
        grid_dependency_wait();
        if (prm.table && threadIdx.x >= CW * 32 - 32 && lane < prm.count) s_absent[lane] = __ldcg(prm.sel[lane]) < 0;
        // the columns of x of this CTA's steps, as fp16: [step][half of a lane's 32 columns][16-byte piece][row][thread column]
        auto piece = [&](int i, int& c, int& m, int& step) {            // piece c of row m's columns of a step
            c = i & 15;
            m = (i >> 4) % TOKS;
            step = (i >> 4) / TOKS;
            if (TOKS != 1 && m >= M) return make_uint4(0u, 0u, 0u, 0u);
            const int du = (pa0 + step) / PT, p = pa0 + step - du * PT;
            const int64_t row = (x_idx ? x_idx[m] : m) + prm.xrow[layer_of(unit0 + du)];
            return *reinterpret_cast<const uint4*>(x + row * K + p * KC + 8 * c);
        };
        const int pieces = n_steps * TOKS * 16;
        if constexpr (S::SCALED) {
            for (int i = threadIdx.x; i < pieces; i += CW * 32) {
                int c, m, step;
                const uint4 v = piece(i, c, m, step);
                uint32_t mx = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
                mx = max(mx & 0xffffu, mx >> 16);
                if (mx) atomicMax(&s_max[m], mx);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");
        }
        for (int i = threadIdx.x; i < pieces; i += CW * 32) {
            int c, m, step;
            const uint4 raw = piece(i, c, m, step);
            const uint4 v = stage8<TOKS != 1>(raw, S::SCALED ? __uint_as_float((uint32_t)(254 - row_exponent(m)) << 23) : 1.f);
            sts128(x_area + step * S::X_STEP + ((2 * ((c >> 1) & 1) + (c & 1)) * TOKS + m) * 64 + (c >> 2) * 16, v.x, v.y, v.z, v.w);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");

        const int g = lane >> 2, t = lane & 3;
        const uint32_t code_off = (uint32_t)(warp * MEMBERS * KC + g * KC), sw = (uint32_t)g;
        uint32_t x_at = x_area;                                     // of the present step
        int st = 0;
        uint32_t par = 0;
        bool ok = true;
        for (int unit = unit0, pa = pa0, left = n_steps; left > 0 && ok; ++unit, pa = 0) {
            const int pb_all = min(PT, pa + left);
            left -= pb_all - pa;
            const int l = layer_of(unit);
            const int rho = (unit - prm.unit0[l]) * CW + warp;
            const int G = prm.G[l];
            const bool live = rho * PER < G;
            const int pb = prm.table && s_absent[l] ? pa : pb_all;
            // the residue whose scales this lane decodes, its row of bytes in a stage, and its row of fp16 values
            const int slot = TOKS == 1 ? (g & 3) : (lane >> 3);
            const int brow = warp * PER + slot;
            const uint32_t byte_off = (uint32_t)(CODE_BYTES + brow * KC);
            const uint32_t bsw = (uint32_t)(brow & 7);
            const int cls = (PER * rho + slot) % period;
            const int slot_idx = unit == unit0 ? slot0 : 0;

            if constexpr (TOKS == 1) {
                // Lanes g and g + 4 share slot g % 4: each decodes scale and zero of 16 of the 32 columns (half u = g / 4).
                const int du = g >> 2;
                const uint32_t m_step = (uint32_t)(period * META_ROW), m_off = (uint32_t)(META_OFF + cls * META_ROW + du * 128 + t * 16);
                const uint32_t c_off0 = code_off + (((2 * t) ^ sw) << 4), c_off1 = code_off + (((2 * t + 1) ^ sw) << 4);
                const uint32_t b_off = byte_off + (((2 * t + du) ^ bsw) << 4);
                uint32_t xa = x_at + du * 128 + 16 * t;
                float acc[4][4], cor = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
                // x * s of this lane's columns of the step in the stage at sb, (0, 2), (1, 3) of every word, and the zeros' sum
                auto decode = [&](uint32_t sb, uint32_t (&own)[8]) {
                    const uint4 s16 = lds128(sb + b_off), z16 = lds128(sb + b_off + SZ_BYTES);
                    const uint32_t sw4[4] = {s16.x, s16.y, s16.z, s16.w}, zw4[4] = {z16.x, z16.y, z16.z, z16.w};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t ma = sb + m_off + h * 64;
                        const uint4 m0 = lds128(ma), m1 = lds128(ma + m_step), m2 = lds128(ma + 2 * m_step), m3 = lds128(ma + 3 * m_step);
                        const uint4 xv = lds128(xa + h * 64);
                        const uint32_t mss[4] = {m0.x, m0.y, m0.z, m0.w}, mzs[4] = {m1.x, m1.y, m1.z, m1.w};
                        const uint32_t msz[4] = {m2.x, m2.y, m2.z, m2.w}, mzz[4] = {m3.x, m3.y, m3.z, m3.w};
                        const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            uint32_t v[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int i = 2 * j + e;
                                const uint32_t sel = e ? 0x4342u : 0x4140u;
                                const uint32_t sc = h2mul(h2sub(h2sub(perm(sw4[2 * h + j], 0x64646464u, sel), 0x64006400u), mzs[i]), mss[i]);
                                const uint32_t z = h2mul(h2sub(h2sub(perm(zw4[2 * h + j], 0x64646464u, sel), 0x64006400u), mzz[i]), msz[i]);
                                v[e] = h2mul(sc, xs[i]);
                                cor = fma_half(v[e], z, cor, 0);
                                cor = fma_half(v[e], z, cor, 1);
                            }
                            own[4 * h + 2 * j] = perm(v[0], v[1], 0x5410u);
                            own[4 * h + 2 * j + 1] = perm(v[0], v[1], 0x7632u);
                        }
                    }
                };
                for (int p = pa; p < pb; ++p) {
                    if (!wait(full + 8 * st, par)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sb = ring + st * stage_bytes;
                    if (live) {
                        uint32_t own[8];
                        decode(sb, own);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t ca = sb + (u ? c_off1 : c_off0);
                            const uint4 q0 = lds128(ca), q1 = lds128(ca + 8 * KC);
                            const uint32_t r0[4] = {q0.x, q0.y, q0.z, q0.w}, r1[4] = {q1.x, q1.y, q1.z, q1.w};
#pragma unroll
                            for (int wd = 0; wd < 4; ++wd) {
                                // B column g: of lanes 0-15 only; the second half's come from the lanes that decoded it
                                const uint32_t b0 = u ? __shfl_down_sync(0xffffffffu, own[2 * wd], 16) : own[2 * wd];
                                const uint32_t b1 = u ? __shfl_down_sync(0xffffffffu, own[2 * wd + 1], 16) : own[2 * wd + 1];
                                const uint32_t v0 = r0[wd] >> 8, v1 = r1[wd] >> 8;
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const uint32_t mask = 0x00030003u << (6 - 2 * i);
                                    mma(acc[i], r0[wd] & mask, r1[wd] & mask, v0 & mask, v1 & mask, b0, b1);
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * st) : "memory");
                    xa += S::X_STEP;
                    if (++st == stages) {
                        st = 0;
                        par ^= 1;
                    }
                }
                // slot s: column s of its tile, in lanes t = s / 2; its zeros' sum over the lanes g % 4 = s
                if (live && ok) {
                    cor += __shfl_xor_sync(0xffffffffu, cor, 1);
                    cor += __shfl_xor_sync(0xffffffffu, cor, 2);
                    cor += __shfl_xor_sync(0xffffffffu, cor, 16);
                    const float ca = __shfl_sync(0xffffffffu, cor, 8 * (t & 1));
                    const float cb = __shfl_sync(0xffffffffu, cor, 8 * (t & 1) + 4);
                    if (t < 2) {
                        // 2^(24 - p), p = 6 - 2 s
                        const float fa = t ? 4194304.f : 262144.f, fb = t ? 16777216.f : 1048576.f;
                        float* dst = partial + (int64_t)slot_idx * M_total * prm.col0[prm.count] + prm.col0[l] + PER * rho + 2 * t + (int64_t)g * G;
                        const float a0 = t ? acc[2][0] : acc[0][0], a8 = t ? acc[2][2] : acc[0][2];
                        const float b0 = t ? acc[3][1] : acc[1][1], b8 = t ? acc[3][3] : acc[1][3];
                        *reinterpret_cast<float2*>(dst) = make_float2(a0 * fa - ca, b0 * fb - cb);
                        *reinterpret_cast<float2*>(dst + (int64_t)8 * G) = make_float2(a8 * fa - ca, b8 * fb - cb);
                    }
                }
            } else {
                // eight columns of half u: thread column mt0, piece lane % 2
                const int mt0 = (lane & 7) >> 1;
                const uint32_t m_step = (uint32_t)(period * META_ROW), m_off = (uint32_t)(META_OFF + cls * META_ROW + (lane & 1) * 64 + mt0 * 16);
                constexpr bool FINE_Z = S::FINE_Z;
                constexpr int CORS = FINE_Z ? S::PAIRS : 2;
                float acc[4][4], cor[CORS][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int i = 0; i < CORS; ++i) cor[i][j] = 0.f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][j] = 0.f;
                }
                const uint32_t ex = exch + warp * EXCH_BYTES, ez = ex + 512;
                // the corner of shared memory: [slot][piece][thread column] scales, [row][piece][thread column] zeros (the pieces of odd rows
                // change places, so that the eight lanes of a load phase touch all banks)
                const uint32_t s_put = ex + slot * 128 + (lane & 1) * 64 + ((lane & 7) >> 1) * 16;
                const uint32_t z_put = ez + (FINE_Z ? slot * 128 + ((lane ^ slot) & 1) * 64 : slot * 64 + (lane & 1) * 8) + ((lane & 7) >> 1) * 16;
                // this lane's B column: row of x and slot inside the fragment
                const int xm = S::SPB == 2 ? (g & 3) : g;
                const uint32_t s_get = ex + (S::SPB == 2 ? (g >> 2) * 128 : 0) + t * 16, z_get = ez + (FINE_Z ? g * 128 + (g & 1) * 64 : g * 64) + t * 16;
                uint32_t xa = x_at + xm * 64 + t * 16;
                for (int p = pa; p < pb; ++p) {
                    if (!wait(full + 8 * st, par)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sb = ring + st * stage_bytes;
                    if (live) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            // ---- scale and zero of eight columns of a residue
                            const uint32_t ba = sb + byte_off + (((2 * ((lane & 7) >> 1) + u) ^ bsw) << 4) + 8 * (lane & 1);
                            const uint2 s8 = lds64(ba), z8 = lds64(ba + SZ_BYTES);
                            const uint32_t ca = sb + code_off + (((2 * t + u) ^ sw) << 4);
                            const uint4 q0 = lds128(ca), q1 = lds128(ca + 8 * KC);
                            const uint32_t ma = sb + m_off + u * 128;
                            const uint4 mt[4] = {lds128(ma), lds128(ma + m_step), lds128(ma + 2 * m_step), lds128(ma + 3 * m_step)};
                            uint32_t sc[4], zh[4], zl[4];
                            {
                                const uint32_t sq[2] = {s8.x, s8.y}, zq[2] = {z8.x, z8.y};
                                const uint32_t mss[4] = {mt[0].x, mt[0].y, mt[0].z, mt[0].w}, mzs[4] = {mt[1].x, mt[1].y, mt[1].z, mt[1].w};
                                const uint32_t msz[4] = {mt[2].x, mt[2].y, mt[2].z, mt[2].w}, mzz[4] = {mt[3].x, mt[3].y, mt[3].z, mt[3].w};
#pragma unroll
                                for (int j = 0; j < 2; ++j) {
                                    uint32_t v[2], hi[2], lo[2];
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        const int i = 2 * j + e;
                                        const uint32_t sel = e ? 0x4342u : 0x4140u;
                                        v[e] = h2mul(h2sub(h2sub(perm(sq[j], 0x64646464u, sel), 0x64006400u), mzs[i]), mss[i]);
                                        // (byte - zero) * scale: the rounded difference d and what it leaves, and the same of the product
                                        const uint32_t zb = h2sub(perm(zq[j], 0x64646464u, sel), 0x64006400u);
                                        const uint32_t d = h2sub(zb, mzz[i]);
                                        hi[e] = h2mul(d, msz[i]);
                                        if constexpr (FINE_Z) {
                                            const uint32_t rest = h2sub(h2sub(zb, d), mzz[i]);
                                            lo[e] = h2fma(rest, msz[i], h2fma(d, msz[i], hi[e] ^ 0x80008000u));
                                        }
                                    }
                                    sc[2 * j] = perm(v[0], v[1], 0x5410u);
                                    sc[2 * j + 1] = perm(v[0], v[1], 0x7632u);
                                    zh[2 * j] = perm(hi[0], hi[1], 0x5410u);
                                    zh[2 * j + 1] = perm(hi[0], hi[1], 0x7632u);
                                    if constexpr (FINE_Z) {
                                        zl[2 * j] = perm(lo[0], lo[1], 0x5410u);
                                        zl[2 * j + 1] = perm(lo[0], lo[1], 0x7632u);
                                    }
                                }
                            }
                            sts128(s_put, sc[0], sc[1], sc[2], sc[3]);
                            if constexpr (FINE_Z) {
                                sts128(z_put, zh[0], zh[1], zh[2], zh[3]);
                                sts128(z_put + 4 * 128, zl[0], zl[1], zl[2], zl[3]);
                            } else {                            // rows 0-3: even registers, 4-7: odd ones
                                sts64(z_put, zh[0], zh[2]);
                                sts64(z_put + 4 * 64, zh[1], zh[3]);
                            }
                            __syncwarp();
                            // ---- products
                            uint32_t zf[FINE_Z ? 8 : 4];
                            {
                                const uint4 za = lds128(z_get);
                                zf[0] = za.x; zf[1] = za.y; zf[2] = za.z; zf[3] = za.w;
                                if constexpr (FINE_Z) {
                                    const uint4 zc = lds128(z_get ^ 64u);
                                    zf[4] = zc.x; zf[5] = zc.y; zf[6] = zc.z; zf[7] = zc.w;
                                }
                            }
                            const uint32_t r0[4] = {q0.x, q0.y, q0.z, q0.w}, r1[4] = {q1.x, q1.y, q1.z, q1.w};
                            const uint4 xlo = lds128(xa + 2 * u * TOKS * 64), xhi = lds128(xa + (2 * u + 1) * TOKS * 64);
                            const uint32_t xf[8] = {xlo.x, xlo.y, xlo.z, xlo.w, xhi.x, xhi.y, xhi.z, xhi.w};
#pragma unroll
                            for (int pr = 0; pr < S::PAIRS; ++pr) {
                                uint32_t bf[2][8];
#pragma unroll
                                for (int f = 0; f < 2; ++f) {
                                    const uint32_t at = s_get + (2 * pr + f) * S::SPB * 128;
                                    const uint4 a = lds128(at), b = lds128(at + 64);
                                    const uint32_t sv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                                    for (int i = 0; i < 8; ++i) bf[f][i] = h2mul(xf[i], sv[i]);
                                }
                                if constexpr (!FINE_Z) {
                                    // rows g: the even registers against columns 0-3, rows 8 + g: the odd ones against columns 4-7
#pragma unroll
                                    for (int f = 0; f < 2; ++f)
#pragma unroll
                                        for (int h = 0; h < 2; ++h)
                                            mma(cor[f], bf[f][4 * h], bf[f][4 * h + 1], bf[f][4 * h + 2], bf[f][4 * h + 3], zf[2 * h], zf[2 * h + 1]);
                                } else
#pragma unroll
                                for (int wd = 0; wd < 4; ++wd)
                                    mma(cor[pr], bf[0][2 * wd], bf[1][2 * wd], bf[0][2 * wd + 1], bf[1][2 * wd + 1], zf[(2 * wd) % (FINE_Z ? 8 : 4)], zf[(2 * wd + 1) % (FINE_Z ? 8 : 4)]);
#pragma unroll
                                for (int wd = 0; wd < 4; ++wd) {
                                    const uint32_t v0 = r0[wd] >> 8, v1 = r1[wd] >> 8;
                                    constexpr int SLOTS = 4 / S::PAIRS;      // slots of the pair
#pragma unroll
                                    for (int i = 0; i < SLOTS; ++i) {
                                        const int s = pr * SLOTS + i;
                                        const uint32_t mask = 0x00030003u << (6 - 2 * s);
                                        mma(acc[s], r0[wd] & mask, r1[wd] & mask, v0 & mask, v1 & mask, bf[i / S::SPB][2 * wd], bf[i / S::SPB][2 * wd + 1]);
                                    }
                                }
                            }
                            __syncwarp();                       // the corner is written again
                        }
                    } else {
                        __syncwarp();
                    }
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * st) : "memory");
                    xa += S::X_STEP;
                    if (++st == stages) {
                        st = 0;
                        par ^= 1;
                    }
                }
                if (live && ok) {
                    // zeros' sums: row (row of x or slot of the pair's half), column slot and slot + 4: in lane t = slot / 2 and t + 2
#pragma unroll
                    for (int i = 0; i < CORS; ++i) {
                        if constexpr (FINE_Z) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) cor[i][j] += __shfl_xor_sync(0xffffffffu, cor[i][j], 2);
                        } else {                                // fragment i, row g: slot 2 i + g / 4
                            const float v = t < 2 ? (g < 4 ? cor[i][0] : cor[i][1]) : (g < 4 ? cor[i][2] : cor[i][3]);
                            cor[i][0] = v + __shfl_xor_sync(0xffffffffu, v, 2);
                        }
                    }
                    // the accumulators hold columns 2t and 2t + 1: rows of x (TOKS 4: of one slot of the fragment's two)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int m = TOKS == 4 ? ((2 * t + e) & 3) : 2 * t + e;
                        float z[4];
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            const float v = TOKS == 4 ? cor[s >> 1][0] : cor[s >> 1][3 * (s & 1)];
                            z[s] = __shfl_sync(0xffffffffu, v, (TOKS == 4 ? ((s & 1) * 4 + m) * 4 : m * 4) + (s >> 1));
                        }
                        if (m < M) {
                            const float up = S::SCALED ? __uint_as_float((uint32_t)row_exponent(m) << 23) : 1.f;
                            float* dst = partial + ((int64_t)slot_idx * M_total + m) * prm.col0[prm.count] + prm.col0[l] + PER * rho + (int64_t)g * G;
#pragma unroll
                            for (int half = 0; half < 2; ++half) {
                                float y[4];
#pragma unroll
                                for (int s = 0; s < 4; ++s) y[s] = (acc[s][2 * half + e] * (float)(1 << (18 + 2 * s)) - z[s]) * up;
                                float* at = dst + (int64_t)8 * half * G;
                                if constexpr (TOKS == 4) {          // lanes t < 2 hold slots 0 and 2, the others 1 and 3
                                    at[t >> 1] = t < 2 ? y[0] : y[1];
                                    at[2 + (t >> 1)] = t < 2 ? y[2] : y[3];
                                } else {
                                    *reinterpret_cast<float4*>(at) = make_float4(y[0], y[1], y[2], y[3]);
                                }
                            }
                        }
                    }
                }
            }
            x_at += (uint32_t)(pb_all - pa) * S::X_STEP;
        }
        if (!ok) s_failed = 1;
    }
    // ---- a wait ran out: copies may still be on their way to this CTA's shared memory
    __syncthreads();
    if (s_failed) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        if (threadIdx.x == 0 && prm.error_flag) atomicExch(prm.error_flag, 1);
    }
}

static int stage_bytes(int period) { return META_OFF + (4 * period * META_ROW + 1023) / 1024 * 1024; }
static size_t smem_bytes(int toks, int stages, int period, int steps) {
    return 1024 + (size_t)stages * stage_bytes(period) + (toks > 1 ? (size_t)CW * EXCH_BYTES : 0) + (size_t)steps * toks * KC * 2;
}
static int toks_for(int64_t M) { return M <= 1 ? 1 : (M <= 4 ? 4 : 8); }
static int stages_for(int toks, int period, int steps) {
    for (int s = MAX_STAGES; s >= 2; --s)
        if (smem_bytes(toks, s, period, steps) <= 226 * 1024) return s;
    return 0;
}

// Residues until (residue * K) mod C repeats; 0: more than a stage has room for.
static int period_of(int K, int C) {
    for (int p = 1; p <= MAX_PERIOD; ++p)
        if ((int64_t)p * K % C == 0) return p;
    return 0;
}

template <int TOKS>
static bool prepare(size_t smem) {
    static size_t configured[MAX_DEVICES];
    size_t& have = configured[current_device_slot()];
    if (have >= smem) return true;
    if (cudaFuncSetAttribute(gemv_rows_kernel<TOKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    have = smem;
    return true;
}

}  // namespace rows

bool gemv_rows_plan(const hqm_weight* const* ws, int count, int64_t M, StreamPlan* plan) {
    using namespace rows;
    if (count < 1 || count > STREAM_MAX_LAYERS || M < 1 || M > STREAM_ROWS_MAX || tma_encode_entry() == nullptr) return false;
    const hqm_weight* w = ws[0];
    plan->count = count;
    plan->rho0[0] = 0;
    plan->col0[0] = 0;
    for (int l = 0; l < count; ++l) {
        const hqm_weight* v = ws[l];
        int G, C;
        if (check_weight(v, &G, &C) != HQM_OK || !gemv_rows_shape_ok(v, G, C) || v->K != w->K) return false;
        if (period_of(v->K, C) == 0 || (l > 0 && C != plan->C[0])) return false;
        plan->G[l] = G;
        plan->C[l] = C;
        plan->rho0[l + 1] = plan->rho0[l] + (G / PER + CW - 1) / CW;
        plan->col0[l + 1] = plan->col0[l] + v->N;
    }
    plan->nbits = 2;
    plan->nb = 1;
    plan->PT = w->K / KC;
    const int64_t total = (int64_t)plan->rho0[count] * plan->PT;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t grid = std::min<int64_t>(total, sms);
    if (total * grid >= ((int64_t)1 << 31)) return false;
    const int steps = (int)((total + grid - 1) / grid);
    plan->toks = toks_for(M);
    if (stages_for(plan->toks, period_of(w->K, plan->C[0]), steps) == 0) return false;
    plan->grid = plan->warps = (int)grid;
    plan->slots = (int)((plan->PT + total / grid - 1) / (total / grid)) + 1;
    plan->kind = STREAM_ROWS;
    return true;
}

int launch_gemv_rows(float* partial, const uint16_t* x, const int32_t* x_idx, int64_t M, const StreamJob& job, const StreamPlan& plan,
                     cudaStream_t st) {
    using namespace rows;
    Params prm{};
    prm.count = plan.count;
    prm.K = job.w[0]->K;
    prm.PT = plan.PT;
    for (int l = 0; l < plan.count; ++l) {
        const hqm_weight* w = job.w[l];
        prm.unit0[l] = plan.rho0[l];
        prm.col0[l] = plan.col0[l];
        prm.G[l] = plan.G[l];
        prm.C[l] = plan.C[l];
        prm.xrow[l] = job.xrow[l];
        prm.sel[l] = job.sel[l];
        prm.which[l] = job.which[l];
        if (!job.table) {
            prm.ly[l].meta[0] = w->ms_scale;
            prm.ly[l].meta[1] = w->mz_scale;
            prm.ly[l].meta[2] = w->ms_zero;
            prm.ly[l].meta[3] = w->mz_zero;
            if (!rows_cached_maps(w, plan.G[l], prm.ly[l].maps)) {
                set_error("gemv_rows: cuTensorMapEncodeTiled failed for a %dx%d layer", w->N, w->K);
                return HQM_ERR_CUDA;
            }
        }
    }
    prm.unit0[plan.count] = plan.rho0[plan.count];
    prm.col0[plan.count] = plan.col0[plan.count];
    prm.table = job.table;
    prm.sel_settled = job.sel_settled;
    prm.experts = job.experts;
    prm.M = (int)M;
    prm.error_flag = tc_error_ptr();
    const Split sp = work_split_of(plan);
    const int steps = (int)((sp.total() + plan.grid - 1) / plan.grid);
    prm.period = period_of(prm.K, plan.C[0]);
    prm.stage_bytes = stage_bytes(prm.period);
    prm.stages = stages_for(plan.toks, prm.period, steps);
    const size_t smem = smem_bytes(plan.toks, prm.stages, prm.period, steps);
#define HQM_ROWS(T) \
    if (plan.toks == T) { \
        if (!prepare<T>(smem)) { \
            set_error("gemv_rows: cannot configure %zu bytes of shared memory", smem); \
            return HQM_ERR_CUDA; \
        } \
        launch_overlapped(gemv_rows_kernel<T>, plan.grid, THREADS, smem, st, partial, x, x_idx, (int)M, prm, sp); \
        HQM_LAUNCH_CHECK(); \
        return HQM_OK; \
    }
    HQM_ROWS(1) HQM_ROWS(4) HQM_ROWS(8)
#undef HQM_ROWS
    set_error("gemv_rows: no kernel for %d rows", plan.toks);
    return HQM_ERR_ARG;
}

}  // namespace hqm
