// Shared by the kernels for few rows of x (gemv_rows.cu, gemv_lists.cu): a stage of shared memory and its copies, and the
// arithmetic of a run of steps.  What bounds it and why it is built so stands in gemv_rows.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "kernels.cuh"

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
// Bounded wait.  (The lanes of a warp poll together.  A vote on the outcome costs 1.5 % of an expert's time at one row.)
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

// Of a row's factor, biased, from the row's largest |x| as bf16: the factor brings it into [16, 32).
__device__ __forceinline__ int exponent_of(uint32_t largest) { return min(max((int)(largest >> 7), 30), 250) - 4; }

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

// What a computing warp needs to know of a run of steps of one unit.
struct Segment {
    uint32_t ring, full, empty, corner;        // shared memory: stages, barriers, this warp's corner
    int stage_bytes, stages, period;
    int cls;                                   // row of fp16 values of the residue whose scales this lane decodes
    int M, G, row_len;                         // rows of x; residues of the layer; columns of a partial row
    bool live;                                 // the warp has a storage-row residue
};

// A layer as it lies in memory, a run of steps of one unit, and the rows of x: what sum_again() reads.
struct Again {
    const uint8_t *codes, *scale_q, *zero_q;
    const uint16_t *ms_scale, *mz_scale, *ms_zero, *mz_zero;
    int K, G, C, rho, k0, k1;                  // the warp's storage-row residue; columns of the run
    const uint16_t* x;                         // a bf16 row, multiplied with `down` ...
    float down;
    const unsigned char* staged;               // ... or (not null) row m of a staged list of `cap` rows
    int m, cap;
    __device__ __forceinline__ void layer(const hqm_weight& w) {
        codes = static_cast<const uint8_t*>(w.W_q);
        scale_q = w.scale_q;
        zero_q = w.zero_q;
        ms_scale = w.ms_scale;
        mz_scale = w.mz_scale;
        ms_zero = w.ms_zero;
        mz_zero = w.mz_zero;
    }
};
// One row's sums over a run of steps once more, with the weights that dequantize() makes and fp32 products, where a sum that
// rows_segment() left at `to` (16 members, G apart, of 4 residues) is not finite.  With the tensor cores' factors that happens for
// inputs that are fine: x * s leaves fp16 where a scale is 2048 or more (x is staged below 32), and an infinite x meets codes of 0
// and makes the zeros' sum a difference of infinities, though its products with the weights have a sign.  The warps come
// here behind all of their steps, when one has seen such a sum: beside them the call would cost the steps 60 to 190 bytes of spilled
// registers.  Returns the largest finite |sum| it formed, 0 where all were finite as they were.
__device__ __noinline__ static float sum_again(const Again& a, float* to, float up) {
    const int lane = threadIdx.x & 31;
    __syncwarp();                                  // other lanes have stored some of the sums
    const float2 have = *reinterpret_cast<const float2*>(to + (int64_t)(lane >> 1) * a.G + 2 * (lane & 1));
    if (__all_sync(0xffffffffu, isfinite(have.x) && isfinite(have.y))) return 0.f;
    float largest = 0.f;
    for (int s = 0; s < PER; ++s) {
        float sum[MEMBERS];
#pragma unroll
        for (int j = 0; j < MEMBERS; ++j) sum[j] = 0.f;
        for (int k = a.k0 + 4 * lane; k < a.k1; k += 128) {
            const uint8_t* codes = a.codes + (int64_t)a.rho * a.K + k;
            uint32_t q[MEMBERS];
#pragma unroll
            for (int j = 0; j < MEMBERS; ++j) q[j] = *reinterpret_cast<const uint32_t*>(codes + (int64_t)j * (a.G / PER) * a.K) >> (6 - 2 * s);
            const int64_t at = (int64_t)(PER * a.rho + s) * a.K + k;
            const uint32_t sq = *reinterpret_cast<const uint32_t*>(a.scale_q + at), zq = *reinterpret_cast<const uint32_t*>(a.zero_q + at);
            const int col = (int)(at % a.C);
            float x[4];
            if (a.staged) {
                const uint2 v = *reinterpret_cast<const uint2*>(a.staged + few_staged_at(k & ~7, a.m, a.cap) + (k & 4) * 2);
                const uint32_t w[2] = {v.x, v.y};                                 // columns (0, 2), (1, 3)
#pragma unroll
                for (int c = 0; c < 4; ++c) x[c] = f16_bits_to_float((uint16_t)(w[c & 1] >> (8 * (c & 2))));
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) x[c] = bf16_bits_to_float(a.x[k + c]) * a.down;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float scale = __fmul_rn(__fsub_rn((float)((sq >> (8 * c)) & 255u), f16_bits_to_float(a.mz_scale[col + c])), f16_bits_to_float(a.ms_scale[col + c]));
                const float zero = __fmul_rn(__fsub_rn((float)((zq >> (8 * c)) & 255u), f16_bits_to_float(a.mz_zero[col + c])), f16_bits_to_float(a.ms_zero[col + c]));
#pragma unroll
                for (int j = 0; j < MEMBERS; ++j) sum[j] = fmaf(x[c], __fmul_rn(__fsub_rn((float)((q[j] >> (8 * c)) & 3u), zero), scale), sum[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < MEMBERS; ++j) {
            const float v = warp_sum(sum[j]) * up;
            if (lane == 0) to[(int64_t)j * a.G + s] = v;
            if (isfinite(v)) largest = fmaxf(largest, fabsf(v));
        }
    }
    return largest;
}

// TOKS > 1 rows over `steps` steps, from stage st (phase par) on.  x: at x0, x_step bytes further with every step, or (x_step 0) at x0 of
// the stage.  dst: the warp's first column of row 0; up(m): factor of row m; again (shared memory): set to 1 where a sum is not finite (see sum_again());
// largest + *largest_at (shared memory; null: not asked for): of row m, the largest |sum| as bits, but for rows that are formed again.
// (What is needed behind the steps only waits in shared memory, as they want all registers.)  False where a wait ran out.
template <int TOKS, bool FINE_Z, typename Up>
__device__ __forceinline__ bool rows_segment(const Segment& sg, int steps, int& st, uint32_t& par, uint32_t x0, uint32_t x_step, float* dst,
                                             const Up& up, int& again, uint32_t* largest = nullptr, const int* largest_at = nullptr) {
    using S = Shape<TOKS>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t code_off = (uint32_t)(warp * MEMBERS * KC + g * KC), sw = (uint32_t)g;
    const int slot = lane >> 3, brow = warp * PER + slot;
    const uint32_t byte_off = (uint32_t)(CODE_BYTES + brow * KC), bsw = (uint32_t)(brow & 7);
    // eight columns of half u: thread column mt0, piece lane % 2
    const int mt0 = (lane & 7) >> 1;
    const uint32_t m_step = (uint32_t)(sg.period * META_ROW), m_off = (uint32_t)(META_OFF + sg.cls * META_ROW + (lane & 1) * 64 + mt0 * 16);
    constexpr int CORS = FINE_Z ? S::PAIRS : 2;
    float acc[4][4], cor[CORS][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < CORS; ++i) cor[i][j] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] = 0.f;
    }
    const uint32_t ex = sg.corner, ez = ex + 512;
    // the corner of shared memory: [slot][piece][thread column] scales, [row][piece][thread column] zeros (the pieces of odd rows
    // change places, so that the eight lanes of a load phase touch all banks)
    const uint32_t s_put = ex + slot * 128 + (lane & 1) * 64 + ((lane & 7) >> 1) * 16;
    const uint32_t z_put = ez + (FINE_Z ? slot * 128 + ((lane ^ slot) & 1) * 64 : slot * 64 + (lane & 1) * 8) + ((lane & 7) >> 1) * 16;
    // this lane's B column: row of x and slot inside the fragment
    const int xm = S::SPB == 2 ? (g & 3) : g;
    const uint32_t s_get = ex + (S::SPB == 2 ? (g >> 2) * 128 : 0) + t * 16, z_get = ez + (FINE_Z ? g * 128 + (g & 1) * 64 : g * 64) + t * 16;
    uint32_t xa = x0 + xm * 64 + t * 16;
    for (int p = 0; p < steps; ++p) {
        if (!wait(sg.full + 8 * st, par)) return false;
        const uint32_t sb = sg.ring + st * sg.stage_bytes;
        if (x_step == 0) xa = sb + x0 + xm * 64 + t * 16;          // x comes with the stage
        if (sg.live) {
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
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sg.empty + 8 * st) : "memory");
        xa += x_step;
        if (++st == sg.stages) {
            st = 0;
            par ^= 1;
        }
    }
    if (sg.live) {
        // zeros' sums: row (row of x or slot of the pair's half), column slot and slot + 4: in lane t = slot / 2 and t + 2
#pragma unroll
        for (int i = 0; i < CORS; ++i) {
            if constexpr (FINE_Z && TOKS == 4) {                // both fragments, row g: slots g / 4 and 2 + g / 4
                const float v0 = g < 4 ? cor[i][0] : cor[i][1], v1 = g < 4 ? cor[i][2] : cor[i][3];
                cor[i][0] = v0 + __shfl_xor_sync(0xffffffffu, v0, 2);
                cor[i][1] = v1 + __shfl_xor_sync(0xffffffffu, v1, 2);
            } else if constexpr (FINE_Z) {
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
                const float v = TOKS == 8 ? cor[(s >> 1) % CORS][3 * (s & 1)] : (FINE_Z ? cor[0][s >> 1] : cor[(s >> 1) % CORS][0]);
                z[s] = __shfl_sync(0xffffffffu, v, (TOKS == 4 ? ((s & 1) * 4 + m) * 4 : m * 4) + (s >> 1));
            }
            uint32_t most = 0;                      // of the |sums| this lane writes, as bits: infinities and NaN are the largest
            if (m < sg.M) {
                const float f = up(m);
                float* to = dst + (int64_t)m * sg.row_len + (int64_t)g * sg.G;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float y[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) y[s] = (acc[s][2 * half + e] * (float)(1 << (18 + 2 * s)) - z[s]) * f;
                    auto bits = [](float v) { return __float_as_uint(v) & 0x7fffffffu; };
                    float* at = to + (int64_t)8 * half * sg.G;
                    if constexpr (TOKS == 4) {          // lanes t < 2 hold slots 0 and 2, the others 1 and 3
                        const float a = t < 2 ? y[0] : y[1], b = t < 2 ? y[2] : y[3];
                        at[t >> 1] = a;
                        at[2 + (t >> 1)] = b;
                        most = max(most, max(bits(a), bits(b)));
                    } else {
                        *reinterpret_cast<float4*>(at) = make_float4(y[0], y[1], y[2], y[3]);
                        most = max(max(most, max(bits(y[0]), bits(y[1]))), max(bits(y[2]), bits(y[3])));
                    }
                }
            }
            if (most >= 0x7f800000u) again = 1;
            if (largest) {                          // lanes of one row: same t (TOKS 4: and t + 2)
#pragma unroll
                for (int o = TOKS == 4 ? 2 : 4; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
                if (lane < (TOKS == 4 ? 2 : 4) && m < sg.M && most < 0x7f800000u) atomicMax(largest + *largest_at + m, most);
            }
        }
    }
    return true;
}

// The copying warp's part of a step: three tiles, and the rows of fp16 values of its columns.  A step's fp16 values: rows (array,
// class) of 16 pieces of 16 bytes; a lane copies piece lane % 16 of the arrays lane / 16 and 2 + lane / 16 (src0, src1, at the
// step's column `col` of class 0).  Piece 4 t + 2 u + h is put where (u, h, t) says.  `more`: bytes that the caller adds to the
// barrier.
struct StepCopy {
    int period, lane;
    uint32_t C, k_col;                         // columns until the values repeat; K mod C
    bool elected;
    __device__ __forceinline__ void operator()(uint32_t dst, uint32_t bar, const CUtensorMap* maps, int k, int rho, const uint16_t* src0,
                                               const uint16_t* src1, uint32_t col, uint32_t more = 0) const {
        if (elected) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)META_OFF + more) : "memory");
            tma_3d(dst, maps, k, 0, rho, bar);
            tma_3d(dst + CODE_BYTES, maps + 1, k, PER * rho, 0, bar);
            tma_3d(dst + CODE_BYTES + SZ_BYTES, maps + 2, k, PER * rho, 0, bar);
        }
        const int c16 = lane & 15, hi = lane >> 4;
        uint32_t to = dst + (uint32_t)(META_OFF + hi * period * META_ROW + (c16 & 3) * 64 + (c16 >> 2) * 16), at = col;
        src0 += 8 * c16;
        src1 += 8 * c16;
        for (int cls = 0; cls < period; ++cls) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src0 + at) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 2 * period * META_ROW), "l"(src1 + at) : "memory");
            to += META_ROW;
            at += k_col;
            at = at >= C ? at - C : at;
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    }
};
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}
// A stage is filled when the tiles and 32 lanes' copies are there, free when the computing warps have read it.
__device__ __forceinline__ void init_barriers(uint32_t full, uint32_t empty, int stages) {
    for (int i = 0; i < stages; ++i) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 33;" ::"r"(full + 8 * i));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8 * i), "n"(CW));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Bytes of a stage behind which x may follow.
inline int meta_end(int period) { return META_OFF + (4 * period * META_ROW + 1023) / 1024 * 1024; }
// Residues until (residue * K) mod C repeats; 0: more than a stage has room for.
inline int period_of(int K, int C) {
    for (int p = 1; p <= MAX_PERIOD; ++p)
        if ((int64_t)p * K % C == 0) return p;
    return 0;
}

}  // namespace rows
}  // namespace hqm
