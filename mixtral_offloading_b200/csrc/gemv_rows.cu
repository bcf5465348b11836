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
#include <algorithm>

#include "gemv_rows.cuh"
#include "shared_limit.h"
#include "stream_split.cuh"

namespace hqm {

namespace rows {

struct LayerParams {
    const uint16_t* meta[4];                            // ms_scale, mz_scale, ms_zero, mz_zero
    const uint8_t* data[3];                             // codes, scale bytes, zero bytes
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
    __device__ __forceinline__ int layer_of(int unit) const {
        int l = 0;
#pragma unroll
        for (int i = 1; i < STREAM_MAX_LAYERS; ++i) l += (i < count && unit >= unit0[i]) ? 1 : 0;
        return l;
    }
};

// sum_again() for the runs of this warp.  (A function of its own that finds them anew, called where the warps' roles have come
// together: what the runs are known by would otherwise stay in registers beside the steps, 3 to 4 % of the time at 5 to 8 rows.)
template <bool SCALED>
__device__ __noinline__ void rows_again(const Params& prm, const Split& sp, float* partial, const uint16_t* x, const int32_t* x_idx, int M_total,
                                        const uint32_t* s_max, const int* s_absent) {
    const int warp = threadIdx.x >> 5, K = prm.K, PT = prm.PT;
    const uint32_t first = sp.begin(blockIdx.x);
    const int unit0 = (int)(first / (uint32_t)PT), slot0 = (int)blockIdx.x - sp.owner((uint32_t)unit0 * (uint32_t)PT);
    int pa = (int)(first - (uint32_t)unit0 * (uint32_t)PT), left = (int)(sp.begin(blockIdx.x + 1) - first);
    for (int unit = unit0; left > 0; ++unit, pa = 0) {
        const int pb = min(PT, pa + left);
        left -= pb - pa;
        const int l = prm.layer_of(unit), rho = (unit - prm.unit0[l]) * CW + warp;
        if (rho * PER >= prm.G[l] || (prm.table && s_absent[l])) continue;
        const LayerParams& ly = prm.ly[l];
        Again a{ly.data[0], ly.data[1], ly.data[2], ly.meta[0], ly.meta[1], ly.meta[2], ly.meta[3], K, prm.G[l], prm.C[l], rho, pa * KC, pb * KC};
        if (prm.table) a.layer(prm.table[3 * __ldcg(prm.sel[l]) + prm.which[l]].w);
        const int64_t row_len = prm.col0[prm.count], slot = unit == unit0 ? slot0 : 0;
        for (int m = 0; m < prm.M; ++m) {
            const int e = SCALED ? exponent_of(s_max[m]) : 127;
            a.x = x + ((x_idx ? x_idx[m] : m) + prm.xrow[l]) * (int64_t)K;
            a.down = __uint_as_float((uint32_t)(254 - e) << 23);
            sum_again(a, partial + (slot * M_total + m) * row_len + prm.col0[l] + PER * rho, __uint_as_float((uint32_t)e << 23));
        }
    }
}

template <int TOKS>
__global__ void __launch_bounds__(THREADS, 1)
gemv_rows_kernel(float* __restrict__ partial, const uint16_t* __restrict__ x, const int32_t* __restrict__ x_idx, int M_total,
                 const __grid_constant__ Params prm, const __grid_constant__ Split sp) {
    using S = Shape<TOKS>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ int s_absent[STREAM_MAX_LAYERS];
    __shared__ int s_failed, s_again;
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
        init_barriers(full, empty, stages);
        s_failed = s_again = 0;
    }
    if (threadIdx.x < 8) s_max[threadIdx.x] = 0u;
    __syncthreads();
    // this CTA's steps: from step pa0 of unit0 on; how many CTAs hold a piece of that unit in front of this one
    const uint32_t L0 = sp.begin(blockIdx.x), L1 = sp.begin(blockIdx.x + 1);
    const int unit0 = (int)(L0 / (uint32_t)PT), pa0 = (int)(L0 - (uint32_t)unit0 * (uint32_t)PT), n_steps = (int)(L1 - L0);
    const int slot0 = (int)blockIdx.x - sp.owner((uint32_t)unit0 * (uint32_t)PT);
    auto layer_of = [&](int unit) { return prm.layer_of(unit); };
    auto row_exponent = [&](int m) { return exponent_of(s_max[m]); };

    if (warp == CW) {
        // =========================== copies ===========================
        // (the weights are never written by a kernel of the chain: unless the experts are chosen by a kernel in front, the copies
        // start while that kernel is still running)
        const uint32_t C0 = (uint32_t)prm.C[0], pa_col = (uint32_t)pa0 * KC % C0;
        const StepCopy copy{period, lane, C0, (uint32_t)K % C0, elect_one()};
        const int hi = lane >> 4;
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
            uint32_t col = pa ? pa_col : 0u;                  // of class 0
            for (int p = pa; p < pb; ++p) {
                if (!wait(empty + 8 * st, par)) {
                    // The warps that free a stage may still be waiting for the kernel in front, which has no limit: its time does not
                    // count.  (Waiting for it ahead of the first stage that is not free instead: 0.4 us of 30.5 at one row.)
                    grid_dependency_wait();
                    if (!wait(empty + 8 * st, par)) {
                        ok = false;
                        break;
                    }
                }
                copy(ring + st * stage_bytes, full + 8 * st, maps, p * KC, rho, src0, src1, col);
                col += KC;
                col = col >= C0 ? col - C0 : col;
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
                const Segment sg{ring, full, empty, exch + warp * EXCH_BYTES, stage_bytes, stages, period, cls, M, G, prm.col0[prm.count], live};
                ok = rows_segment<TOKS, S::FINE_Z>(sg, pb - pa, st, par, x_at, S::X_STEP,
                                                   partial + (int64_t)slot_idx * M_total * sg.row_len + prm.col0[l] + PER * rho, [&](int m) {
                    return S::SCALED ? __uint_as_float((uint32_t)row_exponent(m) << 23) : 1.f;
                }, s_again);
            }
            x_at += (uint32_t)(pb_all - pa) * S::X_STEP;
        }
        if (!ok) s_failed = 1;
    }
    __syncthreads();
    if (TOKS > 1 && s_again && !s_failed && warp < CW) rows_again<S::SCALED>(prm, sp, partial, x, x_idx, M_total, s_max, s_absent);
    // ---- a wait ran out: copies may still be on their way to this CTA's shared memory
    if (s_failed) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        if (threadIdx.x == 0 && prm.error_flag) atomicExch(prm.error_flag, 1);
    }
}

static size_t smem_bytes(int toks, int stages, int period, int steps) {
    return 1024 + (size_t)stages * meta_end(period) + (toks > 1 ? (size_t)CW * EXCH_BYTES : 0) + (size_t)steps * toks * KC * 2;
}
static int toks_for(int64_t M) { return M <= 1 ? 1 : (M <= 4 ? 4 : 8); }
static int stages_for(int toks, int period, int steps) {
    for (int s = MAX_STAGES; s >= 2; --s)
        if (smem_bytes(toks, s, period, steps) <= 226 * 1024) return s;
    return 0;
}

template <int TOKS>
static bool prepare(size_t smem) {
    static SharedLimits limits;
    return allow_shared(gemv_rows_kernel<TOKS>, limits, smem);
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
            prm.ly[l].data[0] = static_cast<const uint8_t*>(w->W_q);
            prm.ly[l].data[1] = w->scale_q;
            prm.ly[l].data[2] = w->zero_q;
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
    prm.stage_bytes = meta_end(prm.period);
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
