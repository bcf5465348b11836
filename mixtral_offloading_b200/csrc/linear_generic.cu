// Shape-agnostic quantized linear and full dequantisation.
//
// linear_members_kernel is the path for formats, shapes and row alignments that the
// kernels with 16-bit factors do not take: weights, products and sums in fp32.
// linear_generic_kernel decodes scale and zero per element from their 8-bit form
// (instruction bound, by far); it takes what is left and is the independent check of
// all other kernels (HQM_FORCE_GENERIC).
#include "common.cuh"
#include "kernels.cuh"

namespace hqm {

__device__ __forceinline__ void decode_scale_zero(const hqm_weight& w, int64_t idx, int C, int64_t Cz, float& s,
                                                  float& z) {
    const int col = (int)(idx % C);
    const int64_t colz = (Cz == C) ? col : idx % Cz;
    // explicit rounding steps (no fused multiply-add) so the fp32 result equals the CPU restatement bit for bit
    s = __fmul_rn(__fsub_rn((float)w.scale_q[idx], f16_bits_to_float(w.mz_scale[col])), f16_bits_to_float(w.ms_scale[col]));
    z = __fmul_rn(__fsub_rn((float)w.zero_q[idx], f16_bits_to_float(w.mz_zero[colz])), f16_bits_to_float(w.ms_zero[colz]));
}

template <int NBITS>
__device__ __forceinline__ uint32_t load_word(const hqm_weight& w, int64_t R, int64_t k) {
    if (NBITS == 3) return (uint32_t) reinterpret_cast<const int32_t*>(w.W_q)[R * w.K + k];
    return (uint32_t) reinterpret_cast<const uint8_t*>(w.W_q)[R * w.K + k];
}

// One warp per storage row (PER output rows), lanes strided over k, MT rows of x
// per pass.  x rows may be gathered through x_idx.
template <int NBITS, int MT>
__global__ void __launch_bounds__(256)
linear_generic_kernel(uint16_t* __restrict__ y, const uint16_t* __restrict__ x, const int32_t* __restrict__ x_idx,
                      int M, hqm_weight w, int G, int C, const uint16_t* __restrict__ bias) {
    constexpr int PER = codes_per_word(NBITS);
    constexpr uint32_t MASK = (1u << NBITS) - 1u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t R = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    const int64_t rows = storage_rows(w.N, NBITS);
    if (R >= rows) return;
    const int m0 = blockIdx.y * MT;
    const int K = w.K;
    const int64_t Cz = zero_meta_cols(w, G);

    const uint16_t* xr[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int mm = (m0 + m < M) ? (m0 + m) : (M - 1);
        xr[m] = x + (int64_t)(x_idx ? x_idx[mm] : mm) * K;
    }
    float acc[PER][MT];
#pragma unroll
    for (int s = 0; s < PER; ++s)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[s][m] = 0.f;

    for (int k = lane; k < K; k += 32) {
        const uint32_t word = load_word<NBITS>(w, R, k);
        float xv[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) xv[m] = bf16_bits_to_float(xr[m][k]);
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const int64_t n = R * PER + s;
            if (n < w.N) {
                const float code = (float)((word >> (NBITS * (PER - 1 - s))) & MASK);
                float sc, zr;
                decode_scale_zero(w, (n % G) * K + k, C, Cz, sc, zr);
                const float wv = (code - zr) * sc;
#pragma unroll
                for (int m = 0; m < MT; ++m) acc[s][m] = fmaf(wv, xv[m], acc[s][m]);
            }
        }
    }
#pragma unroll
    for (int s = 0; s < PER; ++s) {
        const int64_t n = R * PER + s;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float v = warp_sum(acc[s][m]);
            if (lane == 0 && n < w.N && m0 + m < M) {
                const float b = bias ? bf16_bits_to_float(bias[n]) : 0.f;
                y[(int64_t)(m0 + m) * w.N + n] = float_to_bf16_bits(v + b);
            }
        }
    }
}

// Four neighbouring columns of a meta vector of C columns, from column c on.
__device__ __forceinline__ void meta4(const uint16_t* p, int c, int C, bool vec, float* f) {
    if (vec) {                                // 8-byte aligned and C a multiple of 4
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(p + c));
        f[0] = f16_bits_to_float((uint16_t)v.x); f[1] = f16_bits_to_float((uint16_t)(v.x >> 16));
        f[2] = f16_bits_to_float((uint16_t)v.y); f[3] = f16_bits_to_float((uint16_t)(v.y >> 16));
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            f[j] = f16_bits_to_float(p[c]);
            c = c + 1 == C ? 0 : c + 1;
        }
    }
}
// Scales and zeros of residue g at four columns from k on; c and cz are their columns of the meta vectors.
__device__ __forceinline__ void decode_four(const hqm_weight& w, int g, int k, int c, int cz, int C, int Cz, bool meta_vec, float* sc, float* zr) {
    const int64_t idx = (int64_t)g * w.K + k;
    const uint32_t sq = *reinterpret_cast<const uint32_t*>(w.scale_q + idx), zq = *reinterpret_cast<const uint32_t*>(w.zero_q + idx);
    float ms[4], mz[4], zs[4], zz[4];
    meta4(w.ms_scale, c, C, meta_vec, ms);
    meta4(w.mz_scale, c, C, meta_vec, mz);
    meta4(w.ms_zero, cz, Cz, meta_vec, zs);
    meta4(w.mz_zero, cz, Cz, meta_vec, zz);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sc[j] = __fmul_rn(__fsub_rn((float)((sq >> (8 * j)) & 255u), mz[j]), ms[j]);
        zr[j] = __fmul_rn(__fsub_rn((float)((zq >> (8 * j)) & 255u), zz[j]), zs[j]);
    }
}
// The packed codes of storage row R at four columns from k on (3 bit: a word per column, else one for the four), and code
// j of them at bit `shift` of its byte or word, as fp32: an OR into 2^23 and an exact subtraction.
template <int NBITS>
__device__ __forceinline__ void load_four(const hqm_weight& w, uint32_t R, int k, uint32_t (&v)[4]) {
    if (NBITS == 3) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const int32_t*>(w.W_q) + (int64_t)R * w.K + k));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        v[0] = __ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(w.W_q) + (int64_t)R * w.K + k));
    }
}
template <int NBITS>
__device__ __forceinline__ float code_of(const uint32_t (&v)[4], int j, int shift) {
    const uint32_t code = (NBITS == 3 ? v[j] >> shift : v[0] >> (8 * j + shift)) & ((1u << NBITS) - 1u);
    return __fsub_rn(__uint_as_float(0x4B000000u | code), 8388608.f);
}

// A CTA: RES neighbouring residues of MC members (OUT output rows) times MT rows of x; its warps take every eighth block of
// 128 columns, a lane 4 columns of it, and add up at the end in warp order.  A scale and a zero are decoded once for MC
// members, a weight once for MT rows: per weight it is the code's shift, mask and conversion, one subtraction, one product
// and MT fused multiply-adds, which bound it; 3 bit: the words, each read for one of its ten codes only.  RES is the number
// of codes in a byte where G is a multiple of it, else 1.  us, before (a decode for every element) / now:
//   3 bit g64 5120 x 4096, 2 to 4 rows     638 / 29       (OUT 8, three CTAs per SM; 16 and two: 41)
//   4 bit g128 4096 x 4096, 4 / 100 rows   129 / 21, 1587 / 308     (OUT 16 / 8, two CTAs; 8 / 4 and three: 27, 426)
//   2 bit g64 14336 x 4096, 5 / 100 rows   573 / 114, 5808 / 1333
__host__ __device__ constexpr int members_out(int nbits, int mt) { return (nbits == 3 ? 32 : 64) / mt; }
template <int NBITS, int RES, int MT>
__global__ void __launch_bounds__(256, NBITS == 3 ? 3 : 2)
linear_members_kernel(uint16_t* __restrict__ y, const uint16_t* __restrict__ x, const int32_t* __restrict__ x_idx, int M, hqm_weight w,
                      int G, int C, const uint16_t* __restrict__ bias, bool meta_vec, bool x_vec) {
    constexpr int PER = codes_per_word(NBITS), OUT = members_out(NBITS, MT), MC = OUT / RES, WARPS = 8, STEP = 128 * WARPS;
    __shared__ float s_sum[WARPS][OUT * MT];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5, K = w.K;
    const int chunks = (w.group_size + MC - 1) / MC;
    const int g0 = (int)(blockIdx.x / chunks) * RES, m0 = (int)(blockIdx.x % chunks) * MC, t0 = (int)blockIdx.y * MT;
    const int Cz = (int)zero_meta_cols(w, G);
    const int k0 = 4 * lane + 128 * wi;
    int c[RES], cz[RES];
#pragma unroll
    for (int r = 0; r < RES; ++r) {
        const int64_t idx = (int64_t)(g0 + r) * K + k0;
        c[r] = (int)(idx % C);
        cz[r] = (int)(idx % Cz);
    }
    const int step = STEP % C, stepz = STEP % Cz;
    const uint16_t* xr[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int t = min(t0 + i, M - 1);
        xr[i] = x + (int64_t)(x_idx ? x_idx[t] : t) * K;
    }
    float acc[OUT][MT];
#pragma unroll
    for (int o = 0; o < OUT; ++o)
#pragma unroll
        for (int i = 0; i < MT; ++i) acc[o][i] = 0.f;

    for (int k = k0; k < K; k += STEP) {
        float sc[RES][4], zr[RES][4], xv[MT][4];
#pragma unroll
        for (int r = 0; r < RES; ++r) {
            decode_four(w, g0 + r, k, c[r], cz[r], C, Cz, meta_vec, sc[r], zr[r]);
            c[r] += step;
            cz[r] += stepz;
            c[r] -= c[r] >= C ? C : 0;
            cz[r] -= cz[r] >= Cz ? Cz : 0;
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            if (x_vec) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(xr[i] + k));
                xv[i][0] = __uint_as_float(v.x << 16); xv[i][1] = __uint_as_float(v.x & 0xffff0000u);
                xv[i][2] = __uint_as_float(v.y << 16); xv[i][3] = __uint_as_float(v.y & 0xffff0000u);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) xv[i][j] = bf16_bits_to_float(xr[i][k + j]);
            }
        }
#pragma unroll
        for (int m = 0; m < MC; ++m) {
            if (m0 + m >= w.group_size) break;
            const uint32_t n0 = (uint32_t)((m0 + m) * G + g0), R = n0 / PER;          // < N
            const int s0 = RES > 1 ? 0 : (int)(n0 - R * PER);
            uint32_t v[4];
            load_four<NBITS>(w, R, k, v);
#pragma unroll
            for (int r = 0; r < RES; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float wv = __fmul_rn(__fsub_rn(code_of<NBITS>(v, j, NBITS * (PER - 1 - s0 - r)), zr[r][j]), sc[r][j]);
#pragma unroll
                    for (int i = 0; i < MT; ++i) acc[m * RES + r][i] = fmaf(wv, xv[i][j], acc[m * RES + r][i]);
                }
        }
    }
#pragma unroll
    for (int o = 0; o < OUT; ++o)
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const float v = warp_sum(acc[o][i]);
            if (lane == 0) s_sum[wi][o * MT + i] = v;
        }
    __syncthreads();
    for (int e = threadIdx.x; e < OUT * MT; e += 256) {
        const int o = e / MT, t = t0 + e % MT, m = m0 + o / RES;
        if (t >= M || m >= w.group_size) continue;
        const int64_t n = (int64_t)m * G + g0 + o % RES;
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) v += s_sum[i][e];
        y[(int64_t)t * w.N + n] = float_to_bf16_bits(v + (bias ? bf16_bits_to_float(bias[n]) : 0.f));
    }
}

// K a multiple of 4, packed tensors aligned for four columns at a time.
static bool four_columns_ok(const hqm_weight* w, int G) {
    auto aligned = [](const void* p, size_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; };
    return w->K % 4 == 0 && aligned(w->W_q, w->nbits == 3 ? 16 : 4) && aligned(w->scale_q, 4) && aligned(w->zero_q, 4) &&
           zero_meta_cols(*w, G) <= INT32_MAX;
}
static bool meta_four_ok(const hqm_weight* w, int G, int C) {
    auto a8 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; };
    return C % 4 == 0 && zero_meta_cols(*w, G) % 4 == 0 && a8(w->ms_scale) && a8(w->mz_scale) && a8(w->ms_zero) && a8(w->mz_zero);
}

template <int NBITS, int RES>
static void linear_members(uint16_t* y, const uint16_t* x, const int32_t* x_idx, int64_t M, const hqm_weight* w, int G, int C,
                           const uint16_t* bias, cudaStream_t st) {
    const bool meta_vec = meta_four_ok(w, G, C), x_vec = (reinterpret_cast<uintptr_t>(x) & 7u) == 0;
    auto go = [&](auto kern, int mt, int mc) {
        const int64_t blocks = (int64_t)(G / RES) * ((w->group_size + mc - 1) / mc);
        kern<<<dim3((unsigned)blocks, (unsigned)((M + mt - 1) / mt)), 256, 0, st>>>(y, x, x_idx, (int)M, *w, G, C, bias, meta_vec, x_vec);
    };
    if (M <= 4) go(linear_members_kernel<NBITS, RES, 4>, 4, members_out(NBITS, 4) / RES);
    else go(linear_members_kernel<NBITS, RES, 8>, 8, members_out(NBITS, 8) / RES);
}

int launch_linear_generic(uint16_t* y, const uint16_t* x, const int32_t* x_idx, int64_t M, const hqm_weight* w, int G,
                          int C, const uint16_t* bias, cudaStream_t st) {
    if (!force_generic() && four_columns_ok(w, G)) {
        if (w->nbits == 3) linear_members<3, 1>(y, x, x_idx, M, w, G, C, bias, st);
        else if (w->nbits == 2) G % 4 == 0 ? linear_members<2, 4>(y, x, x_idx, M, w, G, C, bias, st) : linear_members<2, 1>(y, x, x_idx, M, w, G, C, bias, st);
        else G % 2 == 0 ? linear_members<4, 2>(y, x, x_idx, M, w, G, C, bias, st) : linear_members<4, 1>(y, x, x_idx, M, w, G, C, bias, st);
        HQM_LAUNCH_CHECK();
        return HQM_OK;
    }
    constexpr int MT = 4;
    const int64_t rows = storage_rows(w->N, w->nbits);
    dim3 grid((unsigned)((rows + 7) / 8), (unsigned)((M + MT - 1) / MT));
    switch (w->nbits) {
        case 2: linear_generic_kernel<2, MT><<<grid, 256, 0, st>>>(y, x, x_idx, (int)M, *w, G, C, bias); break;
        case 3: linear_generic_kernel<3, MT><<<grid, 256, 0, st>>>(y, x, x_idx, (int)M, *w, G, C, bias); break;
        default: linear_generic_kernel<4, MT><<<grid, 256, 0, st>>>(y, x, x_idx, (int)M, *w, G, C, bias); break;
    }
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

// ---- full dequantisation (HQQLinearTritonSavable.dequantize) ----------------
template <typename T> __device__ __forceinline__ T cast_out(float v);
template <> __device__ __forceinline__ __nv_bfloat16 cast_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half cast_out<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ float cast_out<float>(float v) { return v; }

template <int NBITS, typename T>
__global__ void dequantize_kernel(T* __restrict__ out, hqm_weight w, int G, int C) {
    constexpr int PER = codes_per_word(NBITS);
    constexpr uint32_t MASK = (1u << NBITS) - 1u;
    const int64_t rows = storage_rows(w.N, NBITS);
    const int64_t total = rows * w.K;
    const int64_t Cz = zero_meta_cols(w, G);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t R = i / w.K, k = i % w.K;
        const uint32_t word = load_word<NBITS>(w, R, k);
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const int64_t n = R * PER + s;
            if (n < w.N) {
                const float code = (float)((word >> (NBITS * (PER - 1 - s))) & MASK);
                float sc, zr;
                decode_scale_zero(w, (n % G) * w.K + k, C, Cz, sc, zr);
                out[n * w.K + k] = cast_out<T>(__fmul_rn(__fsub_rn(code, zr), sc));
            }
        }
    }
}

// The same for K a multiple of 4 and aligned tensors.  A scale and a zero belong to every G-th row: a thread takes RES
// neighbouring residues and 4 columns, decodes their scales and zeros once and goes through `members` rows of each.  RES is
// the number of codes in a byte where G is a multiple of it (a byte then holds the same residues in every member), else 1.
// Bound by the writes.  Per element it is the code's shift, mask and conversion (an OR into 2^23 and an exact subtraction),
// one subtraction, one product; decoding per element with a 64-bit remainder each took 238 us for
// 14336 x 4096 in 2 bits, this takes 33 (floor 21), and 11 for 4096 x 4096 in 4 bits.
template <typename T> struct Four;
template <> struct Four<float> {
    __device__ static void store(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct Four<__half> {
    __device__ static void store(__half* p, const float* v) {
        __half2 h[2] = {__floats2half2_rn(v[0], v[1]), __floats2half2_rn(v[2], v[3])};
        *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(h);
    }
};
template <> struct Four<__nv_bfloat16> {
    __device__ static void store(__nv_bfloat16* p, const float* v) {
        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
        *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(h);
    }
};
constexpr int DEQ_THREADS = 128;
template <int NBITS, int RES, typename T>
__global__ void __launch_bounds__(DEQ_THREADS) dequantize_members_kernel(T* __restrict__ out, hqm_weight w, int G, int C, int members, bool meta_vec) {
    constexpr int PER = codes_per_word(NBITS);
    constexpr uint32_t MASK = (1u << NBITS) - 1u;
    const int K4 = w.K / 4;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= (int64_t)(G / RES) * K4) return;
    const int g0 = (int)(i / K4) * RES, k = (int)(i % K4) * 4;
    const int Cz = (int)zero_meta_cols(w, G);
    // (written out: through decode_four and load_four the 2-bit weight in fp32 takes 2 % longer)
    float sc[RES][4], zr[RES][4];
#pragma unroll
    for (int r = 0; r < RES; ++r) {
        const int64_t idx = (int64_t)(g0 + r) * w.K + k;
        const uint32_t sq = *reinterpret_cast<const uint32_t*>(w.scale_q + idx), zq = *reinterpret_cast<const uint32_t*>(w.zero_q + idx);
        const int c = (int)(idx % C), cz = Cz == C ? c : (int)(idx % Cz);
        float ms[4], mz[4], zs[4], zz[4];
        meta4(w.ms_scale, c, C, meta_vec, ms);
        meta4(w.mz_scale, c, C, meta_vec, mz);
        meta4(w.ms_zero, cz, Cz, meta_vec, zs);
        meta4(w.mz_zero, cz, Cz, meta_vec, zz);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            sc[r][j] = __fmul_rn(__fsub_rn((float)((sq >> (8 * j)) & 255u), mz[j]), ms[j]);
            zr[r][j] = __fmul_rn(__fsub_rn((float)((zq >> (8 * j)) & 255u), zz[j]), zs[j]);
        }
    }
    const int m0 = blockIdx.y * members, m1 = min(m0 + members, w.group_size);
#pragma unroll 4
    for (int m = m0; m < m1; ++m) {
        const uint32_t n0 = (uint32_t)(m * G + g0);           // < N
        const uint32_t R = n0 / PER;
        const int s0 = RES > 1 ? 0 : (int)(n0 - R * PER);
        uint32_t v[4];                                        // NBITS == 3: a word per column, else one for the four
        if (NBITS == 3) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const int32_t*>(w.W_q) + (int64_t)R * w.K + k));
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
            v[0] = __ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(w.W_q) + (int64_t)R * w.K + k));
        }
#pragma unroll
        for (int r = 0; r < RES; ++r) {
            const int shift = NBITS * (PER - 1 - s0 - r);
            float o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t code = (NBITS == 3 ? v[j] >> shift : v[0] >> (8 * j + shift)) & MASK;
                const float c = __fsub_rn(__uint_as_float(0x4B000000u | code), 8388608.f);
                o[j] = __fmul_rn(__fsub_rn(c, zr[r][j]), sc[r][j]);
            }
            Four<T>::store(out + (int64_t)(n0 + r) * w.K + k, o);
        }
    }
}

// 2 bit, 16-bit results, G a multiple of 4: a residue's four values in a column are computed and rounded once, and a byte
// permutation picks one for every member: the low bytes of two columns' values by one PRMT (the two codes are its selector), the
// high bytes by another, a third interleaves them.  9 instructions for 4 weights instead of 22; the same bits.
// A thread takes two of a byte's four residues: with four its tables leave room for 9 CTAs on an SM, 1.35 waves of 14336 x 4096
// (39 us; the kernel above 35.2, this 31.1: 4.5 TB/s; 14336 x 14336 101 -> 86: 5.7 TB/s).
template <typename T> __device__ __forceinline__ uint32_t pack_two(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack_two<__half>(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack_two<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
template <typename T>
__global__ void __launch_bounds__(DEQ_THREADS) dequantize_tables_kernel(T* __restrict__ out, hqm_weight w, int G, int C, int members, bool meta_vec) {
    constexpr int RES = 2;
    const int K4 = w.K / 4;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= (int64_t)(G / RES) * K4) return;
    const int g0 = (int)(i / K4) * RES, k = (int)(i % K4) * 4;
    const int Cz = (int)zero_meta_cols(w, G);
    uint32_t low[RES][4], high[RES][4];                       // the four values' low and high bytes
#pragma unroll
    for (int r = 0; r < RES; ++r) {
        const int64_t idx = (int64_t)(g0 + r) * w.K + k;
        const uint32_t sq = *reinterpret_cast<const uint32_t*>(w.scale_q + idx), zq = *reinterpret_cast<const uint32_t*>(w.zero_q + idx);
        const int c = (int)(idx % C), cz = Cz == C ? c : (int)(idx % Cz);
        float ms[4], mz[4], zs[4], zz[4];
        meta4(w.ms_scale, c, C, meta_vec, ms);
        meta4(w.mz_scale, c, C, meta_vec, mz);
        meta4(w.ms_zero, cz, Cz, meta_vec, zs);
        meta4(w.mz_zero, cz, Cz, meta_vec, zz);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sc = __fmul_rn(__fsub_rn((float)((sq >> (8 * j)) & 255u), mz[j]), ms[j]);
            const float zr = __fmul_rn(__fsub_rn((float)((zq >> (8 * j)) & 255u), zz[j]), zs[j]);
            const uint32_t a = pack_two<T>(__fmul_rn(__fsub_rn(0.f, zr), sc), __fmul_rn(__fsub_rn(1.f, zr), sc));
            const uint32_t b = pack_two<T>(__fmul_rn(__fsub_rn(2.f, zr), sc), __fmul_rn(__fsub_rn(3.f, zr), sc));
            low[r][j] = __byte_perm(a, b, 0x6420);
            high[r][j] = __byte_perm(a, b, 0x7531);
        }
    }
    const int m0 = blockIdx.y * members, m1 = min(m0 + members, w.group_size);
    const int64_t K = w.K, P = G / 4;
    const int shift = (g0 & 2) ? 0 : 4;                       // of the second residue's field; the first one's lies above it
    const uint8_t* codes = reinterpret_cast<const uint8_t*>(w.W_q) + ((int64_t)m0 * P + (g0 >> 2)) * K + k;
    T* to = out + ((int64_t)m0 * G + g0) * K + k;
#pragma unroll 8
    for (int m = m0; m < m1; ++m, codes += P * K, to += (int64_t)G * K) {
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(codes)) >> shift;
#pragma unroll
        for (int r = 0; r < RES; ++r) {
            const uint32_t sel = ((v >> (2 - 2 * r)) & 0x03030303u) | 0x04000400u, sel2 = sel >> 16;
            const uint32_t a = __byte_perm(__byte_perm(low[r][0], low[r][1], sel), __byte_perm(high[r][0], high[r][1], sel), 0x6240);
            const uint32_t b = __byte_perm(__byte_perm(low[r][2], low[r][3], sel2), __byte_perm(high[r][2], high[r][3], sel2), 0x6240);
            *reinterpret_cast<uint2*>(to + r * K) = make_uint2(a, b);
        }
    }
}

template <int NBITS, int RES, typename T>
static void dequantize_members(T* out, const hqm_weight* w, int G, int C, cudaStream_t st) {
    const int64_t threads = (int64_t)(G / RES) * (w->K / 4);
    // Rows per residue of a thread: all of a group, halved down to 4 while that leaves the SMs half empty (a quarter
    // empty or full instead: 35 and 41 us for the 33 above, as every thread decodes the same scales again).
    int members = w->group_size;
    while (members > 4 && threads * ((w->group_size + members - 1) / members) < 148 * 1024) members = (members + 1) / 2;
    const bool meta_vec = meta_four_ok(w, G, C);
    auto grid = [&](int res) {
        return dim3((unsigned)(((int64_t)(G / res) * (w->K / 4) + DEQ_THREADS - 1) / DEQ_THREADS), (unsigned)((w->group_size + members - 1) / members));
    };
    if constexpr (NBITS == 2 && RES == 4 && sizeof(T) == 2) dequantize_tables_kernel<T><<<grid(2), DEQ_THREADS, 0, st>>>(out, *w, G, C, members, meta_vec);
    else dequantize_members_kernel<NBITS, RES, T><<<grid(RES), DEQ_THREADS, 0, st>>>(out, *w, G, C, members, meta_vec);
}

template <typename T>
static int launch_dequantize(void* out, const hqm_weight* w, int G, int C, cudaStream_t st) {
    if (four_columns_ok(w, G) && (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(T) - 1)) == 0 && w->group_size <= 65535) {
        T* o = (T*)out;
        if (w->nbits == 3) dequantize_members<3, 1>(o, w, G, C, st);
        else if (w->nbits == 2) G % 4 == 0 ? dequantize_members<2, 4>(o, w, G, C, st) : dequantize_members<2, 1>(o, w, G, C, st);
        else G % 2 == 0 ? dequantize_members<4, 2>(o, w, G, C, st) : dequantize_members<4, 1>(o, w, G, C, st);
        HQM_LAUNCH_CHECK();
        return HQM_OK;
    }
    const int64_t total = storage_rows(w->N, w->nbits) * w->K;
    int64_t blocks = (total + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    switch (w->nbits) {
        case 2: dequantize_kernel<2, T><<<(int)blocks, 256, 0, st>>>((T*)out, *w, G, C); break;
        case 3: dequantize_kernel<3, T><<<(int)blocks, 256, 0, st>>>((T*)out, *w, G, C); break;
        default: dequantize_kernel<4, T><<<(int)blocks, 256, 0, st>>>((T*)out, *w, G, C); break;
    }
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

}  // namespace hqm

extern "C" int hqm_dequantize(void* W_out, int out_dtype, const hqm_weight* w, void* stream) {
    using namespace hqm;
    int G, C;
    int rc = check_weight(w, &G, &C);
    if (rc != HQM_OK) return rc;
    HQM_CHECK_ARG(W_out != nullptr, "dequantize: null output");
    cudaStream_t st = (cudaStream_t)stream;
    switch (out_dtype) {
        case 0: return launch_dequantize<__nv_bfloat16>(W_out, w, G, C, st);
        case 1: return launch_dequantize<__half>(W_out, w, G, C, st);
        case 2: return launch_dequantize<float>(W_out, w, G, C, st);
        default: set_error("dequantize: out_dtype must be 0 (bf16), 1 (fp16) or 2 (fp32)"); return HQM_ERR_ARG;
    }
}
