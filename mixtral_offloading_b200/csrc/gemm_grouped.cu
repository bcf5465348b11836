// Quantized GEMM on the 5th-generation tensor cores: sums[m, n] = sum_k x[m, k] * W_est[n, k] for one weight or for
// all experts of a MoE block in one launch, each with its own list of rows whose length only the device knows.
// Replaces the reference's Triton kernels (triton_kernels.py:37-131, 225-319), its per-call scale / zero decode
// (custom_layers.py:62-66) and, with the epilogues below, the per-expert loop around them (custom_layers.py:243-256,
// 295-312) for more than a few rows.
//
// The weight is the MMA's A operand: 128 output rows per tile, the rows of x are its N dimension (any multiple of 16
// up to 256: no padding to a fixed tile).  What bounds the kernel is the dequantisation on the CUDA cores, not the
// tensor core and not HBM, so everything is arranged around it:
//
//   * A lives in TMEM.  A dequantised pair of weights goes from registers to tensor memory (tcgen05.st), never
//     through shared memory; `tcgen05.mma` reads it there.  (16 KB per 128 x 64 tile written to and read from shared
//     memory would cost 256 of the ~260 cycles that HBM needs for a tile of 128 columns.)
//   * The 16x256b store shape gives a thread 4 rows x 16 columns of a 32-row quadrant.  Rows are dealt so that its 4
//     rows are members of ONE quantisation group: one (s, -z*s) pair per column serves four weights.
//   * The order of k inside a 64-column block is free as long as x follows it.  A thread takes 16 neighbouring bytes of
//     a storage row (one 128-bit shared-memory load) and pairs columns (k, k+2), which one AND isolates; x is staged
//     in the matching order (tile_pos below).
//   * fp16: a field of a byte, left where it is, IS an fp16 denormal c * 2^(p-24); one fused multiply-add with
//     s * 2^(24-p-2) and -z*s * 2^-2 gives a quarter of the weight.  One AND and one FMA per two weights; the sums are
//     multiplied by 4 at the end.  -z*s is formed from an fp32 z: with z in fp16 the two roundings of z are the largest
//     errors of all (4 bit: 1.07e-3 of the result against 5.5e-4; the streaming kernels' fp16 x * s give 9.8e-4).  Where s * 2^(22-p) leaves the fp16 range (s >= 1/4), the warp takes the longer way
//     for that unit: OR into 1024, exact subtract, FMA.  x is staged as fp16 with a power-of-two factor per row.
//   * bf16 (down projections of more than GG_F16_ROWS rows): OR into 128, exact subtract, FMA.  h has no factor per row, as
//     a row's largest value is not known until every tile of it is finished.  Up to GG_F16_ROWS rows it is fp16 all the same:
//     like the streaming kernels, which took those row counts before and have the same limit, such a launch overflows
//     where |h| exceeds 65504, and one with more rows does not; it keeps three more bits of every h for that.
//
// Measured on B200 (148 SMs): LOP3 / SHF / PRMT and HFMA2 both issue every second cycle per scheduler but on two
// pipes; tcgen05.st of a 128 x 64 tile takes 65 cycles; tcgen05.mma (K = 16, A in TMEM) 15 / 32 / 64 / 128 cycles at
// N = 16 / 64 / 128 / 256 when issued from warp-uniform code (45 when one lane of a diverged warp issues it).
//
// A unit of work is 128 columns of a tile.  Roles of the 24 warps of a CTA (one CTA per SM, persistent):
//   warps 0-15   four groups of four warps; group u % 4 dequantises unit u, warp q of it the TMEM lanes 32q .. 32q+31.
//                A warp decodes the scales and zeros of its own rows into a private corner of shared memory: no barrier
//                between warps.
//   warps 16-19  epilogue
//   warps 20, 21 copies of the packed codes, scale bytes and zero bytes of a unit (tiled TMA, 6 to a unit)
//   warp 22      copies of the staged rows of x (untiled: a tile's rows are contiguous and already swizzled)
//   warp 23      issues the MMAs
//
// Work split: the units of all tiles of all problems follow each other, weighted by what a unit costs with its list's
// row count, and every CTA takes an equal contiguous share (a launch whose rows the host knows: the layout's share, so that
// whole tiles stay whole where their number is no multiple of the CTAs').  A tile cut by a share's boundary is summed from fp32
// pieces in scratch memory by whichever CTA arrives last, in CTA order (no atomics on results, deterministic).
//
// Measured (before: the same layers through a kernel that staged A in shared memory, expert by expert): up + gate of 8
// experts, 4096 -> 14336, 33 tokens: 201 us alone, down 103 us; the whole block 943 -> 299 us (lists of up to 8 rows go to
// gemv_lists.cu by now).  One expert with 512 rows 325 -> 205 us.  A unit takes ~930 cycles (2500 warp instructions) at few rows, with 63 % of the issue
// slots, 6 % of the tensor pipe and 23 % of HBM in use; without the decoding of scales and zeros, the weights' arithmetic
// and the MMAs the same pipeline runs at ~430.  With 256 rows a unit takes 1200 while the MMAs run (1024 their own), but a tile of
// 256 rows has the accumulator to itself, and writing it out took 14.7 us beside the 20.5 of its 32 units; a cut tile of 256 rows
// took another 30 to 38 us to be summed, behind everything else.  What was done about that, one expert with 512 rows, us (224 before):
//   * a CTA takes the tiles that it shares with others first: they are summed under the MMAs of the next ones;
//   * the pieces of a cut tile come by asynchronous copies, 16 rows of several pieces under way (a thread reads what it copied
//     itself); with 8 rows a time 214, with 16 205, and a 4-bit layer of 16 rows 11.35 and 11.12 (11.20 before);
//   * the next 16 rows' sums are asked for before the present ones are worked on; exponential and reciprocal without the branches
//     for denormals, roundings before the exchange between lanes.
//   * where whole tiles are all there is, their addresses and factors are worked out before the sums are waited for, and the room of the
//     pieces holds packed units: 4-bit 6144 x 1024, 40 rows 10.86 -> 10.58, 3-bit 11264 x 4096, 400 rows (whole tiles that used to
//     be cut, as their number is no multiple of the CTAs') 116 -> 106.
// (A second group of epilogue warps, for 8 registers less in each dequantising one: no gain at 512 rows, and 3-bit layers 7 % slower.)
//
// 3-bit layers (ten codes of one column in 32 bits; 10 does not divide the number of groups): storage rows rho + i * P3 hold
// the same residues in the same slots, so a tile is again 8 neighbouring residues x 16 members, from one or two rho.  The
// two bytes that hold a thread's field are picked out of two columns' words by one PRMT and multiplied up to bit 4; the rest
// is as above.  14336 x 4096, 100 rows: 112 us before (decoded tables of scales in memory, dequantisation bound by the
// latency of loads that nothing ran ahead of, A in shared memory), 40 now.
//
// Every wait is bounded; a wait that runs out sets the error flag, all roles leave, TMEM is freed.
#include <cuda.h>
#include <type_traits>

#include "gemm_grouped.cuh"

#include <algorithm>
#include "tc_common.cuh"

namespace hqm {

bool stream_cached_maps(const hqm_weight* w, int G, void* out3);      // gemv_tma.cu

namespace gg {
using namespace tc;

constexpr int GROUPS = 4;                  // dequantising groups of four warps
constexpr int WARP_EPI = 4 * GROUPS, WARP_RAW = WARP_EPI + 4, WARP_B = WARP_RAW + 2, WARP_MMA = WARP_B + 1;
constexpr int NTHREADS = (WARP_MMA + 1) * 32;
// Registers per thread after the roles have split (80 at the launch): 16 x 96 + 4 x 64 + 4 x 32 = 24 x 80.
constexpr int REGS_DEQUANT = 96, REGS_EPI = 64, REGS_ISSUE = 32;
template <int N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int MAX_B_STAGES = 16, MAX_RAW = 2 * GROUPS;
// Cycles of 128 columns of a tile with n rows, the weights of the work split (measured in an expert's up projection, the
// epilogue and cut tiles included: 930 at 16, 1060 at 64, 1400 at 128, 2660 at 256).
__host__ __device__ constexpr int unit_cycles(bool f16, int n) {
    return n > 128 ? n * 10 + (f16 ? 0 : 200) : (f16 ? 900 : 1170) + 4 * n;
}
constexpr int NA = 6;                      // A slots of 128 columns (64 TMEM columns each) at most
// raw full, raw empty, A full, A empty (even and odd rounds of the slots), B full, B empty, accumulator full, empty
constexpr int N_BARS = 2 * MAX_RAW + 3 * NA + 2 * MAX_B_STAGES + 4;
constexpr int TILE_BYTES = 16 * 128 * 2;   // 16 rows of a finished tile, 16 bit; two of them
constexpr int GG_MAX_LAYERS = 4;           // of a launch without a table
constexpr int MERGE_BYTES = 16 * 128 * 4;  // 16 rows of a piece of a cut tile, on their way to the sum
constexpr int EPI_BYTES = 2 * TILE_BYTES + 3 * GG_MAX_ROWS * 4;     // and per row of a chunk: factor, weight, output row
constexpr float F16_SCALE = 4.f;           // A holds a quarter of the weight in fp16 mode

struct Weight {                            // one layer on the device
    const uint16_t* meta[4];               // ms_scale, mz_scale, ms_zero, mz_zero
    const CUtensorMap* maps;               // codes, scale bytes, zero bytes
};
struct Problem {
    Weight w[2];                           // [1]: w3 of GG_UP
    int cnt, n, chunks, cost;              // rows; rows per chunk (padded); chunks; cost of a unit
    int row0, list0;                       // first row in the staged x, first entry in the row list
    int tiles, G, P, C;
    int N, blocks;                         // output rows; blocks of 16 members
    int R, full, left;                     // 3 bit: residues (G is then the rows from member to member); Members3
    int f16;
};

// How a list's rows share the ring of staged x: a stage holds 256 columns of all rows of a chunk (128 beyond 64 rows, 64
// beyond 128 or in a small ring), as a wait, an expectation and a copy together cost the copying warp about 340 cycles.
struct BClass {
    int bytes, stages, blocks;             // bytes reserved per stage, stages in the ring, 64-column blocks in a stage
    __device__ __forceinline__ static BClass of(int n, int ring) {
        BClass c;
        c.blocks = n > 128 || (n > 64 && ring < 128 * 1024) ? 1 : (n > 64 ? 2 : 4);
        const int rows = n <= 16 ? 16 : (n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : 256)));
        c.bytes = rows * 128 * c.blocks;
        c.stages = min(MAX_B_STAGES, ring / c.bytes);
        return c;
    }
};
// TMEM columns: up to 64 rows per chunk in the whole launch, D in two buffers of 64 and six A slots behind them;
// otherwise D in two buffers of 128 (or one of 256) and four A slots.
struct TmemMap {
    uint32_t d_step, a_base;
    int slots;
    __device__ __forceinline__ static TmemMap of(int n_max) {
        return n_max <= 64 ? TmemMap{64u, 128u, 6} : TmemMap{128u, 256u, 4};
    }
};

struct HostProblem {
    CUtensorMap maps[2][3];
    const uint16_t* meta[2][4];
    int G, P, C, tiles, N, blocks, R, full, left;
    void* y;
    const uint16_t* bias;
};

struct Params {
    HostProblem hp[4];
    int problems, K, units_k, subs_k;      // units and 64-column blocks of K
    int chunks;                            // row chunks of n_max rows (one list shared by all problems)
    int N;                                 // output rows of a problem (table mode: common to all)
    const StreamEntry* table;
    int which0, which1;
    const int32_t* counts;
    int rows, few;
    int share, cut;                        // units of a CTA (0: shares of equal cost); some tile may be cut
    const unsigned char* xt;
    int64_t xt_rows;
    const float* row_scale;                // of the staged rows (null: 1)
    int y_f16;
    unsigned char* ht;
    void* out;
    const int32_t* out_idx;
    const float* row_w;
    int accumulate;
    float* parts;                          // [grid][2][n_max][128]
    int n_max;
    uint32_t* counters;
    int* error_flag;
};

// ---- the split of a launch's units over its CTAs -------------------------------------------------------------------
template <int PROBLEMS>
struct Shared {
    Problem pr[PROBLEMS];
    int ubase[PROBLEMS + 1];               // first unit of each problem
    unsigned long long cbase[PROBLEMS + 1];            // cost in front of each problem
    int begin[256];                        // first unit of each CTA ([grid]: all units)
    int last;                              // epilogue: this CTA completes the tile
    uint32_t tmem;
    volatile int failed;
};

// A tile is 8 neighbouring residues (the codes of PARTS neighbouring bytes) of 16 members of their groups; GG_UP: 4 of w1
// and the same 4 of w3.  Larger groups are several blocks of 16 members, each a tile that decodes the scales again: eight
// neighbouring output rows make one 16-byte store.  (4-bit layers with whole groups of 64 in a tile wrote two rows, 4
// bytes, at a time: 3000 cycles per 16 rows of x, more than the tile's own time from 128 rows on.)
template <int NBITS_>
struct Fmt {
    static constexpr int NBITS = NBITS_, MEMBERS = 16;
    static constexpr bool WORDS = NBITS == 3;              // ten codes of one column in 32 bits
    // Residues in a byte.  (3 bit: 8 neighbouring ones as two parts of four; they lie in one or two storage rows.)
    static constexpr int PER = WORDS ? 4 : codes_per_word(NBITS);
    static constexpr int PARTS = 8 / PER;                  // storage-row residues of a tile
    // Columns of a unit.  What a warp does once per unit (waits, decoding, hand-over) takes about as long as the weights of
    // 128 columns of a 2-bit tile, and those layers are large; 4-bit layers decode little and may be small.
    static constexpr int UK = 128;
    static constexpr int BLOCKS = UK / 64;
    static constexpr int SLW = 2;                          // rows of scales a warp needs: its slot of two parts
    static constexpr int CODE_PART = MEMBERS * 128 * (WORDS ? 4 : 1);             // packed bytes of a part of 128 columns
    static constexpr int SZ_PART = PER * 128;
    static constexpr int SQ_OFF = PARTS * CODE_PART, ZQ_OFF = SQ_OFF + PARTS * SZ_PART;
    static constexpr int RAW_TX = ZQ_OFF + PARTS * SZ_PART;
    static constexpr int RAW_BYTES = (RAW_TX + 1023) / 1024 * 1024;
    static constexpr int DC = UK * SLW / 32;               // columns a lane decodes
    static_assert(UK == 128 && DC == 8, "an A slot holds a unit; a lane's columns are one 16-byte load of fp16");
    static constexpr int ST_WARP = SLW * UK * 4;           // s and t of a warp's rows
    static constexpr int ST_BLOCK = 2 * SLW * 64, ST_T = BLOCKS * ST_BLOCK;
    // Launches of up to 64 rows per chunk need few staged rows in flight and many packed bytes, others the reverse.
    __host__ __device__ static constexpr int b_ring(int n_max) { return WORDS ? 80 * 1024 : (n_max <= 64 ? 64 * 1024 : 128 * 1024); }
    // (Even: a slot is filled by one of the two copying warps then, and its phases are waited for in order.)
    // (2 bit, wide chunks: 8 where no tile is cut and nothing is summed: 3072 x 2048, 80 rows 12.9 us with 6, 12.6 with 8.)
    __host__ __device__ static constexpr int n_raw(int n_max, bool cut) { return WORDS || (n_max > 64 && (cut || PARTS == 4)) ? 6 : 8; }
    // Pieces of 16 rows in flight while a cut tile is summed: as many as there is room for.
    __host__ __device__ static constexpr int n_merge(int n_max) { return WORDS ? 1 : (n_max <= 64 ? 4 : (PARTS == 4 ? 1 : 3)); }
    static constexpr int ST_OFF = 0, EPI_OFF = ST_OFF + 4 * GROUPS * ST_WARP, BAR_OFF = EPI_OFF + EPI_BYTES, RING_OFF = BAR_OFF + 1024;
    __host__ __device__ static constexpr int smem(int n_max, bool cut) {
        return (RING_OFF + 1023) / 1024 * 1024 + b_ring(n_max) + n_raw(n_max, cut) * RAW_BYTES + (cut ? n_merge(n_max) * MERGE_BYTES : 0) + 1024;
    }
    static constexpr int max2(int a, int b) { return a > b ? a : b; }
    static constexpr int MOST = max2(max2(smem(64, false), smem(64, true)), max2(smem(256, false), smem(256, true)));
    static constexpr int SHARED = NBITS == 2 ? (int)sizeof(Shared<GG_MAX_PROBLEMS>) : (int)sizeof(Shared<GG_MAX_LAYERS>);
    static_assert(MOST + SHARED <= 227 * 1024, "shared memory");
    // Which row of the tile TMEM lane 32 q + 8 j + g holds (q: warp of a group, j = 0..3): part, slot of the byte, member.
    // A thread of the 16x256b store shape holds j = 0..3 at one g: four members of one quantisation group.
    __device__ __forceinline__ static int part_of(int q, int g) { return (NBITS == 4 ? 2 * (q >> 1) : 0) + (g & 1); }
    __device__ __forceinline__ static int slot_of(int q) { return NBITS == 4 ? q & 1 : q; }
    __device__ __forceinline__ static int member_of(int g, int j) { return (g >> 1) + 4 * j; }
};
// Position of column k of a 64-column block in the staged order (and in the A tile).  (3 bit: a thread column takes words
// 16 i + 4 c .. + 3 instead, so that four neighbouring lanes read 64 contiguous bytes: bits 2-3 and 4-5 of k change places.)
__host__ __device__ constexpr int tile_pos(int k) {
    const int c = k >> 4, i = (k >> 2) & 3, e = k & 3;                  // thread column, word, byte
    return 16 * i + 4 * c + ((e & 1) << 1 | (e >> 1));                  // bytes in the order 0, 2, 1, 3
}

__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for a phase; false when the limit ran out.  try_wait suspends the warp for a while by itself.
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 18); ++i) {
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
// The same as straight-line code (the loop is inside the assembly), for the warps whose values have to stay uniform in the
// compiler's eyes: a branch on a wait's outcome would move every operand of the copies and MMAs behind it to vector
// registers.  `limit`: polls left; 0 once a wait has run out, and every later one then returns at once.
__device__ __forceinline__ void wait_limited(uint32_t bar, uint32_t parity, uint32_t& limit) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 n;\n\t"
        "mov.u32 n, %0;\n\t"
        "GG_WAIT:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra.uni GG_DONE;\n\t"
        "setp.eq.u32 p, n, 0;\n\t"
        "@p bra.uni GG_OUT;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "bra.uni GG_WAIT;\n\t"
        "GG_OUT:\n\t"
        "mov.u32 %0, 0;\n\t"
        "GG_DONE:\n\t}"
        : "+r"(limit)
        : "r"(bar), "r"(parity)
        : "memory");
}
constexpr uint32_t WAIT_LIMIT = 1u << 18;
// A look at a phase without waiting, and the wait that is skipped when the look found it complete: the ~90 cycles of the
// look pass under whatever is issued between the two.
__device__ __forceinline__ uint32_t peek(uint32_t bar, uint32_t parity) {
    uint32_t ready;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ready)
        : "r"(bar), "r"(parity)
        : "memory");
    return ready;
}
__device__ __forceinline__ void wait_peeked(uint32_t bar, uint32_t parity, uint32_t ready, uint32_t& limit) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 n;\n\t"
        "setp.ne.u32 p, %3, 0;\n\t"
        "@p bra.uni GG_DONE;\n\t"
        "mov.u32 n, %0;\n\t"
        "GG_WAIT:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra.uni GG_DONE;\n\t"
        "setp.eq.u32 p, n, 0;\n\t"
        "@p bra.uni GG_OUT;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "bra.uni GG_WAIT;\n\t"
        "GG_OUT:\n\t"
        "mov.u32 %0, 0;\n\t"
        "GG_DONE:\n\t}"
        : "+r"(limit)
        : "r"(bar), "r"(parity), "r"(ready)
        : "memory");
}
__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Four K = 16 steps of one 64-column block; A in TMEM (8 columns per step), B in shared memory (32 bytes per step).
#define GG_MMA4(A, B) \
    "add.u32 a, " A ", 8;\n\tadd.u64 b, " B ", 2;\n\t" \
    "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t" \
    "add.u32 a, a, 8;\n\tadd.u64 b, b, 2;\n\t" \
    "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t" \
    "add.u32 a, a, 8;\n\tadd.u64 b, b, 2;\n\t" \
    "tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t"
__device__ __forceinline__ void mma_block(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b32 a;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        GG_MMA4("%1", "%2") "}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The two blocks of a unit: the second one's rows of x lie `step` descriptor units further on.
__device__ __forceinline__ void mma_unit(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint64_t step) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b32 a, a2;\n\t.reg .b64 b, b2;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"
        "add.u32 a2, %1, 32;\n\tadd.u64 b2, %2, %5;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        GG_MMA4("%1", "%2")
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, q;\n\t"
        GG_MMA4("a2", "b2") "}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "l"(step)
        : "memory");
}
#undef GG_MMA4
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
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
__device__ __forceinline__ uint32_t perm(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ float half_at(uint32_t pair, int hi) { return f16_bits_to_float((uint16_t)(hi ? pair >> 16 : pair)); }
__device__ __forceinline__ float byte_at(uint32_t v, int i) {           // 2^23 + b is exact
    return __uint_as_float(perm(v, 0x4B000000u, 0x7650u + (uint32_t)i)) - 8388608.f;
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
// -z * s / 4 of two columns, z = (byte - zz) * zs in fp32 from bytes i and i + 1 of q and halves zz, zs; s as halves
__device__ __forceinline__ void neg_quarter_zs(uint32_t q, int i, uint32_t zz, uint32_t zs, uint32_t s, float& lo, float& hi) {
    // 2^23 + byte, then -byte / 4, exact
    uint64_t b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "r"(perm(q, 0x4B000000u, 0x7650u + (uint32_t)i)), "r"(perm(q, 0x4B000000u, 0x7651u + (uint32_t)i)));
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(b) : "l"(0xBE800000BE800000ull), "l"(0x4A0000004A000000ull));
    float b0, b1;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(b));
    uint64_t t, u;
    asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "f"(fma_half(zz, 0x34003400u, b0, 0)), "f"(fma_half(zz, 0x34003400u, b1, 1)));
    asm("mov.b64 %0, {%1, %2};" : "=l"(u) : "f"(fma_half(zs, s, 0.f, 0)), "f"(fma_half(zs, s, 0.f, 1)));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(t) : "l"(u));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(t));
}
__device__ __forceinline__ uint32_t bf2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// a / (1 + e^-a): the exponential and the reciprocal of the special function unit, without the branches that keep denormals (the
// result is rounded to bf16; beyond |a| = 87 it is a or zero either way).
__device__ __forceinline__ float silu(float a) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(a * -1.44269504f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    return a * r;
}

__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b) {      // one rounding, as of the fp32 product
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// 16 rows x 32 columns of A from a warp's registers.
__device__ __forceinline__ void store_a(uint32_t at, const uint32_t (&o)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(at), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]),
        "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15])
        : "memory");
}
// The field of slot s (0..9, bits 27 .. 0) of a 3-bit word.
struct Field3 {
    uint32_t sel, up, mask;                // PRMT selector for two words, factor, mask
    int fpos;                              // first bit of the field, less 4
    __device__ __forceinline__ static Field3 of(int s) {
        const uint32_t bit = 3u * (9u - (uint32_t)s), b0 = bit >> 3, b1 = min(b0 + 1, 3u), p = bit & 7;
        Field3 f;
        f.sel = b0 | (b1 << 4) | ((4 + b0) << 8) | ((4 + b1) << 12);
        f.up = p < 4 ? 16u : 1u;
        f.fpos = (int)(p < 4 ? p : p - 4);
        f.mask = (7u << (4 + f.fpos)) * 0x00010001u;
        return f;
    }
};

// A run of this CTA's units inside one tile.
struct Seg {
    int p, tile, chunk, k0, k1;            // problem, tile, row chunk, 128-column units [k0, k1)
    int u, u0;                             // first unit, and where it stands in the CTA's order
};
// This CTA's share, units [begin, end), in the order in which it takes them: the first units of its last tile, where another CTA has the
// rest, then the others.  Tiles that are cut come first this way, at about the same time in both CTAs, and are summed under the
// units that follow instead of behind the last one.
struct Share {
    int begin, end, last;                  // last: units of the last tile, 0 where it is not cut or is the only one
    __device__ __forceinline__ Share(int begin_, int end_, int units_k) : begin(begin_), end(end_), last(end_ % units_k) {
        if (end - last < begin) last = 0;
    }
};
template <int PROBLEMS>
__device__ __forceinline__ bool next_seg(const Shared<PROBLEMS>& sh, const Share& own, int at, int units_k, Seg& s) {
    const bool first = at < own.last;
    const int u = first ? own.end - own.last + at : own.begin + at - own.last, end = first ? own.end : own.end - own.last;
    if (u >= end) return false;
    int p = at <= own.last ? 0 : s.p;
    while (u >= sh.ubase[p + 1]) ++p;
    const int rel = u - sh.ubase[p];
    const int item = rel / units_k;
    s.p = p;
    s.k0 = rel - item * units_k;
    s.k1 = min(units_k, s.k0 + (end - u));
    const int chunks = sh.pr[p].chunks;
    s.tile = item / chunks;
    s.chunk = item - s.tile * chunks;
    s.u = u;
    s.u0 = at;
    return true;
}

template <int NBITS, int MODE>
__global__ void __launch_bounds__(NTHREADS, 1) gg_kernel(const __grid_constant__ Params prm) {
    using F = Fmt<NBITS>;
    constexpr int PER = F::PER, PARTS = F::PARTS, SLW = F::SLW, UK = F::UK, BLOCKS = F::BLOCKS, DC = F::DC;
    extern __shared__ unsigned char smem_raw[];
    __shared__ Shared<MODE == GG_LINEAR ? GG_MAX_LAYERS : GG_MAX_PROBLEMS> sh;
    const uint32_t raw0 = smem_u32(smem_raw);
    unsigned char* base = smem_raw + ((1024u - (raw0 & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(base);
    const int n_raw = F::n_raw(prm.n_max, prm.cut != 0), ring = F::b_ring(prm.n_max);
    const uint32_t b_ring = sbase + (F::RING_OFF + 1023) / 1024 * 1024, raw_ring = b_ring + ring;
    const uint32_t bars = sbase + F::BAR_OFF;
    const uint32_t raw_full = bars, raw_empty = raw_full + 8 * MAX_RAW, a_full = raw_empty + 8 * MAX_RAW, a_empty = a_full + 8 * NA,
                   b_full = a_empty + 16 * NA, b_empty = b_full + 8 * MAX_B_STAGES, acc_full = b_empty + 8 * MAX_B_STAGES,
                   acc_empty = acc_full + 16;
    static_assert(N_BARS * 8 <= 1024, "barrier area");

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int K = prm.K, units_k = prm.units_k;
    const int grid = (int)gridDim.x, cta = (int)blockIdx.x;
    const bool counted = prm.counts != nullptr;

    grid_launch_dependents();
    // ---- set-up: barriers, TMEM, problems side by side on three warps
    if (warp == WARP_RAW) {
        for (int i = lane; i < N_BARS; i += 32) {
            // a slot of packed bytes is released, an A slot filled, by the four warps of a group, an accumulator by four warps
            const bool four = (i >= MAX_RAW && i < 2 * MAX_RAW + NA) || i >= N_BARS - 2;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8 * i), "r"(four ? 4u : 1u));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == WARP_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        if (lane == 0) sh.failed = 0;
    }
    // the row counts come from a kernel in front; without them the copies of the weights may start at once
    if (counted) grid_dependency_wait();
    if (warp == 0) {
        // lane e: problem e, its units and their cost; prefix sums over the lanes
        const int e = lane;
        int cnt = 0, units = 0, rows = 0, cost = 0;
        if (e < prm.problems) {
            Problem& p = sh.pr[e];
            const HostProblem& h = prm.hp[prm.table ? 0 : e];
            cnt = counted ? __ldcg(prm.counts + e) : prm.rows;
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                if (prm.table) {
                    const StreamEntry* en = prm.table + 3 * e + (l ? prm.which1 : prm.which0);
                    p.w[l].meta[0] = en->w.ms_scale;
                    p.w[l].meta[1] = en->w.mz_scale;
                    p.w[l].meta[2] = en->w.ms_zero;
                    p.w[l].meta[3] = en->w.mz_zero;
                    p.w[l].maps = reinterpret_cast<const CUtensorMap*>(en->maps);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) p.w[l].meta[i] = h.meta[l][i];
                    p.w[l].maps = h.maps[l];
                }
            }
            p.G = h.G;
            p.P = h.P;
            p.C = h.C;
            p.tiles = h.tiles;
            p.N = h.N;
            p.blocks = h.blocks;
            p.R = h.R;
            p.full = h.full;
            p.left = h.left;
            p.cnt = cnt;
            const GgRows r = counted ? GgRows::of(cnt) : GgRows{prm.chunks, prm.n_max};
            p.n = r.n;
            p.chunks = r.chunks;
            p.f16 = (MODE != GG_DOWN || cnt <= GG_F16_ROWS) ? 1 : 0;
            // cycles of 128 columns: the dequantisation, or the MMAs (4 per row)
            cost = unit_cycles(p.f16, p.n);
            p.cost = cost;
            rows = r.padded();
            units = cnt <= prm.few ? 0 : h.tiles * r.chunks * units_k;
        }
        int row1 = rows, list1 = cnt, u1 = units;
        unsigned long long c1 = (unsigned long long)units * (unsigned)cost;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, row1, o), b = __shfl_up_sync(0xffffffffu, list1, o), c = __shfl_up_sync(0xffffffffu, u1, o);
            const unsigned long long d = __shfl_up_sync(0xffffffffu, c1, o);
            if (lane >= o) {
                row1 += a;
                list1 += b;
                u1 += c;
                c1 += d;
            }
        }
        if (e < prm.problems) {
            sh.pr[e].row0 = counted ? row1 - rows : 0;
            sh.pr[e].list0 = counted ? list1 - cnt : 0;
            sh.ubase[e + 1] = u1;
            sh.cbase[e + 1] = c1;
        }
        if (e == 0) {
            sh.ubase[0] = 0;
            sh.cbase[0] = 0;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (prm.share > 0) {
        if ((int)threadIdx.x <= grid) sh.begin[threadIdx.x] = min(sh.ubase[prm.problems], (int)threadIdx.x * prm.share);
    } else if ((int)threadIdx.x <= grid) {
        const unsigned long long total = sh.cbase[prm.problems];
        const unsigned long long at = total * (unsigned long long)threadIdx.x / (unsigned)grid;
        int e = 0;
        while (e < prm.problems - 1 && at >= sh.cbase[e + 1]) ++e;
        const unsigned long long rel = at - sh.cbase[e];
        const unsigned cost = (unsigned)max(1, sh.pr[e].cost);
        sh.begin[threadIdx.x] = (int)threadIdx.x == grid ? sh.ubase[prm.problems] : sh.ubase[e] + (int)((rel + cost - 1) / cost);
    }
    __syncthreads();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem, 0);
    const Share own(sh.begin[cta], sh.begin[cta + 1], units_k);
    const TmemMap tmap = TmemMap::of(prm.n_max);
    const int slots = tmap.slots;

    if (warp < WARP_EPI) {
        regs_up<REGS_DEQUANT>();
        // =========================== dequantisation ===========================
        const int group = warp >> 2, q = warp & 3, g = lane >> 2, c = lane & 3;
        const int part = F::part_of(q, g), slot = F::slot_of(q);
        // the row of scales / zeros this lane decodes: DC columns of it
        const int dlocal = lane >> 4, dpart = F::part_of(q, dlocal);
        const int dcol = DC * (lane & (UK / DC - 1));
        // The field of the warp's slot inside a byte.  2 bit: slots 0, 1 at bits 7-6, 5-4, slots 2, 3 at 3-2, 1-0; 4 bit: 7-4 or
        // 3-0.  `upper`: it lies in the upper half of the byte; fpos: its first bit inside that half.
        const bool upper = (NBITS == 2) ? q < 2 : (q & 1) == 0;
        const int fpos = (NBITS == 2) ? ((q & 1) ? 0 : 2) : 0;              // (3 bit: set for every tile)
        const uint32_t field = (NBITS == 2) ? 3u : 15u;
        const uint32_t mask_hi = (field << (4 + fpos)) * 0x00010001u;      // field in bits 7-4 of each half
        const uint32_t mask_lo = (field << fpos) * 0x00010001u;            // field in bits 3-0 of each half
        // s / t of the warp: [block][half][part][thread column][8 values], s first; 16-byte pieces, so that the eight lanes of
        // a load phase touch 128 contiguous bytes
        const uint32_t st_area = sbase + F::ST_OFF + warp * F::ST_WARP;
        const uint32_t st_read = st_area + (g & 1) * 64 + c * 16;
        // this thread's bytes of a staged row: 16 of a 64-column block, members j = 0, 1 (the 128-byte swizzle)
        uint32_t code_off[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int m = F::member_of(g, j);
            code_off[j] = (uint32_t)(part * F::CODE_PART + m * 128 + ((c ^ (m & 7)) << 4));
        }
        constexpr int J2 = 8 * 128;                      // from members j = 0, 1 to j = 2, 3

        Seg s;
        s.p = 0;
        int at = 0;
        // meta values (fp16 scale / zero of the 8-bit scale and zero bytes), requested a unit ahead
        uint32_t mt[4][DC / 2];
        int mcol = 0, mC = 1, mstep = 0;
        const uint16_t* mp[4] = {nullptr, nullptr, nullptr, nullptr};
        auto load_meta = [&]() {
            if ((mC & 7) == 0) {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(mp[a] + mcol));
                    mt[a][0] = v.x; mt[a][1] = v.y; mt[a][2] = v.z; mt[a][3] = v.w;
                }
            } else {                                          // a run of columns may wrap around anywhere: one by one
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int j = 0; j < DC / 2; ++j) {
                        const uint32_t lo = __ldg(mp[a] + (mcol + 2 * j) % mC), hi = __ldg(mp[a] + (mcol + 2 * j + 1) % mC);
                        mt[a][j] = lo | (hi << 16);
                    }
            }
        };
        int r = group, v = group;                             // slots of this group's next unit: packed bytes; A, and its phase
        uint32_t r_par = 0, v_round = 0, limit = WAIT_LIMIT, raw_ready = 0, a_ready = 0;
        // The A slot that has been written and not yet handed to the MMAs: the stores are waited for when the next unit's loads
        // are on their way (or before a wait for them).
        uint32_t pending = 0;
        auto hand_over = [&] {
            if (pending) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                if (lane == 0) arrive(pending);
                pending = 0;
            }
        };
        while (next_seg(sh, own, at, units_k, s)) {
            const int n_seg = s.k1 - s.k0;
            at += n_seg;
            int first = group - s.u0 % GROUPS;                // first unit of the run that is this group's
            if (first < 0) first += GROUPS;
            if (first >= n_seg) continue;
            const Problem& pr = sh.pr[s.p];
            const bool f16 = pr.f16 != 0;
            const int wsel = (MODE == GG_UP) ? dpart : 0;
            const int rho = (MODE == GG_UP) ? s.tile : s.tile / pr.blocks * PARTS + dpart;
            // 3 bit: the words of this thread's residue and, in them, its field: two bytes that hold it at bit 0 .. 7, moved up to
            // bit 4 + fpos; the same of the residue whose scales this lane decodes
            Field3 mine{}, decoded{};
            uint32_t words3 = 0;
            if constexpr (F::WORDS) {
                const int q0 = s.tile / pr.blocks * 8, r0 = q0 / 10, e = q0 + PER * part + slot;
                mine = Field3::of(e % 10);
                decoded = Field3::of((PER * rho + slot) % 10);
                words3 = (uint32_t)((e / 10 - r0) * F::CODE_PART + (g >> 1) * 512 + c * 16);
            }
            const int res = F::WORDS ? (PER * rho + slot) % pr.R : min(PER * rho + slot, pr.G - 1);  // (a tile's last parts may lie past the last residue)
            mC = pr.C;
#pragma unroll
            for (int a = 0; a < 4; ++a) mp[a] = pr.w[wsel].meta[a];
            mcol = (int)(((uint64_t)res * (uint32_t)K + (uint32_t)((s.k0 + first) * UK + dcol)) % (uint32_t)mC);
            mstep = (GROUPS * UK) % mC;
            load_meta();
            for (int k = s.k0 + first; k < s.k1; k += GROUPS) {
                if (!raw_ready) hand_over();
                wait_peeked(raw_full + 8 * r, r_par, raw_ready, limit);
                const uint32_t rw = raw_ring + r * F::RAW_BYTES;
                uint4 wv[4];
                auto load_codes = [&](int sub) {
                    if constexpr (F::WORDS) return;
                    const uint32_t c0 = rw + (code_off[0] ^ (64u * sub)), c1 = rw + (code_off[1] ^ (64u * sub));
                    wv[0] = lds128(c0);
                    wv[1] = lds128(c1);
                    wv[2] = lds128(c0 + J2);
                    wv[3] = lds128(c1 + J2);
                };
                // ---- scale and zero of the warp's rows
                bool big = false;
                {
                    const uint32_t sqa = rw + F::SQ_OFF + dpart * F::SZ_PART + slot * 128 + dcol;
                    constexpr int ZS = F::ZQ_OFF - F::SQ_OFF;
                    const uint2 s8 = lds64(sqa), z8 = lds64(sqa + ZS);
                    const uint32_t sq[DC / 4] = {s8.x, s8.y}, zq[DC / 4] = {z8.x, z8.y};
                    load_codes(0);                            // on their way while the scales are decoded
                    hand_over();
                    a_ready = v_round > 0 ? peek(a_empty + 8 * (v + ((v_round & 1) ? 0 : NA)), ((v_round - 1) >> 1) & 1) : 1u;
                    uint32_t S[DC / 2], T[DC / 2];            // per four columns: pair (0, 2), pair (1, 3)
                    if (f16) {
                        // s * 2^(22 - p) and -z * s / 4, p = 4 + fpos the field's first bit.  The second is formed from the rounded s
                        // and an unrounded z: what s is off then scales the whole (c - z) s, and T adds one rounding of its own.
#pragma unroll
                        for (int j = 0; j < DC / 4; ++j) {
                            uint32_t s2[2];
                            float tt[4];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const uint32_t qs = h2sub(perm(sq[j], 0x64646464u, e ? 0x4342u : 0x4140u), 0x64006400u);
                                s2[e] = h2mul(h2sub(qs, mt[1][2 * j + e]), mt[0][2 * j + e]);
                                neg_quarter_zs(zq[j], 2 * e, mt[3][2 * j + e], mt[2][2 * j + e], s2[e], tt[2 * e], tt[2 * e + 1]);
                            }
                            // to the order (0, 2), (1, 3)
                            S[2 * j] = perm(s2[0], s2[1], 0x5410u);
                            S[2 * j + 1] = perm(s2[0], s2[1], 0x7632u);
                            T[2 * j] = h2_of(tt[0], tt[2]);
                            T[2 * j + 1] = h2_of(tt[1], tt[3]);
                        }
                        // |s| * 2^(18 - fpos) must stay finite: |s| < 1/4 (fpos = 2: < 1)
                        uint32_t mx = 0;
#pragma unroll
                        for (int j = 0; j < DC / 2; ++j) mx = __vmaxu2(mx, S[j] & 0x7FFF7FFFu);
                        big = __any_sync(0xffffffffu, (mx & 0xffffu) > 0x33FFu || (mx >> 16) > 0x33FFu);           // 1/4 and more
                        // * 2^(18 - fpos), exact; big: the field will be read as c * 2^(4 + fpos), so s / 4 / 2^(4 + fpos)
                        const uint32_t f1 = big ? 0x3C003C00u : 0x64006400u;
                        const uint32_t f2 = (big ? 0x24002400u : 0x5C005C00u) - (uint32_t)(F::WORDS ? decoded.fpos : fpos) * 0x04000400u;
#pragma unroll
                        for (int j = 0; j < DC / 2; ++j) S[j] = h2mul(h2mul(S[j], f1), f2);
                    } else {
                        // bf16: s * 2^-fpos and -z * s, computed in fp32
                        const float down = fpos ? 0.25f : 1.f;
#pragma unroll
                        for (int j = 0; j < DC / 4; ++j) {
                            float sc[4], tt[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int i = 2 * j + (e >> 1);
                                sc[e] = (byte_at(sq[j], e) - half_at(mt[1][i], e & 1)) * half_at(mt[0][i], e & 1);
                                const float z = (byte_at(zq[j], e) - half_at(mt[3][i], e & 1)) * half_at(mt[2][i], e & 1);
                                tt[e] = -z * sc[e];
                                sc[e] *= down;
                            }
                            S[2 * j] = bf2(sc[0], sc[2]);
                            S[2 * j + 1] = bf2(sc[1], sc[3]);
                            T[2 * j] = bf2(tt[0], tt[2]);
                            T[2 * j + 1] = bf2(tt[1], tt[3]);
                        }
                    }
                    // publish to the warp
                    if constexpr (F::WORDS) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int w64 = (dcol + 4 * h) & 63, blk = (dcol + 4 * h) >> 6, i = w64 >> 4;
                            const uint32_t dst = st_area + blk * F::ST_BLOCK + (i >> 1) * (SLW * 64) + dlocal * 64 + ((w64 >> 2) & 3) * 16 + (i & 1) * 8;
                            asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(dst), "r"(S[2 * h]), "r"(S[2 * h + 1]) : "memory");
                            asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(dst + F::ST_T), "r"(T[2 * h]), "r"(T[2 * h + 1]) : "memory");
                        }
                    } else {
                        const int w64 = dcol & 63, blk = dcol >> 6;
                        const uint32_t dst = st_area + blk * F::ST_BLOCK + ((w64 >> 3) & 1) * (SLW * 64) + dlocal * 64 + (w64 >> 4) * 16;
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(S[0]), "r"(S[1]), "r"(S[2]), "r"(S[3]) : "memory");
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + F::ST_T), "r"(T[0]), "r"(T[1]), "r"(T[2]), "r"(T[3]) : "memory");
                    }
                }
                if (k + GROUPS < s.k1) {                      // the next unit's meta values
                    mcol += mstep;
                    if (mcol >= mC) mcol -= mC;
                    load_meta();
                }
                __syncwarp();
                // ---- the weights, 64 columns at a time
                const int subs = min(BLOCKS, prm.subs_k - BLOCKS * k);
                // The A slot's tile of the round before has been read by its MMAs.  (A parity only tells the last phase from
                // the one before it: even and odd rounds have barriers of their own.)
                if (v_round > 0) wait_peeked(a_empty + 8 * (v + ((v_round & 1) ? 0 : NA)), ((v_round - 1) >> 1) & 1, a_ready, limit);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = tmem + tmap.a_base + 64 * v + ((uint32_t)(32 * q) << 16);
#pragma unroll 1                                  // (unrolled it is 3 % slower: the code of 16 warps at different places)
                for (int sub = 0; sub < 2; ++sub) {
                    if (sub < subs) {
                        const uint32_t sa = st_read + sub * F::ST_BLOCK;
                        const uint4 S0 = lds128(sa), S1 = lds128(sa + SLW * 64), T0 = lds128(sa + F::ST_T), T1 = lds128(sa + F::ST_T + SLW * 64);
                        if (sub) load_codes(sub);
                        const uint32_t SS[8] = {S0.x, S0.y, S0.z, S0.w, S1.x, S1.y, S1.z, S1.w};
                        const uint32_t TT[8] = {T0.x, T0.y, T0.z, T0.w, T1.x, T1.y, T1.z, T1.w};
                        if constexpr (F::WORDS) {
                            const uint32_t at0 = rw + words3 + 256u * sub;
                            auto all3 = [&](auto&& weight) {
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    uint32_t o[16];
#pragma unroll
                                    for (int b = 0; b < 2; ++b)
#pragma unroll
                                        for (int i = 0; i < 4; ++i) {
                                            const uint4 v = lds128(at0 + (2 * h + b) * 2048 + 64 * i);
                                            o[4 * i + 2 * b] = weight(perm(v.x, v.z, mine.sel) * mine.up, SS[2 * i], TT[2 * i]);
                                            o[4 * i + 2 * b + 1] = weight(perm(v.y, v.w, mine.sel) * mine.up, SS[2 * i + 1], TT[2 * i + 1]);
                                        }
                                    store_a(ta + 32 * sub + ((uint32_t)(16 * h) << 16), o);
                                }
                            };
                            const uint32_t magic = 0x64006400u;                                                     // 1024
                            if (!big) all3([&](uint32_t x, uint32_t S, uint32_t T) { return h2fma(x & mine.mask, S, T); });
                            else all3([&](uint32_t x, uint32_t S, uint32_t T) { return h2fma(h2sub(lop_and_or(x, mine.mask, magic), magic), S, T); });
                            continue;
                        }
                        // one pair of weights per (member, word i, e): fields of bytes (0, 2) and (1, 3) of the word
                        auto all = [&](auto&& pair_lo, auto&& pair_hi) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                uint32_t o[16];
#pragma unroll
                                for (int b = 0; b < 2; ++b) {
                                    const uint4 vv = wv[2 * h + b];
                                    const uint32_t w[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        o[4 * i + 2 * b] = pair_lo(w[i], SS[2 * i], TT[2 * i]);
                                        o[4 * i + 2 * b + 1] = pair_hi(w[i], SS[2 * i + 1], TT[2 * i + 1]);
                                    }
                                }
                                store_a(ta + 32 * sub + ((uint32_t)(16 * h) << 16), o);
                            }
                        };
                        // (the shift to the left is written as a product: it then runs beside the ANDs, on the other pipe)
                        if (f16 && !big) {
                            if (upper)
                                all([&](uint32_t x, uint32_t S, uint32_t T) { return h2fma(x & mask_hi, S, T); },
                                    [&](uint32_t x, uint32_t S, uint32_t T) { return h2fma((x >> 8) & mask_hi, S, T); });
                            else
                                all([&](uint32_t x, uint32_t S, uint32_t T) { return h2fma((x * 16u) & mask_hi, S, T); },
                                    [&](uint32_t x, uint32_t S, uint32_t T) { return h2fma((x >> 4) & mask_hi, S, T); });
                        } else if (f16) {
                            const uint32_t magic = 0x64006400u, mul = upper ? 1u : 16u, sh = upper ? 8u : 4u;      // 1024
                            all([&](uint32_t x, uint32_t S, uint32_t T) { return h2fma(h2sub(lop_and_or(x * mul, mask_hi, magic), magic), S, T); },
                                [&](uint32_t x, uint32_t S, uint32_t T) { return h2fma(h2sub(lop_and_or(x >> sh, mask_hi, magic), magic), S, T); });
                        } else {
                            const uint32_t magic = 0x43004300u, sl = upper ? 4u : 0u;                               // 128
                            all([&](uint32_t x, uint32_t S, uint32_t T) { return bf2_fma(bf2_sub(lop_and_or(x >> sl, mask_lo, magic), magic), S, T); },
                                [&](uint32_t x, uint32_t S, uint32_t T) { return bf2_fma(bf2_sub(lop_and_or(x >> (sl + 8u), mask_lo, magic), magic), S, T); });
                        }
                    }
                }
                // The staged bytes have been read.  (Only here: what was loaded has been used by every lane.)
                __syncwarp();
                if (lane == 0) arrive(raw_empty + 8 * r);
                pending = a_full + 8 * v;
                r += GROUPS;
                if (r >= n_raw) {
                    r -= n_raw;
                    r_par ^= 1u;
                }
                v += GROUPS;
                if (v >= slots) {
                    v -= slots;
                    ++v_round;
                }
                raw_ready = peek(raw_full + 8 * r, r_par);
            }
        }
        hand_over();
        if (limit == 0) sh.failed = 1;
    } else if (warp >= WARP_RAW) {
        regs_down<REGS_ISSUE>();
        // The copying and the MMA-issuing warps: all lanes run the same code on the same values and an elected one issues, so
        // that the operands live in uniform registers (a tiled copy then costs 30 cycles, 100 when lanes issue one each).
        const bool leader = elect_one();
        uint32_t limit = WAIT_LIMIT;
        Seg s;
        s.p = 0;
        int at = 0;
        if (warp < WARP_B) {
            // =========================== packed weights: two warps, every other unit each ===========================
            const int turn = warp - WARP_RAW;
            int fenced = -1;
            while (next_seg(sh, own, at, units_k, s)) {
                at += s.k1 - s.k0;
                const Problem& pr = sh.pr[s.p];
                const CUtensorMap* maps[2] = {pr.w[0].maps, pr.w[MODE == GG_UP ? 1 : 0].maps};
                const int quad = (MODE == GG_UP) ? s.tile : s.tile / pr.blocks, rho0 = (MODE == GG_UP) ? quad : quad * PARTS;
                const int m0 = (MODE == GG_UP) ? 0 : 16 * (s.tile - quad * pr.blocks);
                if (prm.table && fenced != s.p) {             // tensor maps in global memory
                    fenced = s.p;
#pragma unroll
                    for (int i = 0; i < 3 * (MODE == GG_UP ? 2 : 1); ++i)
                        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(maps[i / 3] + i % 3) : "memory");
                }
                for (int k = s.k0 + ((s.u0 ^ turn) & 1); k < s.k1; k += 2) {
                    const int u = s.u0 + (k - s.k0), lap = u / n_raw, r = u - lap * n_raw;
                    wait_limited(raw_empty + 8 * r, (lap & 1) ^ 1, limit);
                    const uint32_t bar = raw_full + 8 * r, dst = raw_ring + r * F::RAW_BYTES;
                    if constexpr (F::WORDS) {
                        const int r0 = 8 * quad / 10, two = 8 * quad - 10 * r0 > 2 ? 2 : 1;           // storage rows of a member
                        if (leader) {
                            expect_tx(bar, (uint32_t)(two * 512 * (min(pr.full, 16) + (pr.left ? 1 : 0)) + 2 * 1024));
                            for (int p = 0; p < two; ++p) {
                                tma_3d(dst + p * F::CODE_PART, maps[0], k * UK, r0 + p, m0, bar);
                                if (pr.left) tma_3d(dst + p * F::CODE_PART + pr.full * 512, maps[0] + 3, k * UK, r0 + p, 0, bar);
                            }
                            tma_3d(dst + F::SQ_OFF, maps[0] + 1, k * UK, 8 * quad % pr.R, 0, bar);
                            tma_3d(dst + F::ZQ_OFF, maps[0] + 2, k * UK, 8 * quad % pr.R, 0, bar);
                        }
                        continue;
                    }
                    if (leader) {
                        expect_tx(bar, F::RAW_TX);
#pragma unroll
                        for (int p = 0; p < PARTS; ++p) {
                            const int rho = (MODE == GG_UP) ? rho0 : rho0 + p;
                            const CUtensorMap* map = maps[MODE == GG_UP ? p : 0];
                            tma_3d(dst + p * F::CODE_PART, map, k * UK, rho, m0, bar);
                            tma_3d(dst + F::SQ_OFF + p * F::SZ_PART, map + 1, k * UK, PER * rho, 0, bar);
                            tma_3d(dst + F::ZQ_OFF + p * F::SZ_PART, map + 2, k * UK, PER * rho, 0, bar);
                        }
                    }
                }
            }
        } else if (warp == WARP_B) {
            // =========================== rows of x ===========================
            // Where the stage size changes the ring is emptied first, so that both sides start over at stage 0.
            if (!counted) grid_dependency_wait();
            int cls = 0, st = 0, filled = 0;                  // filled: stages that have been used since the last change
            uint32_t par = 0xffffffffu;                       // bit i: parity that a wait for "stage i is free" expects
            while (next_seg(sh, own, at, units_k, s)) {
                at += s.k1 - s.k0;
                const Problem& pr = sh.pr[s.p];
                const BClass bc = BClass::of(pr.n, ring);
                if (bc.bytes != cls) {
                    for (int i = 0; i < filled; ++i) wait_limited(b_empty + 8 * i, (par >> i) & 1, limit);       // its last use has been read
                    // (the stage's next fill waits for the same phase again, and finds it complete)
                    cls = bc.bytes;
                    st = 0;
                    filled = 0;
                }
                const uint32_t bytes = (uint32_t)pr.n * 128u;
                const unsigned char* src = prm.xt + ((int64_t)(BLOCKS * s.k0) * prm.xt_rows + pr.row0 + s.chunk * pr.n) * 128;
                const int64_t step = prm.xt_rows * 128;
                const int b1 = min(BLOCKS * s.k1, prm.subs_k);
                for (int b = BLOCKS * s.k0; b < b1; b += bc.blocks) {
                    wait_limited(b_empty + 8 * st, (par >> st) & 1, limit);
                    par ^= 1u << st;
                    const int blocks = min(bc.blocks, b1 - b);
                    if (leader) {
                        const uint32_t dst = b_ring + (uint32_t)st * (uint32_t)bc.bytes, bar = b_full + 8 * st;
                        expect_tx(bar, bytes * (uint32_t)blocks);
                        for (int i = 0; i < blocks; ++i) bulk_load(dst + bytes * (uint32_t)i, src + step * i, bytes, bar);
                    }
                    src += step * bc.blocks;
                    if (st + 1 > filled) filled = st + 1;
                    st = (st + 1 == bc.stages) ? 0 : st + 1;
                }
            }
        } else {
            // =========================== MMAs ===========================
            const uint32_t a_first = tmem + tmap.a_base, a_end = a_full + 8 * (uint32_t)slots;
            uint32_t a_bar = a_full, a_tmem = a_first, a_par = 0;            // the A slot of the next 128 columns
            uint32_t par = 0;                                 // bit i: parity that a wait for "stage i is filled" expects
            int cls = 0, st = 0, seg = 0;
            bool prev_wide = false;
            uint32_t ready = 0;
            while (next_seg(sh, own, at, units_k, s)) {
                at += s.k1 - s.k0;
                const Problem& pr = sh.pr[s.p];
                const int n = pr.n;
                const bool wide = n > 128;
                const BClass bc = BClass::of(n, ring);
                if (bc.bytes != cls) {
                    cls = bc.bytes;
                    st = 0;
                }
                const uint32_t idesc = (1u << 4) | (pr.f16 ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
                const int buf = wide ? 0 : seg & 1;
                // the accumulator is free: the run before last has been read; next to a run of more than 128 rows, the last one
                const int need = (wide || prev_wide) ? seg - 1 : seg - 2;
                if (need >= 0) wait_limited(acc_empty + 8 * (need & 1), (need >> 1) & 1, limit);
                prev_wide = wide;
                const uint32_t d = tmem + tmap.d_step * (uint32_t)buf;
                const uint32_t sub_step = (uint32_t)n * 8u;   // descriptor units of a 64-column block: (n rows * 128 bytes) / 16
                const uint64_t desc = (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
                uint32_t acc = 0;
                int left = 0;                                 // units of the current stage of x still to be used
                uint64_t bd = 0;
                for (int k = s.k0; k < s.k1; ++k) {
                    const uint32_t bar = a_bar, ta = a_tmem, a_done = a_bar + (a_par ? 16 * NA : 8 * NA);
                    wait_peeked(bar, a_par, ready, limit);
                    a_bar += 8;
                    a_tmem += 64;
                    if (a_bar == a_end) {
                        a_bar = a_full;
                        a_tmem = a_first;
                        a_par ^= 1u;
                    }
                    ready = peek(a_bar, a_par);               // of the next unit, while this one's MMAs are issued
                    const bool two = 2 * k + 1 < prm.subs_k;  // (K may be an odd number of blocks)
                    if (bc.blocks > 1) {
                        if (left == 0) {
                            wait_limited(b_full + 8 * st, (par >> st) & 1, limit);
                            par ^= 1u << st;
                            left = min(bc.blocks >> 1, s.k1 - k);
                            bd = desc | (((b_ring + (uint32_t)st * (uint32_t)bc.bytes) & 0x3FFFFu) >> 4);
                        }
                        --left;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (leader) {
                            if (two) mma_unit(d, ta, bd, idesc, acc, sub_step);
                            else mma_block(d, ta, bd, idesc, acc);
                            commit(a_done);
                            if (left == 0) commit(b_empty + 8 * st);
                        }
                        bd += 2 * sub_step;
                        if (left == 0) st = (st + 1 == bc.stages) ? 0 : st + 1;
                    } else {                                  // a stage is one block
                        for (int i = 0; i < (two ? 2 : 1); ++i) {
                            wait_limited(b_full + 8 * st, (par >> st) & 1, limit);
                            par ^= 1u << st;
                            bd = desc | (((b_ring + (uint32_t)st * (uint32_t)bc.bytes) & 0x3FFFFu) >> 4);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            if (leader) {
                                mma_block(d, ta + 32 * i, bd, idesc, i ? 1u : acc);
                                commit(b_empty + 8 * st);
                            }
                            st = (st + 1 == bc.stages) ? 0 : st + 1;
                        }
                        if (leader) commit(a_done);
                    }
                    acc = 1;
                }
                if (leader) commit(acc_full + 8 * (seg & 1));
                ++seg;
            }
        }
        if (limit == 0) sh.failed = 1;
    } else {
        regs_down<REGS_EPI>();
        // =========================== epilogue ===========================
        if (!counted) grid_dependency_wait();
        const int q = warp & 3, g = lane & 7, j4 = lane >> 3;         // TMEM lane 32 q + 8 j4 + g
        const int et = threadIdx.x - WARP_EPI * 32;                   // thread of the epilogue
        const int part = F::part_of(q, g), slot = F::slot_of(q), member = F::member_of(g, j4);
        constexpr int RUN = PARTS * PER;                              // neighbouring output rows of a member in a tile
        unsigned char* epi = base + F::EPI_OFF;
        float* s_scale = reinterpret_cast<float*>(epi + 2 * TILE_BYTES);      // per row of the chunk: factor of the sums,
        float* s_weight = s_scale + GG_MAX_ROWS;                              // routing weight,
        int* s_row = reinterpret_cast<int*>(s_weight + GG_MAX_ROWS);          // output row
        auto epi_sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
        Seg s;
        s.p = 0;
        int at = 0, seg = 0, turn = 0;
        bool ok = true;
        while (next_seg(sh, own, at, units_k, s)) {
            at += s.k1 - s.k0;
            const Problem& pr = sh.pr[s.p];
            const int n = pr.n, cnt = pr.cnt;
            const bool wide = n > 128;
            const int buf = wide ? 0 : seg & 1;
            const bool whole = s.k0 == 0 && s.k1 == units_k;
            const int rows_here = min(n, cnt - s.chunk * n);          // rows of this chunk that exist
            const int list = pr.list0 + s.chunk * n;                  // list entry of the chunk's first row
            const int quad = (MODE == GG_UP) ? s.tile : s.tile / pr.blocks, rho0 = (MODE == GG_UP) ? quad : quad * PARTS;
            const int m0 = (MODE == GG_UP) ? 0 : 16 * (s.tile - quad * pr.blocks);
            const int rho = (MODE == GG_UP) ? s.tile : rho0 + part;
            // what the rows need is fetched while the sums are still being formed
            for (int i = et; i < rows_here; i += 128) {
                s_scale[i] = (pr.f16 ? F16_SCALE : 1.f) * (prm.row_scale ? __ldcg(prm.row_scale + pr.row0 + s.chunk * n + i) : 1.f);
                if (MODE == GG_DOWN) {
                    s_weight[i] = prm.row_w ? __ldcg(prm.row_w + list + i) : 1.f;
                    s_row[i] = prm.out_idx ? __ldcg(prm.out_idx + list + i) : list + i;
                }
            }
            float bias = 0.f;
            if (MODE == GG_LINEAR) {
                const uint16_t* bp = prm.hp[s.p].bias;
                if (bp && rho < pr.P && (!F::WORDS || (m0 + member) * pr.G + PER * rho + slot < pr.N)) bias = bf16_bits_to_float(bp[(m0 + member) * pr.G + PER * rho + slot]);
            }
            // What a thread writes of 16 rows of x, from the buffer in which they change places.
            const int wt = et >> 4, wm = et & 15;                 // rows wt and wt + 8; member
            constexpr int TB_ROW = MODE == GG_UP ? 64 : 128;      // values of a row of x in the buffer
            unsigned char* h_dst = nullptr;
            uint16_t* out = nullptr;
            int64_t ld = 0;
            bool runs = true, exists = true;                      // eight neighbouring outputs in one store; the member has these rows
            if constexpr (MODE == GG_UP) {
                const int col = wm * pr.G + PER * rho;            // four neighbouring columns of h, staged at pos .. pos + 3
                const int pos = tile_pos(col & 63), row = pr.row0 + s.chunk * n + wt;       // (row and row + 8, 16, ... share the swizzle)
                h_dst = prm.ht + ((int64_t)(col >> 6) * prm.xt_rows + row) * 128 + ((((pos >> 3) ^ (row & 7)) << 4) | ((pos & 7) * 2));
            } else {
                ld = (MODE == GG_LINEAR) ? pr.N : prm.N;
                out = reinterpret_cast<uint16_t*>(MODE == GG_LINEAR ? prm.hp[s.p].y : prm.out) + (int64_t)(m0 + wm) * pr.G + PER * rho0;
                exists = !F::WORDS || (m0 + wm) * pr.G + PER * rho0 < pr.N;
                runs = !(MODE == GG_DOWN && prm.accumulate) && pr.P - rho0 >= PARTS && ((reinterpret_cast<uintptr_t>(out) | (uintptr_t)(ld * 2)) & 15) == 0;
                if (MODE == GG_LINEAR) out += (int64_t)(list + wt) * ld;
            }
            const int at0 = MODE == GG_UP ? (lane & 1) * 8 * 64 + member * 4 + (((slot & 1) << 1) | (slot >> 1)) : member * RUN + part * PER + slot;
            epi_sync();                                               // s_scale and the others are complete
            if (!wait(acc_full + 8 * (seg & 1), (seg >> 1) & 1)) ok = false;
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t td = tmem + tmap.d_step * (uint32_t)buf + ((uint32_t)(32 * q) << 16);
            // 16 rows of x of this thread's tile row: asked for, and there
            uint32_t acc[16];
            auto ask = [&](int c0) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(acc[0]), "=r"(acc[1]), "=r"(acc[2]), "=r"(acc[3]), "=r"(acc[4]), "=r"(acc[5]), "=r"(acc[6]), "=r"(acc[7]),
                      "=r"(acc[8]), "=r"(acc[9]), "=r"(acc[10]), "=r"(acc[11]), "=r"(acc[12]), "=r"(acc[13]), "=r"(acc[14]), "=r"(acc[15])
                    : "r"(td + (uint32_t)c0));
            };
            auto have = [&] {
                asm volatile("tcgen05.wait::ld.sync.aligned;"
                             : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]), "+r"(acc[7]),
                               "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]), "+r"(acc[14]), "+r"(acc[15])
                             :
                             : "memory");
            };
            ask(0);
            auto release = [&] {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive(acc_empty + 8 * (seg & 1));
            };
            int c_first = cta, c_last = cta, parts_n = 1;
            bool finish = true;
            if (!whole) {
                // the tile's units are cut over the CTAs c_first .. c_last: leave this CTA's piece, the last one to arrive adds them
                const int t0 = s.u - s.k0;
                while (c_first > 0 && sh.begin[c_first] > t0) --c_first;
                parts_n = 0;
                while (c_last + 1 < grid && sh.begin[c_last + 1] < t0 + units_k) ++c_last;
                for (int c = c_first; c <= c_last; ++c) parts_n += sh.begin[c + 1] > sh.begin[c] ? 1 : 0;
                // [4 rows of x][128 tile rows][4]: a warp writes and reads 512 contiguous bytes at a time
                float4* mine = reinterpret_cast<float4*>(prm.parts) + (size_t)(2 * cta + (s.k0 == 0 ? 1 : 0)) * prm.n_max * 32 + 32 * q + lane;
                for (int c0 = 0; c0 < rows_here; c0 += 16) {
                    have();
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        __stcg(reinterpret_cast<uint4*>(mine) + (size_t)(c0 / 4 + i) * 128, make_uint4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]));
                    if (c0 + 16 < rows_here) ask(c0 + 16);
                }
                release();
                __threadfence();                                      // (by every thread: 0.5 us sooner than one for all of them)
                epi_sync();
                if (et == 0) {
                    const unsigned arrived = atomicAdd(prm.counters + c_first, 1u);
                    if (arrived >= (unsigned)parts_n && prm.error_flag) atomicExch(prm.error_flag, 3);
                    sh.last = arrived == (unsigned)(parts_n - 1);
                    if (sh.last) prm.counters[c_first] = 0u;
                    __threadfence();
                }
                epi_sync();
                finish = sh.last != 0;
            }
            if (finish) {
                // A cut tile: the pieces in CTA order (a CTA without a unit has none), 16 rows at a time.  What this costs is latency,
                // so several are under way; a thread copies what it will read itself, which needs no barrier.
                const uint32_t merge = raw_ring + (uint32_t)(n_raw * F::RAW_BYTES) + 16u * et;
                const int n_merge = F::n_merge(prm.n_max);
                const bool dense = parts_n == c_last - c_first + 1;
                const uint32_t step = (uint32_t)prm.n_max * 32u;      // of a CTA's two pieces
                const float4* fetch_src = reinterpret_cast<const float4*>(prm.parts) + 32 * q + lane;
                int fetch_c = c_first, fetch_r = 0, fetch_at = 0, merge_at = 0;
                auto fetch = [&] {
                    if (fetch_r < rows_here) {
                        const float4* src = fetch_src + (uint32_t)(2 * fetch_c + (fetch_c == c_first ? 1 : 0)) * (size_t)step;
                        const uint32_t dst = merge + (uint32_t)(fetch_at * MERGE_BYTES);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(i * MERGE_BYTES / 4)), "l"(src + i * 128) : "memory");
                        fetch_at = fetch_at + 1 == n_merge ? 0 : fetch_at + 1;
                        ++fetch_c;
                        if (!dense)
                            while (fetch_c <= c_last && sh.begin[fetch_c + 1] <= sh.begin[fetch_c]) ++fetch_c;
                        if (fetch_c > c_last) {
                            fetch_c = c_first;
                            fetch_r += 16;
                            fetch_src += 16 * 32;
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                };
                auto add_pieces = [&](float (&v)[16]) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = 0.f;
#pragma unroll 1
                    for (int c = 0; c < parts_n; ++c) {
                        // the oldest of n_merge groups has arrived
                        if (n_merge == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
                        else if (n_merge == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
                        else asm volatile("cp.async.wait_group 0;" ::: "memory");
                        const uint32_t at = merge + (uint32_t)(merge_at * MERGE_BYTES);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 f = lds128(at + (uint32_t)(i * MERGE_BYTES / 4));
                            v[4 * i] += __uint_as_float(f.x);
                            v[4 * i + 1] += __uint_as_float(f.y);
                            v[4 * i + 2] += __uint_as_float(f.z);
                            v[4 * i + 3] += __uint_as_float(f.w);
                        }
                        merge_at = merge_at + 1 == n_merge ? 0 : merge_at + 1;
                        fetch();
                    }
                };
                if (!whole)
                    for (int i = 0; i < n_merge; ++i) fetch();
#pragma unroll 1
                for (int c0 = 0; c0 < rows_here; c0 += 16) {
                    float v[16];
                    if (whole) {
                        have();
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(acc[i]);
                    } else {
                        add_pieces(v);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 f = *reinterpret_cast<const float4*>(s_scale + c0 + 4 * i);
                        const float ff[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[4 * i + e] *= ff[e];
                    }
                    if (whole) {                                      // the next rows are on their way under this arithmetic
                        if (c0 + 16 < rows_here) ask(c0 + 16);
                        else release();
                    }
                    uint16_t* tb = reinterpret_cast<uint16_t*>(epi + turn * TILE_BYTES) + at0;
                    turn ^= 1;                                        // two buffers: one barrier per 16 rows
                    if constexpr (MODE == GG_UP) {
                        // neighbouring lanes hold the gate (even) and the up (odd) sums of one row of h; each finishes 8 rows of x, two at
                        // a time: packed roundings and products
                        const bool up = (lane & 1) != 0;
                        uint32_t p[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) p[i] = bf2(v[2 * i], v[2 * i + 1]);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t other = __shfl_xor_sync(0xffffffffu, up ? p[i] : p[i + 4], 1);
                            const uint32_t a2 = up ? other : p[i], b2 = up ? p[i + 4] : other;
                            const float a0 = __uint_as_float(a2 << 16), a1 = __uint_as_float(a2 & 0xffff0000u);
                            const uint32_t g2 = bf2(silu(a0), silu(a1));
                            uint32_t h2 = bf2_mul(g2, b2);
                            if (cnt <= GG_F16_ROWS) h2 = h2_of(__uint_as_float(h2 << 16), __uint_as_float(h2 & 0xffff0000u));
                            tb[2 * i * 64] = (uint16_t)h2;            // [row][member][slot in the order 0, 2, 1, 3]
                            tb[(2 * i + 1) * 64] = (uint16_t)(h2 >> 16);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            uint32_t o;
                            if (MODE == GG_LINEAR) {
                                const float y0 = v[2 * i] + bias, y1 = v[2 * i + 1] + bias;
                                o = prm.y_f16 ? h2_of(y0, y1) : bf2(y0, y1);
                            } else {
                                const float2 w = *reinterpret_cast<const float2*>(s_weight + c0 + 2 * i);
                                const uint32_t r = bf2(v[2 * i], v[2 * i + 1]);
                                o = bf2(__uint_as_float(r << 16) * w.x, __uint_as_float(r & 0xffff0000u) * w.y);
                            }
                            tb[2 * i * 128] = (uint16_t)o;
                            tb[(2 * i + 1) * 128] = (uint16_t)(o >> 16);
                        }
                    }
                    epi_sync();
                    const uint16_t* from = reinterpret_cast<const uint16_t*>(epi + (turn ^ 1) * TILE_BYTES) + wt * TB_ROW;
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        const int t = wt + 8 * jj;
                        if (c0 + t >= rows_here || !exists) continue;
                        if constexpr (MODE == GG_UP) {
                            *reinterpret_cast<uint2*>(h_dst + (int64_t)(c0 + 8 * jj) * 128) = *reinterpret_cast<const uint2*>(from + jj * 8 * 64 + wm * 4);
                        } else {
                            const uint16_t* src = from + jj * 8 * 128 + wm * RUN;
                            uint16_t* dst = MODE == GG_DOWN ? out + (int64_t)s_row[c0 + t] * ld : out + (int64_t)(c0 + 8 * jj) * ld;
                            if (runs) {
                                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
                            } else {
                                const int valid = min(PARTS, pr.P - rho0) * PER;      // neighbouring rows that exist
                                const bool add = MODE == GG_DOWN && prm.accumulate;
                                for (int x = 0; x < valid; ++x) dst[x] = add ? float_to_bf16_bits(bf16_bits_to_float(src[x]) + bf16_bits_to_float(dst[x])) : src[x];
                            }
                        }
                    }
                }
            }
            epi_sync();                                               // the row values are replaced by the next run's
            ++seg;
        }
        if (!ok) sh.failed = 1;
    }
    // ---- teardown
    if (sh.failed) {                          // copies may still be in flight towards this CTA's shared memory
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WARP_MMA) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (threadIdx.x == 0 && sh.failed && prm.error_flag) atomicExch(prm.error_flag, 1);
}

// Rows of x -> staged tiles [K / 64][row][64] in fp16: the rows of a chunk are contiguous, columns in tile_pos order,
// 16-byte pieces swizzled by the row as the MMA's shared-memory descriptor expects.  A row is scaled by a power of two
// so that its largest value lies in [16, 32): every bf16 row then fits fp16 without loss (values 2^-18 and more below the
// largest become fp16 denormals), the epilogue multiplies by the inverse.  One CTA per row.
template <bool X_F16>
__global__ void __launch_bounds__(256) gg_stage_kernel(unsigned char* __restrict__ xt, float* __restrict__ row_scale, int64_t xt_rows,
                                                       const uint16_t* __restrict__ x, const int32_t* __restrict__ idx,
                                                       const int32_t* __restrict__ counts, int lists, int K, bool words, GgFew few) {
    __shared__ float s_max[8];
    grid_launch_dependents();
    grid_dependency_wait();
    const int li = blockIdx.x;
    int row = li, few_row = 0, few_cap = 0;           // (of a short list: its first staged row, and how many it has)
    if (counts) {
        int list0 = 0, row0 = 0, e = 0;
        for (; e < lists; ++e) {
            const int c = __ldcg(counts + e), cap = c <= few.most ? (c <= 4 ? (c ? 4 : 0) : 8) : 0;
            if (li < list0 + c) {
                few_cap = cap;
                break;
            }
            list0 += c;
            row0 += GgRows::of(c).padded();
            few_row += cap;
        }
        if (e == lists) return;                       // the lists together are shorter than the grid
        row = few_cap ? li - list0 : row0 + (li - list0);
    }
    const uint16_t* src = x + (int64_t)(idx ? __ldcg(idx + li) : li) * K;
    auto pair = [](uint32_t v, float& lo, float& hi) {
        if (X_F16) {
            lo = half_at(v, 0);
            hi = half_at(v, 1);
        } else {
            lo = __uint_as_float(v << 16);
            hi = __uint_as_float(v & 0xffff0000u);
        }
    };
    float mx = 0.f;
    for (int i = threadIdx.x; i < K / 8; i += 256) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + 8 * i);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo, hi;
            pair(w[j], lo, hi);
            mx = fmaxf(mx, fmaxf(fabsf(lo), fabsf(hi)));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = s_max[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) mx = fmaxf(mx, s_max[w]);
    // 2^(exponent of mx - 4); zero, tiny and infinite rows keep a finite factor
    const int e = min(max((int)(__float_as_uint(mx) >> 23), 30), 250) - 4;
    const float down = __uint_as_float((uint32_t)(254 - e) << 23);
    if (threadIdx.x == 0) (few_cap ? few.scale[li] : row_scale[row]) = __uint_as_float((uint32_t)e << 23);
    if (few_cap && threadIdx.x < 2) few.largest[2 * li + threadIdx.x] = 0u;
    if (few_cap) {
        unsigned char* to = few.data + (size_t)few_row * K * 2;
        for (int i = threadIdx.x; i < K / 8; i += 256) {
            const uint4 v = *reinterpret_cast<const uint4*>(src + 8 * i);
            const uint32_t o[4] = {perm(v.x, v.y, 0x5410u), perm(v.x, v.y, 0x7632u), perm(v.z, v.w, 0x5410u), perm(v.z, v.w, 0x7632u)};
            uint32_t h[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                float lo, hi;
                pair(o[w], lo, hi);
                h[w] = h2_of(lo * down, hi * down);
            }
            *reinterpret_cast<uint4*>(to + few_staged_at(8 * i, row, few_cap)) = make_uint4(h[0], h[1], h[2], h[3]);
        }
        return;
    }
    for (int i = threadIdx.x; i < K / 8; i += 256) {
        const int b = i >> 3, ch = i & 7;
        // piece ch of the staged block: words (thread column 2 (ch & 1), word ch >> 1) and the next thread column
        const int k0 = b * 64 + (words ? 8 * (ch & 1) + 16 * (ch >> 1) : 32 * (ch & 1) + 4 * (ch >> 1));
        const uint2 a = *reinterpret_cast<const uint2*>(src + k0), d = *reinterpret_cast<const uint2*>(src + k0 + (words ? 4 : 16));
        const uint32_t o[4] = {perm(a.x, a.y, 0x5410u), perm(a.x, a.y, 0x7632u), perm(d.x, d.y, 0x5410u), perm(d.x, d.y, 0x7632u)};
        uint32_t h[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            float lo, hi;
            pair(o[w], lo, hi);
            const __half2 v = __floats2half2_rn(lo * down, hi * down);
            h[w] = *reinterpret_cast<const uint32_t*>(&v);
        }
        *reinterpret_cast<uint4*>(xt + ((int64_t)b * xt_rows + row) * 128 + ((ch ^ (row & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

}  // namespace gg

// --------------------------------------------------------------------------- host side
static int gg_sm_count() {
    static int counts[MAX_DEVICES];
    int& c = counts[current_device_slot()];
    if (c == 0) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            sms <= 0)
            sms = 148;
        c = sms > 255 ? 255 : sms;
    }
    return c;
}

bool gg_supported(const hqm_weight* w, int G, int C) {
    if (tma_encode_entry() == nullptr || C < 1 || w->K % 64 != 0 || w->K < 128) return false;
    if (w->nbits != 3) return tensor_maps_ok(w, G);
    if (!meta_uniform(w) || w->group_size % 16 != 0 || G % 8 != 0 || (int64_t)G * w->K >= ((int64_t)1 << 31)) return false;
    // members in whole blocks of 16, or all of them (and the last rows) in one
    const Members3 m = Members3::of(w, G);
    if (m.full < 1 || (m.full + (m.left ? 1 : 0) > 16 && (m.left != 0 || m.full % 16 != 0))) return false;
    auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return a16(w->W_q) && a16(w->scale_q) && a16(w->zero_q) && a16(w->ms_scale) && a16(w->mz_scale) && a16(w->ms_zero) &&
           a16(w->mz_zero);
}

// The kernel multiplies with fp16 weights.  That is no loss where the alternative has 16-bit factors too: the streaming
// kernels up to their row limit, and beyond it the formats whose groups make whole tiles of 128 rows; 3 bit from five
// rows on.  Everything else belongs to the shape-agnostic kernel, which computes in fp32: its results are as exact as bf16
// holds them (1.66e-3 from 64 bits; 1.75e-3 here), and take longer (3 bit 5120 x 4096, 2 to 4 rows: 29 us, 18 here; 4 bit
// g128 4096 x 4096, 5 / 100 rows: 32 / 308, 16 / 22 here).
bool gg_takes(const hqm_weight* w, int G, int C, int64_t M) {
    if (!gg_supported(w, G, C)) return false;
    if (w->nbits == 3) {
        Stream3Plan plan;
        return M > STREAM3_ROWS || gemv_stream3_plan(w, G, C, M, &plan);
    }
    if (M <= STREAM_MAX_ROWS) return gemv_stream_shape_ok(w, G, C);
    const int per = codes_per_word(w->nbits), g = w->group_size;
    const bool format = w->nbits == 2 ? g == 16 || g == 32 : g == 32 || g == 64;
    return format && G / per % (128 / (g * per)) == 0 && C % 4 == 0;
}

static int gg_n_max(int64_t rows) {
    const int64_t n = (rows + 15) / 16 * 16;
    return (int)(n < 16 ? 16 : (n > GG_MAX_ROWS ? GG_MAX_ROWS : n));
}
static size_t gg_piece_bytes(int n) { return (size_t)2 * n * 128 * sizeof(float); }      // of one CTA
size_t gg_scratch_bytes(int n) { return (size_t)gg_sm_count() * gg_piece_bytes(n); }
static int64_t gg_tiles(const hqm_weight* w) {
    if (w->nbits == 3) {
        const Members3 m = Members3::of(w, w->N / w->group_size);
        return (int64_t)m.P3 * 10 / 8 * ((m.full + 15) / 16);
    }
    return (w->N / w->group_size + 7) / 8 * (w->group_size / 16);
}
static int64_t gg_tiles(const hqm_weight* const* ws, int count) {
    int64_t tiles = 0;
    for (int i = 0; i < count; ++i) tiles += gg_tiles(ws[i]);
    return tiles;
}
GgLayout gg_expert_layout(int64_t M) { return GgLayout{GgRows::of((int)M), gg_sm_count(), 0, 0}; }
// Rows per chunk and CTAs of linear layers over the same rows, by what a launch costs in cycles of its longest CTA (fitted to
// 2- and 4-bit layers of 1024 to 14336 outputs with 16 to 500 rows):
//   its units of 128 columns:  850 + 4 n with n rows; beyond 128 rows, with one accumulator, 10 n
//   a finished tile:           400 for every 16 rows
//   a tile cut into p pieces:  5000 until the last CTA has seen that it is the last, and 3000 + 400 (p - 2) for every 16 rows;
//                              twice where shares and tiles are not aligned, as a CTA then holds pieces of two tiles.
//                              4-bit chunks of more than 64 rows have one piece in flight: 1200 (p - 2).  (4-bit 2048 x 9216, 192
//                              rows 31.2 -> 29.9 us, 4096 x 9216, 100 rows 32.0 -> 29.2, 1024 x 9216, 300 rows 29.5 -> 27.9; 3-bit
//                              launches have one as well, but 1024 x 9216, 192 rows 28.4 -> 37.7, as whole tiles are all they have left.)
// Wide chunks dequantise the weights less often; narrow ones give every SM whole tiles, and need less scratch.
GgLayout gg_linear_layout(int64_t M, const hqm_weight* const* ws, int count, size_t bytes) {
    const int64_t tiles = gg_tiles(ws, count), units_k = (ws[0]->K + 127) / 128;
    GgLayout best{};
    int64_t best_cost = INT64_MAX;
    int chunks = 0;
    const int most = ws[0]->nbits == 3 ? 128 : GG_MAX_ROWS;       // (the small ring of a 3-bit launch)
    for (int cap = 16; cap <= most; cap += 16) {
        const GgRows r = GgRows::of((int)M, cap);
        if (r.chunks == chunks) continue;    // the same cut
        chunks = r.chunks;
        const size_t staged = gg_stage_bytes(r.padded(), ws[0]->K, true);
        const int64_t sms = bytes > staged ? std::min<int64_t>(gg_sm_count(), (int64_t)((bytes - staged) / gg_piece_bytes(r.n))) : 0;
        if (sms == 0) {
            if (r.chunks == 1) break;
            continue;
        }
        const int64_t units = tiles * r.chunks * units_k, n16 = r.n / 16, s0 = (units + sms - 1) / sms;
        const int64_t unit = std::max<int64_t>(850 + 4 * r.n, r.n > 128 ? 10 * r.n : 0);
        const int64_t more = ws[0]->nbits == 4 && r.n > 64 ? 1200 : 400;
        auto consider = [&](int64_t share, int64_t pieces, int cuts) {
            const int64_t cost = share * unit + (share + units_k - 1) / units_k * n16 * 400 + cuts * (5000 + n16 * (3000 + more * (pieces - 2)));
            if (cost < best_cost) {
                best_cost = cost;
                best = GgLayout{r, (int)std::min<int64_t>(sms, (units + share - 1) / share), (int)share, cost};
            }
        };
        consider((s0 + units_k - 1) / units_k * units_k, 2, 0);                                  // whole tiles
        for (int64_t d = 2; d <= 8; d *= 2)
            if (units_k % d == 0 && units_k / d >= s0) consider(units_k / d, d, 1);              // tiles in d equal parts
        if (s0 % units_k != 0) consider(s0, s0 > units_k ? 2 : (units_k + s0 - 1) / s0 + 1, 2);  // equal shares of all SMs
        if (r.chunks == 1) break;
    }
    return best;
}

int launch_gg_stage(const GgStaged& to, const void* x, int x_f16, const int32_t* idx, const int32_t* counts, int lists, int64_t rows,
                    int K, int nbits, cudaStream_t st, const GgFew& few) {
    auto kern = x_f16 ? gg::gg_stage_kernel<true> : gg::gg_stage_kernel<false>;
    launch_overlapped(kern, (int)rows, 256, 0, st, (unsigned char*)to.data, to.scale, to.rows, (const uint16_t*)x, idx, counts, lists, K, nbits == 3, few);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

template <int NBITS, int MODE>
static int gg_launch_one(const gg::Params& p, int grid, cudaStream_t st) {
    using F = gg::Fmt<NBITS>;
    auto kern = gg::gg_kernel<NBITS, MODE>;
    static bool attr_done[MAX_DEVICES];
    bool& done = attr_done[current_device_slot()];
    if (!done) {
        HQM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F::MOST));
        done = true;
    }
    launch_overlapped(kern, grid, gg::NTHREADS, F::smem(p.n_max, p.cut != 0), st, p);
    HQM_LAUNCH_CHECK();
    return HQM_OK;
}

int launch_gg(const GgJob& job, uint32_t* counters, void* scratch, size_t scratch_bytes, cudaStream_t st) {
    gg::Params p{};
    const int host_problems = job.table ? 1 : job.problems;
    const hqm_weight* first = job.table ? job.shape : job.w0[0];
    const int nbits = first->nbits, gs = first->group_size, per = nbits == 3 ? 4 : codes_per_word(nbits);
    const int parts = 8 / per;
    HQM_CHECK_ARG(job.problems >= 1 && job.problems <= GG_MAX_PROBLEMS && host_problems <= 4, "gemm: %d problems in a launch", job.problems);
    HQM_CHECK_ARG(job.mode != GG_UP || (parts == 2 && gs == 16), "gemm: the fused gate needs 2-bit layers with groups of 16");
    int64_t tiles_all = 0;
    for (int i = 0; i < host_problems; ++i) {
        gg::HostProblem& h = p.hp[i];
        for (int l = 0; l < 2; ++l) {
            const hqm_weight* w = job.table ? job.shape : (l && job.mode == GG_UP ? job.w1[i] : job.w0[i]);
            int G, C;
            const int rc = check_weight(w, &G, &C);
            if (rc != HQM_OK) return rc;
            h.G = G;
            h.C = C;
            h.P = G / per;
            h.N = w->N;
            h.blocks = gs / 16;
            h.tiles = job.mode == GG_UP ? h.P : (h.P + parts - 1) / parts * h.blocks;
            if (nbits == 3) {
                const Members3 m = Members3::of(w, G);
                h.R = G;
                h.G = 10 * m.P3;
                h.P = h.G / per;
                h.full = m.full;
                h.left = m.left;
                h.blocks = (m.full + 15) / 16;
                h.tiles = h.G / 8 * h.blocks;
                if (l == 0 && !stream_cached_maps3(w, G, m, h.maps[0])) {
                    set_error("gemm: cuTensorMapEncodeTiled failed for a %dx%d 3-bit layer", w->N, w->K);
                    return HQM_ERR_CUDA;
                }
            }
            if (!job.table) {
                h.meta[l][0] = w->ms_scale;
                h.meta[l][1] = w->mz_scale;
                h.meta[l][2] = w->ms_zero;
                h.meta[l][3] = w->mz_zero;
                if (nbits != 3 && (l == 0 || job.mode == GG_UP) && !stream_cached_maps(w, G, h.maps[l])) {
                    set_error("gemm: cuTensorMapEncodeTiled failed for a %dx%d %d-bit layer", w->N, w->K, w->nbits);
                    return HQM_ERR_CUDA;
                }
            }
        }
        h.y = job.y[i];
        h.bias = job.bias[i];
        tiles_all += h.tiles;
    }
    if (job.table) tiles_all *= job.problems;
    p.problems = job.problems;
    p.K = first->K;
    p.subs_k = p.K / 64;
    p.units_k = (p.subs_k + 1) / 2;
    p.N = first->N;
    p.table = job.table;
    p.which0 = job.which0;
    p.which1 = job.which1;
    p.counts = job.counts;
    p.rows = job.rows;
    p.few = job.few;
    p.xt = (const unsigned char*)job.x.data;
    p.row_scale = job.x.scale;
    p.xt_rows = job.x.rows;
    p.y_f16 = job.y_f16;
    p.ht = (unsigned char*)job.ht;
    p.out = job.out;
    p.out_idx = job.out_idx;
    p.row_w = job.row_w;
    p.accumulate = job.accumulate;
    p.parts = (float*)scratch;
    p.n_max = job.counts ? gg_n_max(job.rows) : job.layout.rows.n;
    p.chunks = job.layout.rows.chunks;
    p.share = job.counts ? 0 : job.layout.share;
    p.cut = p.share == 0 || p.share % p.units_k != 0;
    p.counters = counters;
    p.error_flag = tc_error_ptr();
    const int grid = job.counts ? gg_sm_count() : job.layout.grid;
    const size_t need = (size_t)grid * gg_piece_bytes(p.n_max);
    if (scratch == nullptr || counters == nullptr || scratch_bytes < need) {
        set_error("gemm: scratch of %zu bytes given, %zu needed", scratch_bytes, need);
        return HQM_ERR_SCRATCH;
    }
#define HQM_GG(B, M) \
    if (nbits == B && job.mode == M) return gg_launch_one<B, M>(p, grid, st);
    HQM_GG(2, GG_LINEAR) HQM_GG(2, GG_UP) HQM_GG(2, GG_DOWN) HQM_GG(4, GG_LINEAR)
    HQM_GG(3, GG_LINEAR)
#undef HQM_GG
    set_error("gemm: no kernel for nbits=%d group_size=%d mode=%d", nbits, gs, (int)job.mode);
    return HQM_ERR_ARG;
}

}  // namespace hqm
