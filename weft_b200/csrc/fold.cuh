// mul_mat for batches of tokens on tcgen05 with the weights as the operand in TENSOR MEMORY.
//
// D[128 weight rows, Nt tokens] += A[128, 256] * B[256, Nt] per 256-element block, kind::f16 with fp32 accumulators.  The A
// operand is the block's integers with the sub-block scales multiplied in, B the activation codes as f16.  One scale pair per
// (row, block) and one per (token, block) is left for the epilogue: acc += x.d * (d * S - dmin * M).
//
// S is an integer, and every accumulator holds its part of it exactly, whatever the order of its terms: operands are cut so that
// no partial sum passes 2^24 (times the power of two that all terms share), with codes up to 128 and every bit of a record set.
//   Q4_K  scale * (q - 8), at most 504 * 128 * 256 in all.  8 * sum(scale * sum of the group's codes), what the centre left
//         out, follows as one K = 16 step, the only one that may round (sums beyond 2^24, by at most 2^-23)
//   Q5_K  scale * (low nibble - 8) in one accumulator; 16 * scale * (fifth bit), multiples of 16, and the centre's step in another
//   Q6_K  16 * (scale / 16) * (q - 32), multiples of 16, in one accumulator, (scale % 16) * (q - 32) in another
// S of two accumulators is their sum, rounded once, as the conversion of an exact integer would be.  (Scales times whole codes
// in one accumulator reach 3.1e7, 6.4e7 and 1.3e8: a block whose terms cancel lost its low bits on the way.)
//
// Why this split.  A weight row is a TMEM lane and a thread: it reads its record, unpacks it in registers and writes it to
// tensor memory with tcgen05.st -- no transposition, no swizzle, no shared-memory round trip, and shared memory (128 bytes a
// clock, the limit of a 128 x 128 f16 tile that reads both operands from it) carries the tokens only.  fp32 accumulators
// need no integer conversion and are overwritten by the next block's first MMA, so the epilogue is one load and three packed
// operations per pair of values.
//
// A CTA takes up to 128 tokens: an MMA with A in tensor memory runs at N / 2 clocks (measured from N = 32 to 128, both operands
// in shared memory: 32 + N / 4) but takes 15 to 25 clocks to issue, so the tokens go into one wide MMA per K step, and one
// expansion of the weights, the largest part of the instructions, serves them all.  Tensor memory (512 columns of 32 bits) bounds
// the rest.  Q4_K: S twice (a block's is read while the next one is summed), M once, A for one block up to 128 tokens, for two up
// to 80.  Two limbs: one set of accumulators above 64 (Q5_K: 48) tokens; its first 64 tokens are completed, and read, before the
// others, so that the reading runs beside the MMAs of the last and of the first A buffer of a block (Q6_K 512 x 4096 x 14336 with
// the set as a whole 160 us, in halves 153, with two sets, which the accumulators no longer leave room for, 137).
// A passes from the expanders to the MMAs in half blocks (Q4_K) or quarter blocks of two operands, the
// quarters being unpacked in registers before the buffer is waited for: 180 to 136 us for Q6_K, 512 x 4096 x 14336; Q4_K, with
// half the MMAs between two hand-overs, lost more to the MMA warp's waits (about 150 clocks each) than it gained.
//
// Roles (28 warps): 16 expanders in four groups that take the blocks in turn (a warp alone issues every four to seven clocks:
// with two groups a Q4_K block took 1900 clocks and a Q6_K block 4700), 8 epilogue warps (lane quarter x every other eight
// tokens), a warp each for the token copies, the weight records and the MMAs.  The records come by TMA.  Rows of Q6_K
// (210 bytes per record) start at any even address; eight rows together are a multiple of 16 bytes, so the matrix is taken as
// super-rows of eight, and row j of each by a box whose columns start at the 16-byte boundary before the record: eight boxes of
// 16 x 240 bytes per block, read with 128-bit loads and a per-thread shift.  Tensor-memory lane l then holds row
// 8 (l % 16) + l / 16 of the tile.  The warps that issue copies and MMAs run as a whole with warp-uniform operands and elect a
// lane for the instruction only: issued from a divergent lane, each operand of each MMA moves to the uniform registers on its
// own, about 100 clocks per instruction.  Few
// tiles: a cluster of CTAs shares a tile, each with a slice of K; the partial sums meet through distributed shared memory in
// rank order.
//
// What bounds it: the hand-overs of A (expanders, MMAs, expanders) and the instructions of the unpacking, 1750 clocks a Q4_K
// block up to 64 tokens and 2500 with 128 against 1088 of tensor work, 5000 against 2048 (Q5_K 2176) for two limbs.  Measured on
// B200 (us, device time with the kernel that makes the planes; before: register tiles, for Q4_K above 128 tokens CTA pairs on int8
// limbs):
//   Q4_K  128 x 4096 x 4096 27.5 -> 18.5   512 x 4096 x 4096 46.8 -> 32.8   512 x 14336 x 4096 110 -> 86   512 x 4096 x 14336 127 -> 86
//   Q5_K  512 x 14336 x 4096 218 -> 149    512 x 4096 x 14336 228 -> 161
//   Q6_K  512 x 14336 x 4096 329 -> 144    512 x 4096 x 14336 338 -> 153
#pragma once

#include "prefill_common.cuh"
#include "kernels.h"

#include <algorithm>
#include <atomic>
#include <type_traits>

namespace weft {

constexpr int FD_WARPS = 28, FD_THREADS = FD_WARPS * 32, FD_ROWS = 128;
constexpr int FD_GROUPS = 4, FD_E_WARP0 = 4 * FD_GROUPS, FD_TMA_WARP = 24, FD_W_WARP = 25, FD_MMA_WARP = 26;
constexpr int FD_TOKENS = 128, FD_AMIN = 4;      // most tokens of a tile; slots of the min term's A operand
constexpr int FD_HALF = 64;                     // tokens of the first half where one set of accumulators is filled and drained in halves
constexpr int FD_W_SLOTS = 4;                   // most blocks of weight records
constexpr int FD_SMEM = 227 * 1024;
constexpr int FD_B_MAX = 6, FD_SLOTS = 8;      // most half-block stages of tokens; slots of the x.d ring
constexpr int FD_DD_SLOTS = 4;
// Registers a thread: at launch, and after the roles have traded (setmaxnreg).  The trade stays inside what the CTA got.
constexpr int FD_REGS = 72, FD_X_REGS = 64, FD_E_REGS = 104, FD_IO_REGS = 40;
static_assert(FD_GROUPS * 128 * FD_X_REGS + 256 * FD_E_REGS + 128 * FD_IO_REGS <= FD_THREADS * FD_REGS, "setmaxnreg would wait for ever");

template <int FMT> struct FoldFormat {
    static constexpr int UNIT = unit_bytes(FMT);
    static constexpr bool MINS = FMT == F_Q4_K || FMT == F_Q5_K;
    static constexpr int LIMBS = FMT == F_Q4_K ? 1 : 2;             // operands of a weight, each with an accumulator of its own
    static constexpr bool SHIFTED = UNIT % 16 != 0;                 // records at any even address: a window of whole 16-byte pieces
    static constexpr int PITCH = SHIFTED ? ((UNIT + 14 + 15) / 16 | 1) * 16 : UNIT;   // an odd number of pieces: 128-bit loads of a warp's rows do not conflict
    static constexpr int PER = LIMBS == 2 ? 1 : 2;                  // quarters of a block in an A buffer of 64 columns
    static constexpr int CHUNKS = 4 / PER;                          // A buffers of a block
    // accumulators of nt columns: the limbs, once or twice (sets: a block's are drained while the next one's are filled), and M
    static constexpr int columns(int nt, int sets) { return (sets * LIMBS + (MINS ? 1 : 0)) * nt; }
};
static_assert(FoldFormat<F_Q4_K>::PITCH / 16 % 2 == 1 && FoldFormat<F_Q5_K>::PITCH / 16 % 2 == 1 && FoldFormat<F_Q6_K>::PITCH / 16 % 2 == 1, "rows in different banks");

// row of the tile that tensor-memory lane l holds
template <int FMT> __device__ __forceinline__ int fold_row_of(int l) { return FoldFormat<FMT>::SHIFTED ? 8 * (l & 15) + (l >> 4) : l; }

struct FoldParams {
    const uint8_t *w;
    const float *xd;             // (nb, pitch)
    float *y;
    long long n, ldy, row_bytes, w_bytes, pitch;
    int m, nb, nt;               // tokens, blocks per row, tokens per tile (a multiple of 16)
    int token_tiles, tiles, slices, b_stages, a_buffers, sets;
    int *status;
};

struct FoldControl {
    uint64_t b_full[FD_B_MAX], b_empty[FD_B_MAX], a_full[4], a_empty[4][FD_GROUPS], d_full[2], d_empty[2], xd_full[FD_SLOTS], w_full[FD_GROUPS], w_empty[FD_W_SLOTS];
    uint32_t tmem_base;
    int abort;
};

// Shared memory, in this order; the token stages must lie on 1024-byte boundaries.
template <int FMT> struct FoldLayout {
    using F = FoldFormat<FMT>;
    static constexpr int CONTROL = 1024;
    // wide tiles keep two blocks of records (one per expander group) so that more tokens can be on their way
    static __host__ __device__ constexpr int w_slots(int tt) { return tt > 64 ? 2 : FD_W_SLOTS; }
    // tt: tokens per tile
    static __host__ __device__ constexpr int stage(int tt) { return tt * 256; }
    static __host__ __device__ constexpr int tokens_at() { return CONTROL; }
    static __host__ __device__ constexpr int raw_at(int tt, int stages) { return tokens_at() + stages * stage(tt); }
    static __host__ __device__ constexpr int dd_at(int tt, int stages) { return raw_at(tt, stages) + w_slots(tt) * FD_ROWS * F::PITCH; }
    static __host__ __device__ constexpr int xd_at(int tt, int stages) { return dd_at(tt, stages) + FD_DD_SLOTS * 2 * FD_ROWS * 4; }
    static __host__ __device__ constexpr int xmin_at(int tt, int stages) { return xd_at(tt, stages) + FD_SLOTS * tt * 4; }
    static __host__ __device__ constexpr int amin_at(int tt, int stages) { return xmin_at(tt, stages) + (F::MINS ? 4 * tt * 32 : 0); }
    // A operands over the sums of 32 codes: FD_AMIN slots for the mins, as many for the scales
    static __host__ __device__ constexpr int bytes(int tt, int stages) { return amin_at(tt, stages) + (F::MINS ? 2 * FD_AMIN * 4096 : 0); }
};

// ------------------------------------------------------------------ instructions

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
          "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
          "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// (a & b) | c as one instruction: with two of the three operands constant the compiler makes it two
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// small unsigned integer (< 1024) as an f16 pair of twice the same value
__device__ __forceinline__ uint32_t small_half2(uint32_t v) { return hadd2(0x64006400u | v | (v << 16), 0xe400e400u); }
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}

// Bounded wait of one thread or a whole warp.  Gives up when another role has, or after the limit; then every role leaves.
__device__ __forceinline__ bool fd_wait(uint64_t *bar, uint32_t parity, FoldControl *ctl, int *status) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 63u && *reinterpret_cast<volatile int *>(&ctl->abort)) return false;
    }
    *reinterpret_cast<volatile int *>(&ctl->abort) = 1;
    report(status, ST_WAIT_TIMEOUT);
    return false;
}

// ------------------------------------------------------------------ unpacking: a quarter of a block (64 elements) of one row
// Word i of the result holds elements {0, 2} (even i) or {1, 3} (odd i) of the i / 2 -th group of four: the order of the
// activation plane.  Q4_K and Q5_K: a code's bits where they lie are an f16 below the normal range, q * 2^-24 (high nibbles
// q * 2^-20); one multiply-add applies the scale and the centre: q * 2^-24 * (scale * 2^10) - 8 * scale * 2^-14, exactly.
// Q6_K: set under the exponent of 1024, the 1024 and the 32 taken out again.

template <int FMT>
struct FoldRow {
    uint32_t exponent;           // 0x64006400 in a register
    const uint8_t *p;            // the record in shared memory (SHIFTED: its window)
    uint32_t skip, select;       // SHIFTED: words of the window before the record, and the byte permute that moves halves into place

    // SHIFTED: four words from byte 16 * piece of the record
    __device__ __forceinline__ void words4(int piece, uint32_t (&out)[4]) const {
        const uint4 a = *reinterpret_cast<const uint4 *>(p + 16 * piece), b = *reinterpret_cast<const uint4 *>(p + 16 * piece + 16);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t t[7], u[5];
#pragma unroll
        for (int i = 0; i < 7; ++i) t[i] = skip & 1u ? w[i + 1] : w[i];
#pragma unroll
        for (int i = 0; i < 5; ++i) u[i] = skip & 2u ? t[i + 2] : t[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) out[i] = __byte_perm(u[i], u[i + 1], select);
    }
};

// the 6-bit scales of a Q4_K / Q5_K record, four to a word: [0] scales 0..3, [1] 4..7; mins alike
template <int FMT> struct FoldScales { uint32_t sc[FMT == F_Q6_K ? 4 : 2], mn[2]; };   // Q6_K: sixteen int8 scales

// The scales of quarter q's two groups and what centres their codes, as f16 pairs
template <int FMT>
struct FoldQuarterScales {
    uint32_t slo, shi, clo, chi;
    __device__ __forceinline__ FoldQuarterScales(int q, const FoldScales<FMT> &s) {
        const uint32_t scales = (q & 2 ? s.sc[1] : s.sc[0]) >> (16 * (q & 1));
        const uint32_t lo = small_half2(scales & 255u), hi = small_half2((scales >> 8) & 255u);
        slo = hmul2(lo, 0x64006400u);                  // * 2^10
        shi = hmul2(hi, 0x54005400u);                  // * 2^6: high nibbles stay where they are
        clo = hmul2(lo, 0x90009000u);                  // * -2^-11
        chi = hmul2(hi, 0x90009000u);
    }
};

// Q4_K: (q - 8) * scale * 2^-14.  Q5_K: the five bits of a code in place, for both limbs.
template <int FMT>
__device__ __forceinline__ void fold_quarter(int q, const FoldRow<FMT> &row, const FoldQuarterScales<FMT> &s, uint32_t (&out)[32]) {
    const uint8_t *codes = row.p + (FMT == F_Q4_K ? 16 : 48) + 32 * q;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const uint4 q4 = *reinterpret_cast<const uint4 *>(codes + 16 * v);
        const uint32_t w4[4] = {q4.x, q4.y, q4.z, q4.w};
        uint32_t f[4] = {0, 0, 0, 0};
        if constexpr (FMT == F_Q5_K) {                       // fifth bits: bit 2 q of the byte for the low nibbles, 2 q + 1 for the high
            const uint4 h4 = *reinterpret_cast<const uint4 *>(row.p + 16 + 16 * v);
            f[0] = h4.x >> (2 * q); f[1] = h4.y >> (2 * q); f[2] = h4.z >> (2 * q); f[3] = h4.w >> (2 * q);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const uint32_t w = o ? w4[i] >> 8 : w4[i];
                uint32_t &l = out[8 * v + 2 * i + o], &h = out[16 + 8 * v + 2 * i + o];
                l = w & 0x000f000fu;
                h = w & 0x00f000f0u;
                if constexpr (FMT == F_Q5_K) {
                    l = and_or(o ? f[i] >> 4 : f[i] << 4, 0x00100010u, l);
                    h = and_or(o ? f[i] >> 1 : f[i] << 7, 0x01000100u, h);
                } else {
                    l = hfma2(l, s.slo, s.clo);
                    h = hfma2(h, s.shi, s.chi);
                }
            }
    }
}

// Q6_K, quarter (h, c) of a block: of the four 32-element groups of half h the sixteen elements from 16 c on, as q - 32 (the
// scales, one per sixteen, are applied by the caller).  K step g of the quarter is K step 2 g + c of the half.
__device__ __forceinline__ void fold_quarter_q6_k(int h, int c, const FoldRow<F_Q6_K> &row, uint32_t (&v)[32]) {
    uint32_t l0[4], l1[4], top[4];
    row.words4(4 * h + c, l0);
    row.words4(4 * h + 2 + c, l1);
    row.words4(8 + 2 * h + c, top);
#pragma unroll
    for (int g = 0; g < 4; ++g) {                            // low nibbles of l0, of l1, high nibbles of l0, of l1
        const uint32_t (&l)[4] = g & 1 ? l1 : l0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int nibble = 8 * o + (g >= 2 ? 4 : 0), pair = 8 * o + 2 * g - 4;   // shifts right that bring bits to 0 and to 4
                const uint32_t t = pair >= 0 ? top[i] >> pair : top[i] << -pair;
                v[8 * g + 2 * i + o] = hadd2(and_or(t, 0x00300030u, and_or(l[i] >> nibble, 0x000f000fu, row.exponent)), 0xe420e420u);
            }
    }
}

// ------------------------------------------------------------------ the kernel

// The CTA's work: tiles first, first + stride, ..., and of each the blocks [begin, end) of its slice of K.
struct FoldAt {
    int tile, b;
    __device__ __forceinline__ void advance(int begin, int end, int stride) { if (++b == end) { b = begin; tile += stride; } }
};

template <int FMT>
__global__ void __launch_bounds__(FD_THREADS, 1) fold_kernel(const __grid_constant__ FoldParams p, const __grid_constant__ CUtensorMap x_codes, const __grid_constant__ CUtensorMap x_mins,
                                                                const __grid_constant__ CUtensorMap w_rows) {
    using F = FoldFormat<FMT>;
    using L = FoldLayout<FMT>;
    extern __shared__ __align__(1024) uint8_t smem[];
    FoldControl *ctl = reinterpret_cast<FoldControl *>(smem);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int nt = p.nt, stages = p.b_stages, abufs = p.a_buffers, sets = p.sets, halves = sets == 1 && nt > FD_HALF ? 2 : 1, w_slots = L::w_slots(nt), w_shift = w_slots == 4 ? 2 : 1;
    const int slice = (int)blockIdx.x % p.slices, first_tile = (int)blockIdx.x / p.slices, stride = (int)gridDim.x / p.slices;
    const int begin = (int)((long long)p.nb * slice / p.slices), end = (int)((long long)p.nb * (slice + 1) / p.slices);
    const int my_tiles = first_tile < p.tiles ? (p.tiles - first_tile + stride - 1) / stride : 0;
    const int total = my_tiles * (end - begin);
    uint8_t *s_tokens = smem + L::tokens_at(), *s_raw = smem + L::raw_at(nt, stages);
    float *s_dd = reinterpret_cast<float *>(smem + L::dd_at(nt, stages)), *s_xd = reinterpret_cast<float *>(smem + L::xd_at(nt, stages));
    uint8_t *s_xmin = smem + L::xmin_at(nt, stages), *s_amin = smem + L::amin_at(nt, stages);

    if (threadIdx.x == 0) {
        for (int s = 0; s < FD_B_MAX; ++s) { mbar_init(&ctl->b_full[s], 1); mbar_init(&ctl->b_empty[s], 1); }
        for (int s = 0; s < 4; ++s) { mbar_init(&ctl->a_full[s], 4); for (int g = 0; g < FD_GROUPS; ++g) mbar_init(&ctl->a_empty[s][g], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&ctl->d_full[s], 1); mbar_init(&ctl->d_empty[s], 8); }
        for (int s = 0; s < FD_SLOTS; ++s) mbar_init(&ctl->xd_full[s], 1);
        for (int s = 0; s < FD_GROUPS; ++s) mbar_init(&ctl->w_full[s], 1);
        for (int s = 0; s < FD_W_SLOTS; ++s) mbar_init(&ctl->w_empty[s], 4);
        ctl->abort = 0;
        ctl->tmem_base = 0xffffffffu;
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == FD_MMA_WARP) tc::tmem_alloc(&ctl->tmem_base, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    constexpr uint32_t tmem = 0u;                                      // all 512 columns are this CTA's
    const uint32_t a_base = tmem + 512u - 64u * (uint32_t)abufs;      // A buffers of 64 columns at the end, accumulators from 0
    // The expander groups take the blocks in turn and the A buffers hold one or two blocks, so a buffer passes from group to
    // group.  A parity wait cannot tell a phase from the one two before: every (buffer, group) has a release barrier of its own,
    // signalled for the group that fills the buffer next, and every group one for its records.
    const int a_blocks = abufs / F::CHUNKS;             // 0: two buffers, each filled twice in a block of four
    // Parity of the release that chunk c of a block waits for, by the number of releases of its (buffer, group) that came before;
    // the first fill of a buffer needs none.
    auto a_parity = [&](int block, int c) {
        const int group = block % FD_GROUPS;
        return a_blocks ? ((uint32_t)(block / FD_GROUPS) & 1u) ^ (group >= a_blocks ? 0u : 1u) : ((uint32_t)(c >> 1) & 1u) ^ (group == 0 ? 1u : 0u);
    };
    const bool tmem_ok = *reinterpret_cast<volatile uint32_t *>(&ctl->tmem_base) == tmem;
    asm volatile("griddepcontrol.launch_dependents;");

    if (!tmem_ok) {
        if (threadIdx.x == 0) { ctl->abort = 1; report(p.status, ST_TMEM_ALLOC); }
    } else if (warp < FD_E_WARP0) {
        // ------------------------------------------------------------------ expanders
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FD_X_REGS));
        const int group = warp >> 2, quarter = warp & 3;
        FoldAt at{first_tile, begin};
        for (int j = 0; j < group; ++j) at.advance(begin, end, stride);
        const uint32_t lane_base = a_base + ((uint32_t)(quarter * 32) << 16);
        uint32_t exponent;
        asm volatile("mov.u32 %0, 0x64006400;" : "=r"(exponent));
        bool ok = true;
        for (int it = group; it < total && ok; it += FD_GROUPS) {
            const int slot = it & (w_slots - 1);
            if (!fd_wait(&ctl->w_full[group], (uint32_t)(it / FD_GROUPS) & 1u, ctl, p.status)) break;
            FoldRow<FMT> row;
            row.exponent = exponent;
            row.p = s_raw + slot * (FD_ROWS * F::PITCH) + (quarter * 32 + lane) * F::PITCH;
            uint32_t skew = 0;
            if constexpr (F::SHIFTED) {
                const long long r = (long long)(at.tile / p.token_tiles) * FD_ROWS + fold_row_of<FMT>(quarter * 32 + lane);
                skew = (uint32_t)((r & 7) * p.row_bytes + (long long)at.b * F::UNIT) & 15u;
                row.skip = skew >> 2;
                row.select = skew & 2u ? 0x5432 : 0x3210;
                if (r >= (p.n & ~7LL) && r < p.n) {             // rows after the last whole super-row: this thread fetches its record
                    const uint16_t *src = reinterpret_cast<const uint16_t *>(p.w + r * p.row_bytes + (long long)at.b * F::UNIT);
                    uint16_t *dst = reinterpret_cast<uint16_t *>(const_cast<uint8_t *>(row.p) + skew);
                    for (int i = 0; i < F::UNIT / 2; ++i) dst[i] = __ldg(src + i);
                    fence_proxy_async();                        // the next box lands on these bytes
                }
            }
            float *dd = s_dd + (it % FD_DD_SLOTS) * (2 * FD_ROWS) + quarter * 32 + lane;
            FoldScales<FMT> s;
            float d[2];
            if constexpr (F::MINS) {
                const uint4 head = *reinterpret_cast<const uint4 *>(row.p);
                d[0] = half_bits_to_float(head.x) * 16384.0f;           // the operands carry 2^-14
                d[1] = -half_bits_to_float(head.x >> 16);
                const Q4KScales u = q4k_unpack_scales(head.y, head.z, head.w);
                s.sc[0] = u.sc_lo; s.sc[1] = u.sc_hi; s.mn[0] = u.mn_lo; s.mn[1] = u.mn_hi;
            } else {
                d[0] = half_bits_to_float(ld_u16(row.p + skew + 208));
                d[1] = 0.0f;
                row.words4(12, s.sc);
            }
            // One loop body for all quarters: the roles' code has to stay in the instruction caches.  Unrolled by quarters, every
            // instruction took 7 to 19 clocks (Q4_K 1.8 to 2.4 thousand clocks a block, Q6_K 4.7 thousand).
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                const int buf = (it * F::CHUNKS + c / F::PER) & (abufs - 1);
                const uint32_t to = lane_base + (uint32_t)(64 * buf + 32 * (c % F::PER));
                uint32_t v[32];
                if constexpr (FMT == F_Q6_K) fold_quarter_q6_k(c >> 1, c & 1, row, v);
                else fold_quarter<FMT>(c, row, FoldQuarterScales<FMT>(c, s), v);
                if (c % F::PER == 0) {
                    if (!fd_wait(&ctl->a_empty[buf][group], a_parity(it, c / F::PER), ctl, p.status)) { ok = false; break; }
                    tc::fence_after_sync();
                }
                if (c == 0) { dd[0] = d[0]; dd[FD_ROWS] = d[1]; }
                if constexpr (FMT == F_Q6_K) {                  // 16 * (scale / 16) into the first columns, scale % 16 into the others
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const uint32_t sc = ((c & 2 ? s.sc[2 + (g >> 1)] : s.sc[g >> 1]) >> (8 * ((c & 1) + 2 * (g & 1)))) & 255u, e = (sc ^ 0x80u) & 0xf0u;
                        const uint32_t high = hadd2(0x64006400u | e | (e << 16), 0xe480e480u), low = small_half2(sc & 15u);
                        uint32_t part[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) part[i] = hmul2(v[8 * g + i], high);
                        tmem_st8(to + 8 * g, part);
#pragma unroll
                        for (int i = 0; i < 8; ++i) part[i] = hmul2(v[8 * g + i], low);
                        tmem_st8(to + 32 + 8 * g, part);
                    }
                } else if constexpr (FMT == F_Q5_K) {           // the nibble, centred, into the first columns, the fifth bit into the others
                    const FoldQuarterScales<FMT> w(c, s);
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        uint32_t part[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) part[i] = hfma2(v[8 * g + i] & (g < 2 ? 0x000f000fu : 0x00f000f0u), g < 2 ? w.slo : w.shi, g < 2 ? w.clo : w.chi);
                        tmem_st8(to + 8 * g, part);
#pragma unroll
                        for (int i = 0; i < 8; ++i) part[i] = hmul2(v[8 * g + i] & (g < 2 ? 0x00100010u : 0x01000100u), g < 2 ? w.slo : w.shi);
                        tmem_st8(to + 32 + 8 * g, part);
                    }
                } else {
                    tmem_st32(to, v);
                }
                if (F::MINS && c == 3) {             // two 16-byte chunks of a K = 16 operand: {m_0 .. m_7 | 64 m_0 .. 64 m_7}, and 8 * 2^-14 times the scales
                    const uint32_t am = smem_addr(s_amin + (it & (FD_AMIN - 1)) * 4096 + (quarter * 32 + lane) * 16), as = am + FD_AMIN * 4096;
                    uint32_t m[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t w = s.mn[i >> 1] >> (16 * (i & 1));
                        m[i] = hadd2(0x64006400u | (w & 63u) | ((w & 0x3f00u) << 8), 0xe400e400u);
                    }
                    sts_u128(am, m[0], m[1], m[2], m[3]);
                    sts_u128(am + 2048, hmul2(m[0], 0x54005400u), hmul2(m[1], 0x54005400u), hmul2(m[2], 0x54005400u), hmul2(m[3], 0x54005400u));
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t w = s.sc[i >> 1] >> (16 * (i & 1));
                        m[i] = hmul2(hadd2(0x64006400u | (w & 63u) | ((w & 0x3f00u) << 8), 0xe400e400u), 0x10001000u);
                    }
                    sts_u128(as, m[0], m[1], m[2], m[3]);
                    sts_u128(as + 2048, hmul2(m[0], 0x54005400u), hmul2(m[1], 0x54005400u), hmul2(m[2], 0x54005400u), hmul2(m[3], 0x54005400u));
                    fence_proxy_async();
                }
                if (c % F::PER == F::PER - 1) {
                    tc::tmem_st_wait();
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->a_full[buf]);
                }
            }
            __syncwarp();                                       // every lane has read its record
            if (lane == 0) mbar_arrive(&ctl->w_empty[slot]);
            for (int j = 0; j < FD_GROUPS; ++j) at.advance(begin, end, stride);
        }
    } else if (warp < FD_TMA_WARP) {
        // ------------------------------------------------------------------ epilogue: lane = weight row, columns = tokens
        asm volatile("griddepcontrol.wait;" ::: "memory");              // Y may still be read by the kernel before
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FD_E_REGS));
        constexpr int OWN = FD_TOKENS / 2;                              // most tokens of a warp
        float acc[OWN];
        const int quarter = warp & 3, group = (warp - FD_E_WARP0) >> 2;
        const int pieces = nt / 16;                                     // eight tokens each: pieces group, group + 2, ...
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + 8u * (uint32_t)group;
        const int row = quarter * 32 + lane;
        FoldAt at{first_tile, begin};
        bool ok = true;
        int it = 0;
        for (int t = 0; t < my_tiles && ok; ++t) {
#pragma unroll
            for (int i = 0; i < OWN; ++i) acc[i] = 0.0f;
            const int tile = at.tile;
            for (int b = begin; b < end; ++b, ++it, at.advance(begin, end, stride)) {
                const int slot = it % FD_SLOTS, buf = sets == 2 ? it & 1 : 0;
                const uint32_t d_phase = (uint32_t)(sets == 2 ? it >> 1 : it) & 1u;
                const float *xd = s_xd + slot * nt + 8 * group, *dd = s_dd + (it % FD_DD_SLOTS) * (2 * FD_ROWS) + row;
                if (!fd_wait(&ctl->xd_full[slot], (uint32_t)(it / FD_SLOTS) & 1u, ctl, p.status) || !fd_wait(&ctl->d_full[buf], d_phase, ctl, p.status)) { ok = false; break; }
                tc::fence_after_sync();
                const float d0 = dd[0], d1 = dd[FD_ROWS];
                const uint64_t s0 = pack2(d0, d0), s1 = pack2(d1, d1);
                const uint32_t from = lane_base + (uint32_t)(buf * F::LIMBS * nt), from_min = lane_base + (uint32_t)(sets * F::LIMBS * nt);
                // eight columns at a time, the next ones on their way while these are added (two limbs: asked for once
                // d * S - dmin * M of these is formed)
                constexpr int AHEAD = F::LIMBS == 2 ? 1 : 2;
                uint32_t v0[AHEAD][8], v1[AHEAD][8], vm[AHEAD][8];
                auto load = [&](int k) {
                    tc::tmem_ld8(from + (uint32_t)(16 * k), v0[k % AHEAD]);
                    if (F::LIMBS == 2) tc::tmem_ld8(from + (uint32_t)(nt + 16 * k), v1[k % AHEAD]);
                    if (F::MINS) tc::tmem_ld8(from_min + (uint32_t)(16 * k), vm[k % AHEAD]);
                };
                auto pair = [&](const uint32_t (&v)[8], int e) { return pack2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])); };
                auto scaled = [&](int k, int e) {                       // d * S - dmin * M
                    uint64_t sum = pair(v0[k % AHEAD], e);
                    // the limbs' sums are exact; S is their sum, rounded once as the integer would be
                    if constexpr (F::LIMBS == 2) sum = add2(sum, pair(v1[k % AHEAD], e));
                    sum = mul2(s0, sum);
                    if constexpr (F::MINS) sum = fma2(s1, pair(vm[k % AHEAD], e), sum);
                    return sum;
                };
                load(0);
                tc::tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < OWN / 8; ++k) {
                    if (F::LIMBS == 2 && k == FD_HALF / 16 && halves == 2) {
                        if (!fd_wait(&ctl->d_full[1], d_phase, ctl, p.status)) { ok = false; break; }
                        tc::fence_after_sync();
                        load(k);
                        tc::tmem_ld_wait();
                    }
                    const int whole = F::LIMBS == 2 && halves == 2 && k < FD_HALF / 16 ? FD_HALF / 16 : pieces;   // pieces whose accumulators are complete
                    if (k < pieces) {
                        uint64_t v[4];
                        if constexpr (AHEAD == 1) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) v[e] = scaled(k, e);
                        }
                        if (k + 1 < whole) load(k + 1);
#pragma unroll
                        for (int i = 0; i < 8; i += 4) {
                            const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(xd + 16 * k + i);
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int j = i + 2 * e;
                                uint64_t a = pack2(acc[8 * k + j], acc[8 * k + j + 1]);
                                a = fma2(e ? x.y : x.x, AHEAD == 1 ? v[j / 2] : scaled(k, j / 2), a);
                                unpack2(a, acc[8 * k + j], acc[8 * k + j + 1]);
                            }
                        }
                        if (k + 1 < whole) tc::tmem_ld_wait();
                    }
                    // all read: the buffers are free
                    if (k == 0 ? whole <= 2 : k + 2 == whole || (F::LIMBS == 2 && k == FD_HALF / 16 && halves == 2 && whole == k + 1)) {
                        tc::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&ctl->d_empty[F::LIMBS == 2 && halves == 2 && k >= FD_HALF / 16 ? 1 : buf]);
                    }
                }
                if (!ok) break;
            }
            if (!ok) break;
            if (p.slices == 1) {
                const long long n = (long long)(tile / p.token_tiles) * FD_ROWS + fold_row_of<FMT>(row);
                const int t0 = (tile % p.token_tiles) * nt + 8 * group;
                if (n < p.n) {
                    float *y = p.y + n;
#pragma unroll
                    for (int i = 0; i < OWN; ++i) {
                        const int token = t0 + 16 * (i >> 3) + (i & 7);
                        if ((i >> 3) < pieces && token < p.m) y[(long long)token * p.ldy] = acc[i];
                    }
                }
            } else {
                // a slice's sums: [token][row] over the token stages, which nothing reads or fills any more
                float *sums = reinterpret_cast<float *>(s_tokens);
#pragma unroll
                for (int i = 0; i < OWN; ++i)
                    if ((i >> 3) < pieces) sums[(8 * group + 16 * (i >> 3) + (i & 7)) * FD_ROWS + row] = acc[i];
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FD_IO_REGS));
        if (warp == FD_TMA_WARP) {
        // ------------------------------------------------------------------ tokens
        FoldAt at{first_tile, begin};
        asm volatile("griddepcontrol.wait;" ::: "memory");              // the planes come from the kernel before
        int issued = 0, s = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int it = 0; it < total && ok; ++it, at.advance(begin, end, stride)) {
            const int t0 = (at.tile % p.token_tiles) * nt;
            for (int h = 0; h < 2; ++h) {
                if (!fd_wait(&ctl->b_empty[s], phase ^ 1u, ctl, p.status)) { ok = false; break; }
                if (elect_one()) {
                    if (h == 0) {
                        const int slot = it % FD_SLOTS;
                        mbar_expect_tx(&ctl->xd_full[slot], (uint32_t)(nt * 4));
                        bulk_g2s(s_xd + slot * nt, p.xd + (long long)at.b * p.pitch + t0, (uint32_t)nt * 4, &ctl->xd_full[slot]);
                    }
                    uint8_t *stage = s_tokens + s * L::stage(nt);
                    uint64_t *full = &ctl->b_full[s];
                    mbar_expect_tx(full, (uint32_t)(nt * 256 + (F::MINS && h == 1 ? nt * 32 : 0)));
                    tma_load_2d(stage, &x_codes, 256 * at.b + 128 * h, t0, full);
                    tma_load_2d(stage + nt * 128, &x_codes, 256 * at.b + 128 * h + 64, t0, full);
                    if (F::MINS && h == 1) {
                        uint8_t *m = s_xmin + (it & 3) * (nt * 32);
                        tma_load_2d(m, &x_mins, 16 * at.b, t0, full);
                        tma_load_2d(m + nt * 16, &x_mins, 16 * at.b + 8, t0, full);
                    }
                }
                __syncwarp();
                ++issued;
                if (++s == stages) { s = 0; phase ^= 1u; }
            }
        }
        // nothing of ours may land after the CTA has left
        for (int k = max(0, issued - stages); k < issued; ++k) mbar_wait(&ctl->b_full[k % stages], (uint32_t)(k / stages) & 1u, 1u << 20);
        for (int k = max(0, (issued + 1) / 2 - FD_SLOTS); k < (issued + 1) / 2; ++k) mbar_wait(&ctl->xd_full[k % FD_SLOTS], (uint32_t)(k / FD_SLOTS) & 1u, 1u << 20);
        } else if (warp >= FD_MMA_WARP) {
        // ------------------------------------------------------------------ MMA issue
        if (warp == FD_MMA_WARP) {
            const uint32_t idesc = tc::idesc_f16_f32acc(FD_ROWS, nt), slab = (uint32_t)nt * 128u;
            const uint64_t b0 = tc::smem_desc_sw128(smem_addr(s_tokens));
            const uint64_t am0 = tc::smem_desc(smem_addr(s_amin), 2048, 128), xm0 = tc::smem_desc(smem_addr(s_xmin), (uint32_t)nt * 16u, 128);
            bool ok = true;
            int s = 0, buf = 0;
            uint32_t b_phase = 0, a_phase = 0;
            // tokens [n0, n0 + n) of the tile: chunk j of the block's products, and what the block's end adds
            auto products = [&](int j, uint32_t a, uint64_t b, uint32_t d, int n0, uint32_t shape) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    // K steps of the half-block in order; two limbs: the four of a quarter for the one and then the other, a
                    // quarter of Q6_K holding every other step of the half
                    const uint32_t at = F::LIMBS == 1 ? (uint32_t)(k >> 2) * slab + 32u * (k & 3)
                                      : FMT == F_Q6_K ? ((uint32_t)(k & 3) >> 1) * slab + 64u * (k & 1) + 32u * (j & 1)
                                                      : (uint32_t)(j & 1) * slab + 32u * (k & 3);
                    mma_f16_ts(d + (uint32_t)(n0 + (F::LIMBS == 2 && k >= 4 ? nt : 0)), a + (uint32_t)(8 * k), b + (uint64_t)((at + 128u * (uint32_t)n0) >> 4), shape, j | (F::LIMBS == 2 ? k & 3 : k));
                }
            };
            // 8 * scales * sums of the codes, what the centred codes left out: into the last limb
            auto centre = [&](int it, uint32_t d, int n0, uint32_t shape) {
                tc::mma_f16(d + (uint32_t)((F::LIMBS - 1) * nt + n0), am0 + (uint64_t)((FD_AMIN + (it & (FD_AMIN - 1))) * (4096 >> 4)),
                            xm0 + (uint64_t)((uint32_t)((it & 3) * nt * 32 + 16 * n0) >> 4), shape, 1);
            };
            auto minimums = [&](int it, uint32_t dm, int n0, uint32_t shape) {
                tc::mma_f16(dm + (uint32_t)n0, am0 + (uint64_t)((it & (FD_AMIN - 1)) * (4096 >> 4)), xm0 + (uint64_t)((uint32_t)((it & 3) * nt * 32 + 16 * n0) >> 4), shape, 0);
            };
            const uint32_t shape0 = tc::idesc_f16_f32acc(FD_ROWS, FD_HALF), shape1 = tc::idesc_f16_f32acc(FD_ROWS, nt - FD_HALF);
            for (int it = 0; it < total && ok; ++it) {
                const int set = sets == 2 ? it & 1 : 0;
                const uint32_t d = tmem + (uint32_t)(set * F::LIMBS * nt), dm = tmem + (uint32_t)(sets * F::LIMBS * nt), d_phase = ((uint32_t)(sets == 2 ? it >> 1 : it) & 1u) ^ 1u;
                // the accumulators have been read: those of this set (two sets with a min term: at the end of the block before)
                const bool at_end = F::MINS && sets == 2;
                if (!at_end && !fd_wait(&ctl->d_empty[set], d_phase, ctl, p.status)) { ok = false; break; }
#pragma unroll 1
                for (int j = 0; j < F::CHUNKS; ++j) {
                    const bool enters = F::CHUNKS == 2 || (j & 1) == 0, leaves = F::CHUNKS == 2 || (j & 1) == 1;   // a half-block of tokens
                    if ((enters && !fd_wait(&ctl->b_full[s], b_phase, ctl, p.status)) || !fd_wait(&ctl->a_full[buf], a_phase, ctl, p.status)) { ok = false; break; }
                    const uint64_t b = b0 + (uint64_t)((uint32_t)(s * L::stage(nt)) >> 4);
                    const uint32_t a = a_base + 64u * (uint32_t)buf;
                    const bool last = j == F::CHUNKS - 1, split = F::LIMBS == 2 && halves == 2 && (j == 0 || last);
                    tc::fence_after_sync();
                    if (split) {
                        // one set of accumulators: the first half of the tokens is complete, and drained, before the second
                        if (elect_one()) {
                            products(j, a, b, d, 0, shape0);
                            if (last) {
                                if (F::MINS) { centre(it, d, 0, shape0); minimums(it, dm, 0, shape0); }
                                tc::commit(&ctl->d_full[0]);
                            }
                        }
                        __syncwarp();
                        if (j == 0) {
                            if (!fd_wait(&ctl->d_empty[1], d_phase, ctl, p.status)) { ok = false; break; }
                            tc::fence_after_sync();
                        }
                    }
                    if (elect_one()) {
                        if (split) products(j, a, b, d, FD_HALF, shape1);
                        else products(j, a, b, d, 0, idesc);
                        tc::commit(&ctl->a_empty[buf][(it * F::CHUNKS + j + abufs) / F::CHUNKS % FD_GROUPS]);
                        if (leaves) tc::commit(&ctl->b_empty[s]);
                        if (last) {
                            if (F::MINS) {
                                centre(it, d, split ? FD_HALF : 0, split ? shape1 : idesc);
                                if (!at_end) minimums(it, dm, split ? FD_HALF : 0, split ? shape1 : idesc);
                            }
                            if (!at_end) tc::commit(&ctl->d_full[split ? 1 : set]);
                        }
                    }
                    __syncwarp();
                    if (++buf == abufs) { buf = 0; a_phase ^= 1u; }
                    if (leaves && ++s == stages) { s = 0; b_phase ^= 1u; }
                }
                if (at_end && ok) {
                    // M of the block before has been read, and so has its S
                    if (it > 0 && !fd_wait(&ctl->d_empty[(it - 1) & 1], (uint32_t)((it - 1) >> 1) & 1u, ctl, p.status)) { ok = false; break; }
                    tc::fence_after_sync();
                    if (elect_one()) {
                        minimums(it, dm, 0, idesc);
                        tc::commit(&ctl->d_full[set]);
                    }
                    __syncwarp();
                }
            }
            // the last commits have to arrive before the CTA leaves
            if (ok && !*reinterpret_cast<volatile int *>(&ctl->abort)) {
                for (int k = max(0, F::CHUNKS * total - abufs); k < F::CHUNKS * total; ++k) {
                    const int next = k + abufs, block = next / F::CHUNKS;
                    mbar_wait(&ctl->a_empty[k & (abufs - 1)][block % FD_GROUPS], a_parity(block, next % F::CHUNKS), 1u << 20);
                }
                for (int k = max(0, 2 * total - stages); k < 2 * total; ++k) mbar_wait(&ctl->b_empty[k % stages], (uint32_t)(k / stages) & 1u, 1u << 20);
            }
        }
        } else if (warp == FD_W_WARP) {
        // ------------------------------------------------------------------ weight records
        FoldAt at{first_tile, begin};
        int issued = 0;
        for (int it = 0; it < total; ++it, at.advance(begin, end, stride)) {
            const int slot = it & (w_slots - 1), row0 = (at.tile / p.token_tiles) * FD_ROWS;
            if (!fd_wait(&ctl->w_empty[slot], ((uint32_t)(it >> w_shift) & 1u) ^ 1u, ctl, p.status)) break;
            if (elect_one()) {
                uint8_t *to = s_raw + slot * (FD_ROWS * F::PITCH);
                mbar_expect_tx(&ctl->w_full[it % FD_GROUPS], FD_ROWS * F::PITCH);
                if constexpr (F::SHIFTED) {
                    int x = at.b * F::UNIT;                             // byte of the record in the super-row, row by row
#pragma unroll 1
                    for (int j = 0; j < 8; ++j, x += (int)p.row_bytes)
                        tma_load_2d(to + j * (16 * F::PITCH), &w_rows, x & ~15, row0 / 8, &ctl->w_full[it % FD_GROUPS]);
                } else {
                    tma_load_2d(to, &w_rows, at.b * (F::UNIT / 4), row0, &ctl->w_full[it % FD_GROUPS]);
                }
            }
            __syncwarp();
            issued = it + 1;
        }
        for (int k = max(0, issued - FD_GROUPS); k < issued; ++k) mbar_wait(&ctl->w_full[k % FD_GROUPS], (uint32_t)(k / FD_GROUPS) & 1u, 1u << 20);
        }
    }

    tc::fence_before_sync();
    __syncthreads();
    if (p.slices > 1) {
        // ---- the slices' sums of the cluster's one tile, added in rank order
        float *sums = reinterpret_cast<float *>(s_tokens);
        tc::cluster_sync_all();
        const int t0 = (first_tile % p.token_tiles) * nt, live = min(nt, p.m - t0);
        const long long n0 = (long long)(first_tile / p.token_tiles) * FD_ROWS;
        if (first_tile < p.tiles && !ctl->abort)
            for (int i = slice * FD_THREADS + (int)threadIdx.x; i < live * FD_ROWS; i += p.slices * FD_THREADS) {
                const long long n = n0 + fold_row_of<FMT>(i & (FD_ROWS - 1));
                if (n >= p.n) continue;
                float sum = 0.0f;
                for (int r = 0; r < p.slices; ++r) {
                    float v;
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(tc::map_to_cta(smem_addr(sums + i), (uint32_t)r)) : "memory");
                    sum += v;
                }
                p.y[(long long)(t0 + i / FD_ROWS) * p.ldy + n] = sum;
            }
        tc::cluster_sync_all();
    }
    if (warp == FD_MMA_WARP) {
        __syncwarp();
        if (tmem_ok) tc::tmem_free(tmem, 512);
    }
}

// ------------------------------------------------------------------ launch (fold_*.cu instantiate one family each)

struct FoldPlan { int nt, slices, stages, a_buffers, sets; double cost; };

template <int FMT>
int fold_stages(int tt) {
    for (int s = FD_B_MAX; s >= 2; --s)
        if (FoldLayout<FMT>::bytes(tt, s) <= FD_SMEM) return s;
    return 0;
}

constexpr int FD_SMEM_LEAST = 118 * 1024;

// How many clusters of `slices` CTAs, one CTA per SM, the device holds at once (0: unknown).  Clusters stay inside a GPC, whose
// SMs are not a multiple of eight, so it is fewer than SMs / slices, and those that do not fit run in a second round: 512 x 2048
// with 64 tokens took 18.0 us on 16 clusters of eight and 10.7 us where the plan asks for no more than fit.
template <int FMT> int fold_clusters(int slices) {
    static std::atomic<int> known[9];
    int n = known[slices].load(std::memory_order_relaxed);
    if (n) return n < 0 ? 0 : n;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)slices);
    cfg.blockDim = dim3(FD_THREADS);
    cfg.dynamicSmemBytes = FD_SMEM_LEAST;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)slices;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (grant_dynamic_smem(reinterpret_cast<const void *>(fold_kernel<FMT>), FD_SMEM_LEAST) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, fold_kernel<FMT>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    known[slices].store(n > 0 ? n : -1, std::memory_order_relaxed);
    return n;
}

template <int FMT> cudaError_t launch_fold_kernel(const FoldParams &params, const CUtensorMap &codes, const CUtensorMap &mins, const CUtensorMap &rows, int sm_count, cudaStream_t stream) {
    // at least half of an SM's shared memory: a second CTA beside this one would wait for the tensor memory this one holds,
    // and two clusters waiting for each other that way would never end
    const int smem = std::max(FoldLayout<FMT>::bytes(params.nt, params.b_stages), FD_SMEM_LEAST);
    cudaError_t e = grant_dynamic_smem(reinterpret_cast<const void *>(fold_kernel<FMT>), smem);
    if (e == cudaSuccess) e = check_launch_registers(reinterpret_cast<const void *>(fold_kernel<FMT>), FD_REGS);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    const int ctas = params.tiles * params.slices;
    cfg.gridDim = dim3((unsigned)(params.slices > 1 || ctas < sm_count ? ctas : sm_count));
    cfg.blockDim = dim3(FD_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)params.slices;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = params.slices > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, fold_kernel<FMT>, params, codes, mins, rows);
}

#define FD_EACH_FORMAT(DO) DO(F_Q4_K) DO(F_Q5_K) DO(F_Q6_K)

}  // namespace weft
