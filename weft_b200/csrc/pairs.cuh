// mul_mat for larger batches of tokens on tcgen05 with CTA PAIRS and the weights as the operand in TENSOR MEMORY.
//
// D[256 weight rows, chunk of tokens] = A[256, 256] * B[256, chunk] per 256-element block.  A CTA of the pair holds 128 of the rows, a
// row to a tensor-memory lane, and half of every chunk of tokens in shared memory; the even CTA issues the MMAs of both.  What is left
// for the epilogue is one scale pair per (row, block) and one scale per (token, block): acc += x.d * (d * S - dmin * M).
//
// S is an exact integer.  Operands and accumulators by format:
//   Q4_K   f16, fp32.  scale * (q - 8) * 2^-14, at most 504 * 128 * 256 < 2^24 in all; 8 * sum(scale * sum of the group's codes), what
//          the centre left out, follows as one K = 16 step, the only one that may round (sums beyond 2^24, by at most 2^-23)
//   Q5_K   int8, int32.  scale * q as 256 * high + low in an accumulator each; int8 MMAs take half the time of f16 ones and half the
//   Q6_K   bytes of tokens, so two limbs cost what one f16 operand does.  |S| <= 2^27 is put together exactly and rounded once
//   TQ1_0  int8, int32.  The digits minus one, in the order in which a table delivers them (the activation plane follows it)
// M (Q4_K, Q5_K): 6-bit mins times the sums of 32 codes as 64 h + l, one K = 16 f16 step.
// int32 sums become floats by adding the bits of 1.5 * 2^23 and taking that out again: I2F runs at 16 lanes a clock (a TQ1_0 block of 256
// tokens took 2600 clocks with it, 2500 without).
//
// Why this split.  Unpacking is paid once per 256 tokens, and a token tile is read once per 256 rows: with 128 x 128 tiles on single
// CTAs (fold.cuh) both were twice as much.  Tokens go in chunks whose accumulators are 96 or 128 columns; two to three chunks and two blocks
// of A fill the 512 columns, so that MMAs, unpacking of the next block and reading of the last chunk overlap.  The sums of a tile are
// 64 registers in each of 512 threads: what else an epilogue thread holds has to fit beside them.  Registers that setmaxnreg adds serve as
// spill space (a kernel of 28 warps is compiled for the 72 it is launched with), so formats whose unpacking is short run it on four warps,
// 24 in all, which are launched with 80 (Q4_K 512 x 14336 x 4096 77.5 -> 75.5 us).
// An MMA takes 20 to 28 clocks to issue beside the other roles and a commit holds its warp for 200, so two warps take the chunks in turn:
// one waits and commits while the other issues.  Without turns, MMAs of two accumulators alternate and take three times as long.
//
// Tiles that do not divide among the pairs are shared: each pair takes a run of blocks, leaves its sums, and pair_parts_kernel adds them in
// the order of the blocks.  (The pair that completes a tile adding them at once took longer: its code cost the loop over the blocks two moves
// a sum.)
//
// Roles: expanders (four warps, a thread per row; eight for two limbs, half a record each), 16 epilogue warps (lane quarter x quarter of
// the chunk), a warp each for token copies and weight records, two for MMAs.  Records come by TMA.  Rows of formats whose records are no
// multiple of 16 bytes start at any even address; eight rows together are a multiple of 16, so the matrix is taken as super-rows of
// eight, and row j of each by a box whose columns start at the 16-byte boundary before the record.  Up to seven rows after the last whole
// super-row come by a copy each into a place of their own; fetched by the expanders two bytes at a time, every block of their tile waited
// for 3 us and more (Q6_K 45 x 9086 x 12288 104.7 -> 57.5 us, 56 x 14735 x 6144 92.3 -> 51.2, 91 x 15300 x 6400 86.6 -> 58.4).
//
// Q4_0 and Q8_0 have a scale pair per 32 elements: every group of 32 is an accumulator of its own (f16 codes, 2 MMAs, at most 127 * 127 * 32
// < 2^24 and exact), acc += x.d * (d * S) eight times a block, and A goes by half blocks.  The epilogue bounds it: a hand-over and 32
// multiply-adds of two per warp for 128 clocks of MMAs, 700 clocks in all.  Tiles of 256 tokens: 173 us where 128 take 158 (the sums do not fit
// the registers); scales of tokens as f16 in shared memory 201; chunks of 32 to 128 tokens chosen at run time 178; the scales read ahead of the
// waits 162.
//
// What bounds it: instructions and their latency.  A block of 256 tokens takes 3400 (Q4_K), 4500 (Q6_K), 2500 (TQ1_0) clocks against 2304,
// 2048 and 1024 of tensor work; issue slots are 50 to 65 % busy and every barrier operation takes 100 to 250 clocks.
// Measured on B200 (us, device time with the kernels before and behind it; before: fold.cuh, TQ1_0 CTA pairs with the tokens as rows):
//   Q4_K   512 x 14336 x 4096  84.2 -> 66.2    512 x 4096 x 14336  83.4 -> 69.7    512 x 28672 x 8192 274 -> 215
//   Q5_K   512 x 14336 x 4096   146 -> 95.9    512 x 4096 x 14336   159 -> 99.0    128 x 14336 x 4096 50.8 -> 37.1
//   Q6_K   512 x 14336 x 4096   141 -> 76.3    512 x 4096 x 14336   150 -> 78.4    512 x 28672 x 8192 495 -> 244
//   Q8_0   512 x 14336 x 4096   247 -> 146     512 x 4096 x 14336   239 -> 148     128 x 14336 x 4096 71.3 -> 46.9   (before: register tiles)
//   Q4_0   512 x 14336 x 4096   221 -> 143     512 x 4096 x 14336   214 -> 146     128 x 14336 x 4096 63.3 -> 45.7
//   TQ1_0  512 x 14336 x 4096  83.2 -> 57.3    512 x 4096 x 14336  80.8 -> 64.3    512 x 28672 x 8192 217 -> 165
// Every wait is bounded; one that runs out raises a flag in both CTAs, every role leaves its loop, copies and MMAs in flight are waited for,
// tensor memory is freed, and the host sees a status code.  Only this GPU's memory is read or written.
#pragma once

#include "prefill_common.cuh"
#include "kernels.h"

#include <cstddef>

namespace weft {

constexpr int PR_ROWS = 256;      // rows of a tile (both CTAs)
constexpr int PR_E_WARPS = 16, PR_MMA_WARPS = 2;
constexpr int PR_RING = 8;                      // slots of the scales' ring
constexpr int PR_SMEM = 227 * 1024;
constexpr float PR_MAGIC = 12582912.0f;         // 1.5 * 2^23

template <int FMT> struct PairFormat {
    static constexpr int UNIT = unit_bytes(FMT);
    static constexpr bool MINS = FMT == F_Q4_K || FMT == F_Q5_K;
    static constexpr bool GROUPED = FMT == F_Q4_0 || FMT == F_Q8_0;     // a scale pair per 32 elements: an accumulator for each, half blocks in turn
    static constexpr bool I8 = FMT != F_Q4_K && !GROUPED;           // int8 operands and int32 accumulators; else f16 and fp32
    static constexpr int HALVES = GROUPED ? 2 : 1, GROUPS = GROUPED ? 4 : 1;     // rounds through A of a block; accumulations of a round
    static constexpr int LIMBS = FMT == F_Q5_K || FMT == F_Q6_K ? 2 : 1;
    static constexpr bool SHIFTED = UNIT % 16 != 0;                 // records at any even address: a window of whole 16-byte pieces
    static constexpr int PITCH = SHIFTED ? ((UNIT + 14 + 15) / 16 | 1) * 16 : UNIT;   // an odd number of pieces: 128-bit loads of a warp's rows do not conflict
    static constexpr int SUMS = LIMBS + (MINS ? 1 : 0);             // accumulators of a token
    static constexpr int CHUNK = SUMS == 3 ? 32 : 128 / SUMS;       // tokens of a chunk
    static constexpr int TOKENS = GROUPED ? 128 : 256;              // tokens of a tile at most; GROUPED: unpacking is the lesser part, half the sums leave registers free
    static constexpr int OWN = CHUNK / 4;                           // columns of a chunk that an epilogue warp takes
    static constexpr int STEPS = (I8 ? 8 : 16) / (HALVES * GROUPS); // MMAs of an accumulation and limb
    static constexpr int A_COLUMNS = LIMBS * STEPS * GROUPS * 8, A_BUFFERS = 2, SLOTS = (512 - A_BUFFERS * A_COLUMNS) / (SUMS * CHUNK);   // tensor memory: accumulators, then A
    static constexpr int STAGE = CHUNK / 2 * (I8 ? 256 : 512 / HALVES);      // this CTA's tokens of a chunk, a block
    static constexpr int STAGES = GROUPED ? 6 : FMT == F_Q4_K ? 8 : FMT == F_Q5_K ? 24 : FMT == F_Q6_K ? 12 : 6;
    static constexpr int W_SLOTS = FMT == F_TQ1_0 ? 6 : FMT == F_Q8_0 ? 2 : 3;
    // expanders, a thread for half a record or a whole one; epilogue; tokens, records and MMAs
    static constexpr int X_WARPS = LIMBS == 2 ? 8 : 4, WARPS = X_WARPS + PR_E_WARPS + 4, THREADS = 32 * WARPS;
    static constexpr int E_WARP0 = X_WARPS, TOKEN_WARP = E_WARP0 + PR_E_WARPS, W_WARP = TOKEN_WARP + 1, MMA_WARP = TOKEN_WARP + 2;
    // Registers a thread: at launch, and after the roles have traded (setmaxnreg).  The trade stays inside what the CTA got.
    // 24 warps: expanders with 64 and copies and MMAs with 32 take 2 % less than with 56 and 40 (Q8_0, TQ1_0; Q4_K and Q4_0 even).
    static constexpr int REGS = WARPS > 24 ? 72 : 80, X_REGS = WARPS > 24 ? 48 : 64, E_REGS = 96, IO_REGS = WARPS > 24 ? 24 : 32;
    static_assert(32 * (X_WARPS * X_REGS + PR_E_WARPS * E_REGS + 4 * IO_REGS) <= THREADS * REGS, "setmaxnreg would wait for ever");
    static constexpr int AMIN = I8 ? 4096 : 8192;                   // A operands over the sums of 32 codes: the mins, and for centred codes the scales
    static constexpr int TABLE = FMT == F_TQ1_0 ? 256 * 8 * 16 : 0;
    // shared memory
    static constexpr int TOKENS_AT = 1024, XMIN_AT = TOKENS_AT + STAGES * STAGE, RAW_AT = XMIN_AT + (MINS ? STAGES * CHUNK * 16 : 0);
    static constexpr int DD_AT = RAW_AT + W_SLOTS * 128 * PITCH, XD_AT = DD_AT + PR_RING * (MINS ? 2 : GROUPS) * 128 * 4;
    static constexpr int AMIN_AT = XD_AT + PR_RING * GROUPS * TOKENS * 4, TABLE_AT = AMIN_AT + (MINS ? A_BUFFERS * AMIN : 0), TAIL_AT = TABLE_AT + TABLE;
    static constexpr int TAIL = SHIFTED ? 7 * PITCH : 0, BYTES = TAIL_AT + W_SLOTS * TAIL;       // rows after the last whole super-row, a slot
    static_assert(BYTES <= PR_SMEM && STAGE % 1024 == 0 && RAW_AT % 128 == 0 && TABLE_AT % 128 == 0, "shared memory");
};

struct PairParams {
    const uint8_t *w;
    const uint32_t *powers;      // TQ1_0
    const float *xd;             // (nb, or eight times that, pitch)
    float *y;
    ulonglong2 *parts;           // sums of the parts of tiles that pairs share: two slots a pair
    long long n, ldy, row_bytes, pitch;
    int m, nb, chunks, token_tiles;
    int pairs, rounds, rest;     // every pair has `rounds` whole tiles; the blocks of the `rest` last tiles are shared out in units
    int unit, per, extra;        // (a block, or a tile's): `per` to a pair, one more to the first `extra` pairs
    bool share;                  // units are blocks: tiles may be shared, and their parts are added behind
    int most_blocks;             // that the record warp fetches before it gives up
    int *status;
    __device__ __forceinline__ int start_of(int pair) const { return (pair * per + min(pair, extra)) * unit; }
    __device__ __forceinline__ int pair_of(int block) const {   // where tiles are shared
        const int longer = extra * (per + 1);
        return block < longer ? block / (per + 1) : extra + (block - longer) / per;
    }
};

struct PairControl {
    uint64_t b_full[24], b_empty[24], a_full[4], a_empty[4], d_full[4], d_empty[4], scales_full[PR_RING], scales_empty[PR_RING], w_full[6], w_empty[6], turn[PR_MMA_WARPS], settled;
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(PairControl) <= 1024, "control block");

// ------------------------------------------------------------------ instructions

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// Columns of tensor memory as packed pairs, eight of two accumulators or sixteen of one.  The pairs are formed behind the wait and inside
// the asm, where no move comes of it.
__device__ __forceinline__ void tmem_pairs(uint32_t a, uint32_t b, uint64_t (&v)[4], uint64_t (&u)[4]) {
    asm volatile("{\n\t.reg .b32 s<8>, t<8>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {s0,s1,s2,s3,s4,s5,s6,s7}, [%8];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {t0,t1,t2,t3,t4,t5,t6,t7}, [%9];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {s0,s1};\n\t"
                 "mov.b64 %1, {s2,s3};\n\t"
                 "mov.b64 %2, {s4,s5};\n\t"
                 "mov.b64 %3, {s6,s7};\n\t"
                 "mov.b64 %4, {t0,t1};\n\t"
                 "mov.b64 %5, {t2,t3};\n\t"
                 "mov.b64 %6, {t4,t5};\n\t"
                 "mov.b64 %7, {t6,t7};\n\t"
                 "}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(u[0]), "=l"(u[1]), "=l"(u[2]), "=l"(u[3]) : "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_pairs(uint32_t a, uint32_t b, uint32_t c, uint64_t (&v)[4], uint64_t (&u)[4], uint64_t (&m)[4]) {
    asm volatile("{\n\t.reg .b32 s<8>, t<8>, w<8>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {s0,s1,s2,s3,s4,s5,s6,s7}, [%12];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {t0,t1,t2,t3,t4,t5,t6,t7}, [%13];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {w0,w1,w2,w3,w4,w5,w6,w7}, [%14];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {s0,s1};\n\t"
                 "mov.b64 %1, {s2,s3};\n\t"
                 "mov.b64 %2, {s4,s5};\n\t"
                 "mov.b64 %3, {s6,s7};\n\t"
                 "mov.b64 %4, {t0,t1};\n\t"
                 "mov.b64 %5, {t2,t3};\n\t"
                 "mov.b64 %6, {t4,t5};\n\t"
                 "mov.b64 %7, {t6,t7};\n\t"
                 "mov.b64 %8, {w0,w1};\n\t"
                 "mov.b64 %9, {w2,w3};\n\t"
                 "mov.b64 %10, {w4,w5};\n\t"
                 "mov.b64 %11, {w6,w7};\n\t"
                 "}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(u[0]), "=l"(u[1]), "=l"(u[2]), "=l"(u[3]), "=l"(m[0]), "=l"(m[1]), "=l"(m[2]), "=l"(m[3]) : "r"(a), "r"(b), "r"(c) : "memory");
}
__device__ __forceinline__ void tmem_pairs(uint32_t a, uint64_t (&v)[8]) {
    asm volatile("{\n\t.reg .b32 s<16>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {s0,s1,s2,s3,s4,s5,s6,s7,s8,s9,s10,s11,s12,s13,s14,s15}, [%8];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {s0,s1};\n\t"
                 "mov.b64 %1, {s2,s3};\n\t"
                 "mov.b64 %2, {s4,s5};\n\t"
                 "mov.b64 %3, {s6,s7};\n\t"
                 "mov.b64 %4, {s8,s9};\n\t"
                 "mov.b64 %5, {s10,s11};\n\t"
                 "mov.b64 %6, {s12,s13};\n\t"
                 "mov.b64 %7, {s14,s15};\n\t"
                 "}"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]), "=l"(v[4]), "=l"(v[5]), "=l"(v[6]), "=l"(v[7]) : "r"(a) : "memory");
}
// two integers (of at most 22 bits and a sign) as the floats PR_MAGIC + integer
__device__ __forceinline__ uint64_t as_floats(uint64_t v) {
    uint64_t r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tadd.u32 lo, lo, 0x4b400000;\n\tadd.u32 hi, hi, 0x4b400000;\n\tmov.b64 %0, {lo, hi};\n\t}" : "=l"(r) : "l"(v));
    return r;
}
__device__ __forceinline__ float half_of(uint64_t v, int i) { return __uint_as_float((uint32_t)(v >> (32 * i))); }
// D (+)= A * B of the pair, A in tensor memory
template <bool I8>
__device__ __forceinline__ void pair_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if (I8)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with A in shared memory
__device__ __forceinline__ void pair_mma_f16_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// an arrival on the barrier at this offset in both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void commit_both(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// into this CTA's shared memory, counted by a barrier that may be the partner's
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}

// Barriers by their address in the shared window, found once: by pointer, every use of one works the address out again.
#define PR_BAR(name, i) (bars + (uint32_t)offsetof(PairControl, name) + 8u * (uint32_t)(i))
__device__ __forceinline__ bool pr_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ void pr_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void pr_expect(uint32_t bar, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
// Bounded wait of a whole warp: false when another role, of either CTA, has given up, or after the limit.  What follows a wait is for whole
// warps, so its lanes must not part: those that are about to give up look once more, together, and a phase that another lane has seen
// complete they see so too.  The role leaves, and says so behind its loop (pair_kernel): said here, at every wait, it cost registers (512 x 14336 x
// 4096 Q8_0 160 us, now 146; Q6_K 78.5, now 76.3).
__device__ __forceinline__ bool pr_wait(uint32_t bar, uint32_t parity, uint32_t bars) {
    for (uint32_t left = 1u << 20; left; --left) {
        if (pr_try(bar, parity)) return true;
        if ((left & 7u) == 0u && lds_u32(bars + (uint32_t)offsetof(PairControl, abort))) left = 2u;
    }
    return false;
}
// Waits for the copies that a barrier counts, whichever of its phases they belong to.  Where a role has given up, a phase may lack arrivals and
// never end: `until` (ns) is then long after its copies have landed.
__device__ __forceinline__ void pr_settle(uint32_t bar, uint64_t until) {
    for (uint32_t parity = 0; parity < 2; ++parity) {
        uint64_t now;
        do asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        while (!__all_sync(0xffffffffu, pr_try(bar, parity)) && __any_sync(0xffffffffu, now < until));
    }
}

// ------------------------------------------------------------------ unpacking: half a block (128 elements) of one row

// the tile row (of this CTA's 128) that tensor-memory lane l holds, and where its record lies among the 128 in shared memory
template <int FMT> __device__ __forceinline__ int pair_row_of(int l) { return PairFormat<FMT>::SHIFTED ? (l & ~31) + 8 * (l & 3) + ((l & 31) >> 2) : l; }
template <int FMT> __device__ __forceinline__ int pair_record_of(int l) { return PairFormat<FMT>::SHIFTED ? 16 * ((l & 31) >> 2) + ((l >> 5) << 2) + (l & 3) : l; }

// a window's words from byte 16 * piece of the record on; skip: words of the window before the record, select: the byte permute
// that moves halves into place
struct Window {
    const uint8_t *p;
    uint32_t skip, select;
    // WORDS words from word FIRST (< 4) of the record's piece
    template <int FIRST, int WORDS> __device__ __forceinline__ void words(int piece, uint32_t (&out)[WORDS]) const {
        constexpr int LAST = FIRST + WORDS + 4, PIECES = (LAST + 3) / 4;       // words FIRST .. LAST - 1 of what is read may be needed
        uint32_t w[4 * PIECES];
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const uint4 v = *reinterpret_cast<const uint4 *>(p + 16 * (piece + i));
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
        uint32_t t[WORDS + 3], u[WORDS + 1];
#pragma unroll
        for (int i = 0; i < WORDS + 3; ++i) t[i] = skip & 1u ? w[FIRST + i + 1] : w[FIRST + i];
#pragma unroll
        for (int i = 0; i < WORDS + 1; ++i) u[i] = skip & 2u ? t[i + 2] : t[i];
#pragma unroll
        for (int i = 0; i < WORDS; ++i) out[i] = __byte_perm(u[i], u[i + 1], select);
    }
};

// Q4_K: word i of 32 elements holds elements {0, 2} (even i) or {1, 3} (odd i) of the i / 2 -th group of four, the order of the
// activation plane.  A code's bits where they lie are an f16 below the normal range, q * 2^-24 (high nibbles q * 2^-20); one
// multiply-add applies the scale and the centre: q * 2^-24 * (scale * 2^10) - 8 * scale * 2^-14, exactly.
__device__ __forceinline__ void pair_expand_q4_k(int half, const uint4 (&codes)[4], const Q4KScales &s, uint32_t to) {
    const uint32_t scales4 = half ? s.sc_hi : s.sc_lo;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint32_t scales = scales4 >> (16 * c);
        const uint32_t lo = small_half2(scales & 255u), hi = small_half2((scales >> 8) & 255u);
        const uint32_t slo = hmul2(lo, 0x64006400u), shi = hmul2(hi, 0x54005400u);            // * 2^10, * 2^6
        const uint32_t clo = hmul2(lo, 0x90009000u), chi = hmul2(hi, 0x90009000u);            // * -2^-11
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const uint4 q4 = codes[2 * c + v];
            const uint32_t w4[4] = {q4.x, q4.y, q4.z, q4.w};
            uint32_t l[8], h[8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const uint32_t w = o ? w4[i] >> 8 : w4[i];
                    l[2 * i + o] = hfma2(w & 0x000f000fu, slo, clo);
                    h[2 * i + o] = hfma2(w & 0x00f000f0u, shi, chi);
                }
            tmem_st8(to + 32 * c + 8 * v, l);
            tmem_st8(to + 32 * c + 16 + 8 * v, h);
        }
    }
}

// the 6-bit values of eight groups as the first of two 16-byte chunks of a K = 16 operand, 64 times them as the second
__device__ __forceinline__ void pair_group_operand(uint32_t lo4, uint32_t hi4, uint32_t factor, uint32_t to) {
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t w = (i < 2 ? lo4 : hi4) >> (16 * (i & 1));
        v[i] = hmul2(hadd2(0x64006400u | (w & 63u) | ((w & 0x3f00u) << 8), 0xe400e400u), factor);
    }
    sts_u128(to, v[0], v[1], v[2], v[3]);
    sts_u128(to + 2048, hmul2(v[0], 0x54005400u), hmul2(v[1], 0x54005400u), hmul2(v[2], 0x54005400u), hmul2(v[3], 0x54005400u));
    fence_proxy_async();
}

// Q5_K: scale * q as 256 * high + low, both int8, four consecutive elements to a word.  Two products to a register, each in its 16 bits
// with 128 added; the low bytes are signed after their top bits are flipped back.
__device__ __forceinline__ void pair_expand_q5_k(int half, const uint8_t *record, const Q4KScales &s, uint32_t to) {
    const uint32_t scales4 = half ? s.sc_hi : s.sc_lo;
#pragma unroll 1
    for (int v = 0; v < 4; ++v) {                               // sixteen bytes of codes: 16 (v & 1) on of 64-element piece 2 half + (v >> 1)
        const int shift = 4 * half + 2 * (v >> 1);              // the fifth bits of the piece's low nibbles
        const uint4 q4 = *reinterpret_cast<const uint4 *>(record + 48 + 64 * half + 16 * v), h4 = *reinterpret_cast<const uint4 *>(record + 16 + 16 * (v & 1));
        const uint32_t w4[4] = {q4.x, q4.y, q4.z, q4.w}, f4[4] = {h4.x, h4.y, h4.z, h4.w}, scales = scales4 >> (16 * (v >> 1));
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t scale = (scales >> (8 * g)) & 255u;
            uint32_t low[4], high[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t q = and_or((f4[i] >> (shift + g)) << 4, 0x10101010u, (g ? w4[i] >> 4 : w4[i]) & 0x0f0f0f0fu);
                const uint32_t even = __byte_perm(q, 0u, 0x4240) * scale + 0x00800080u, odd = __byte_perm(q, 0u, 0x4341) * scale + 0x00800080u;
                low[i] = __byte_perm(even, odd, 0x6240) ^ 0x80808080u;
                high[i] = __byte_perm(even, odd, 0x7351);
            }
            const uint32_t at = to + 16 * (v >> 1) + 8 * g + 4 * (v & 1);
            tmem_st4(at, low);
            tmem_st4(at + 64, high);
        }
    }
}

// Q6_K: scale * (q - 32) as 256 * high + low, both int8; four consecutive elements to a word.  Two products to a register, each in
// its 16 bits with 2^15 + 128 added, so that neither borrows; the bytes are the limbs after their top bits are flipped back.
__device__ __forceinline__ void pair_expand_q6_k(int half, const Window &row, const uint32_t (&sc)[2], uint32_t to) {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {                               // elements 16 c on of each of the four groups of 32
        uint32_t l0[4], l1[4], top[4];
        row.words<0, 4>(4 * half + c, l0);
        row.words<0, 4>(4 * half + 2 + c, l1);
        row.words<0, 4>(8 + 2 * half + c, top);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint32_t (&l)[4] = g & 1 ? l1 : l0;
            const int scale = (int)(int8_t)(sc[g >> 1] >> (8 * (c + 2 * (g & 1))));
            const uint32_t offset = (uint32_t)(32768 + 128 - 32 * scale) * 0x10001u;
            uint32_t low[4], high[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t t = g == 0 ? top[i] << 4 : g == 1 ? top[i] << 2 : g == 2 ? top[i] : top[i] >> 2;
                const uint32_t q = and_or(t, 0x30303030u, (g >= 2 ? l[i] >> 4 : l[i]) & 0x0f0f0f0fu);
                const uint32_t even = __byte_perm(q, 0u, 0x4240) * (uint32_t)scale + offset, odd = __byte_perm(q, 0u, 0x4341) * (uint32_t)scale + offset;
                low[i] = __byte_perm(even, odd, 0x6240) ^ 0x80808080u;
                high[i] = __byte_perm(even, odd, 0x7351) ^ 0x80808080u;
            }
            tmem_st4(to + 8 * g + 4 * c, low);
            tmem_st4(to + 64 + 8 * g + 4 * c, high);
        }
    }
}

// TQ1_0: the digits of a byte come from a table (entry v: digits 0..3 minus one, digit 4 minus one) of sixteen copies.  The order
// of a half's 128 terms is the one the table delivers: 24 words with digits 0..3 of the half's bytes, six with the digits 4 of four
// bytes each, two with the digits of the half's qh bytes.
__host__ __device__ constexpr int tq1_element_of(int j, int n) {   // digit n of record byte j (qs 0..47, qh 48..51)
    return j < 32 ? 32 * n + j : j < 48 ? 160 + 16 * n + (j - 32) : 240 + 4 * n + (j - 48);
}
__host__ __device__ constexpr int tq1_operand_element(int k) {
    const int h = k >> 7, w = (k & 127) >> 2, i = k & 3;
    return w < 24 ? tq1_element_of(24 * h + w, i) : w < 30 ? tq1_element_of(24 * h + 4 * (w - 24) + i, 4) : tq1_element_of(48 + 2 * h + (w - 30), i);
}
constexpr bool tq1_operand_order_is_a_permutation() {
    for (int k = 0; k < 256; ++k) {
        const int e = tq1_operand_element(k);
        if (e < 0 || e > 255) return false;
        for (int other = 0; other < k; ++other)
            if (tq1_operand_element(other) == e) return false;
    }
    return true;
}
static_assert(tq1_operand_order_is_a_permutation(), "every element of a block sits at exactly one operand position");
__device__ __forceinline__ void tq1_lookup(uint32_t table, uint32_t word, int i, uint32_t &x, uint32_t &y) {
    const uint32_t at = table + __byte_perm(word, 0u, 0x4440u + (uint32_t)i) * 128u;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(at));      // the table does not change
}
__device__ __forceinline__ void pair_expand_tq1_0(const uint32_t (&w)[6], uint32_t qh, uint32_t table, uint32_t to) {
    uint32_t fifth[8];
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        uint32_t x[8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) tq1_lookup(table, w[2 * g + (i >> 2)], i & 3, x[i], y[i]);
        tmem_st8(to + 8 * g, x);
        fifth[2 * g] = __byte_perm(__byte_perm(y[0], y[1], 0x0040u), __byte_perm(y[2], y[3], 0x0040u), 0x5410u);
        fifth[2 * g + 1] = __byte_perm(__byte_perm(y[4], y[5], 0x0040u), __byte_perm(y[6], y[7], 0x0040u), 0x5410u);
    }
    uint32_t unused;
    tq1_lookup(table, qh, 0, fifth[6], unused);
    tq1_lookup(table, qh, 1, fifth[7], unused);
    tmem_st8(to + 24, fifth);
}

// Codes as f16, in the order of the activation plane: under the exponent of 1024, where their offset comes out again
__device__ __forceinline__ void pair_bytes_f16(uint32_t codes, uint32_t &even, uint32_t &odd) {
    const uint32_t u = codes ^ 0x80808080u;
    even = hadd2(__byte_perm(u, 0x64646464u, 0x4240), 0xe480e480u);
    odd = hadd2(__byte_perm(u, 0x64646464u, 0x4341), 0xe480e480u);
}
// Two groups of 32 lie in `words` words: a scale, the first's codes a half word off, the other's scale, its codes on a word
template <int FMT> struct PairGroups {
    static constexpr int WORDS = 2 * record_bytes(FMT) / 4, CODES = WORDS / 2;     // words of two groups, of a group's codes
    // the scales of groups 4 half .. 4 half + 3
    static __device__ __forceinline__ void scales(int half, const uint8_t *row, float (&d)[4]) {
        const uint8_t *p = row + 8 * WORDS * half;
#pragma unroll
        for (int g = 0; g < 4; ++g) d[g] = half_bits_to_float(ld_u16(p + g * (2 * WORDS)));
    }
    template <int HALF> static __device__ __forceinline__ void expand(const uint8_t *row, uint32_t to) {
        constexpr int FIRST = 2 * WORDS * HALF & ~3, PIECES = (2 * WORDS * (HALF + 1) - FIRST + 3) / 4, SKIP = 2 * WORDS * HALF - FIRST;
        uint32_t w[4 * PIECES];
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const uint4 v = *reinterpret_cast<const uint4 *>(row + 4 * FIRST + 16 * i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint32_t *from = w + SKIP + (g >> 1) * WORDS + (g & 1 ? CODES + 1 : 0);
            uint32_t c[CODES];
#pragma unroll
            for (int i = 0; i < CODES; ++i) c[i] = g & 1 ? from[i] : __byte_perm(from[i], from[i + 1], 0x5432);
            if constexpr (FMT == F_Q8_0) {
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    uint32_t out[8];
#pragma unroll
                    for (int i = 0; i < 4; ++i) pair_bytes_f16(c[4 * v + i], out[2 * i], out[2 * i + 1]);
                    tmem_st8(to + 16 * g + 8 * v, out);
                }
            } else {
                uint32_t lo[8], hi[8];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const uint32_t q = o ? c[i] >> 8 : c[i];
                        lo[2 * i + o] = hadd2(and_or(q, 0x000f000fu, 0x64006400u), 0xe408e408u);
                        hi[2 * i + o] = hfma2(and_or(q, 0x00f000f0u, 0x64006400u), 0x2c002c00u, 0xd480d480u);      // (1024 + 16 v) / 16 - 72
                    }
                tmem_st8(to + 16 * g, lo);
                tmem_st8(to + 16 * g + 8, hi);
            }
        }
    }
};

// What a thread holds of its record between reading and unpacking it
template <int FMT> struct PairRecord;
template <> struct PairRecord<F_Q4_K> {
    float d0, d1;
    Q4KScales s;
    uint4 codes[4];
    __device__ __forceinline__ void read(int half, const Window &row, uint32_t) {
        const uint4 head = *reinterpret_cast<const uint4 *>(row.p);
        d0 = half_bits_to_float(head.x) * 16384.0f;             // the operands carry 2^-14
        d1 = -half_bits_to_float(head.x >> 16);
        s = q4k_unpack_scales(head.y, head.z, head.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) codes[i] = *reinterpret_cast<const uint4 *>(row.p + 16 + 64 * half + 16 * i);
    }
    __device__ __forceinline__ void expand(int half, const Window &, uint32_t, uint32_t to, uint32_t sums_to) const {
        // the min term's operand, and 8 * 2^-14 times the scales for what the centred codes leave out
        pair_group_operand(half ? s.sc_lo : s.mn_lo, half ? s.sc_hi : s.mn_hi, half ? 0x10001000u : 0x3c003c00u, sums_to);
        pair_expand_q4_k(half, codes, s, to);
    }
};
template <> struct PairRecord<F_Q5_K> {
    float d0, d1;
    Q4KScales s;
    __device__ __forceinline__ void read(int, const Window &row, uint32_t) {
        const uint4 head = *reinterpret_cast<const uint4 *>(row.p);
        d0 = half_bits_to_float(head.x);
        d1 = -half_bits_to_float(head.x >> 16);
        s = q4k_unpack_scales(head.y, head.z, head.w);
    }
    __device__ __forceinline__ void expand(int half, const Window &row, uint32_t, uint32_t to, uint32_t sums_to) const {
        if (half == 0) pair_group_operand(s.mn_lo, s.mn_hi, 0x3c003c00u, sums_to);
        pair_expand_q5_k(half, row.p, s, to);
    }
};
template <> struct PairRecord<F_Q6_K> {
    float d0;
    static constexpr float d1 = 0.0f;
    uint32_t sc[2];                                             // eight int8 scales: group g, elements 16 c on: byte 2 g + c
    __device__ __forceinline__ void read(int half, const Window &row, uint32_t skew) {
        d0 = half_bits_to_float(ld_u16(row.p + skew + 208));
        if (half) row.words<2, 2>(12, sc); else row.words<0, 2>(12, sc);
    }
    __device__ __forceinline__ void expand(int half, const Window &row, uint32_t, uint32_t to, uint32_t) const { pair_expand_q6_k(half, row, sc, to); }
};
template <> struct PairRecord<F_TQ1_0> {
    float d0;
    static constexpr float d1 = 0.0f;
    uint32_t w[6], qh;
    __device__ __forceinline__ void read(int half, const Window &row, uint32_t skew) {
        d0 = half_bits_to_float(ld_u16(row.p + skew + 52));
        qh = ld_u16(row.p + skew + 48 + 2 * half);
        if (half) row.words<2, 6>(1, w); else row.words<0, 6>(0, w);
    }
    __device__ __forceinline__ void expand(int, const Window &, uint32_t table, uint32_t to, uint32_t) const { pair_expand_tq1_0(w, qh, table, to); }
};

template <int FMT> struct PairGroupedRecord {
    static constexpr float d0 = 0.0f, d1 = 0.0f;
    const uint8_t *row;
    __device__ __forceinline__ void read(int, const Window &w, uint32_t) { row = w.p; }
    __device__ __forceinline__ void expand(int half, const Window &, uint32_t, uint32_t to, uint32_t) const {
        if (half) PairGroups<FMT>::template expand<1>(row, to); else PairGroups<FMT>::template expand<0>(row, to);
    }
};
template <> struct PairRecord<F_Q4_0> : PairGroupedRecord<F_Q4_0> {};
template <> struct PairRecord<F_Q8_0> : PairGroupedRecord<F_Q8_0> {};

// where lane `lane` of an epilogue warp leaves its sums of a part, 16 bytes every 512
template <int FMT> __device__ __forceinline__ size_t pair_part(int pair, bool began_before, int rank, int e, int lane) {
    return ((size_t)((2 * pair + (began_before ? 0 : 1)) * 2 + rank) * PR_E_WARPS + e) * (PairFormat<FMT>::TOKENS / 16 * 32) + lane;
}

// ------------------------------------------------------------------ the kernel

template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairFormat<FMT>::THREADS, 1)
pair_kernel(const __grid_constant__ PairParams p, const __grid_constant__ CUtensorMap x_codes, const __grid_constant__ CUtensorMap x_mins, const __grid_constant__ CUtensorMap w_rows) {
    using F = PairFormat<FMT>;
    extern __shared__ __align__(1024) uint8_t smem[];
    PairControl *ctl = reinterpret_cast<PairControl *>(smem);
    const uint32_t base = smem_addr(smem), bars = base;                // the control block lies first
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)tc::cluster_ctarank(), pair = (int)blockIdx.x >> 1, chunks = p.chunks;
    // The pair's blocks: of tiles pair, pair + pairs, ... and then of those that are shared
    const int shared_from = p.rounds * p.nb, shared0 = p.start_of(pair), total = shared_from + p.start_of(pair + 1) - shared0;
    const int first_shared = p.rounds * p.pairs + shared0 / p.nb, first_tile = p.rounds ? pair : first_shared, first_b = p.rounds ? 0 : shared0 % p.nb;
    auto advance = [&](int it, int &tile, int &b) {             // from block it to the next
        if (it + 1 == shared_from) { tile = first_shared; b = shared0 % p.nb; }
        else if (++b == p.nb) { b = 0; tile += it < shared_from ? p.pairs : 1; }
    };
    uint8_t *s_raw = smem + F::RAW_AT;
    float *s_dd = reinterpret_cast<float *>(smem + F::DD_AT), *s_xd = reinterpret_cast<float *>(smem + F::XD_AT);
    constexpr int DD = (F::MINS ? 2 : F::GROUPS) * 128, XD = F::GROUPS * F::TOKENS;     // floats of a round in the rings
    if (threadIdx.x == 0) {
        for (int s = 0; s < F::STAGES; ++s) { mbar_init(&ctl->b_full[s], 1); mbar_init(&ctl->b_empty[s], F::GROUPED ? PR_MMA_WARPS : 1); }
        for (int s = 0; s < F::A_BUFFERS; ++s) { mbar_init(&ctl->a_full[s], 2 * F::X_WARPS); mbar_init(&ctl->a_empty[s], PR_MMA_WARPS); }
        for (int s = 0; s < F::SLOTS; ++s) { mbar_init(&ctl->d_full[s], 1); mbar_init(&ctl->d_empty[s], 2 * PR_E_WARPS); }
        for (int s = 0; s < PR_RING; ++s) { mbar_init(&ctl->scales_full[s], 1 + 4); mbar_init(&ctl->scales_empty[s], PR_E_WARPS); }
        for (int s = 0; s < F::W_SLOTS; ++s) { mbar_init(&ctl->w_full[s], 1); mbar_init(&ctl->w_empty[s], F::X_WARPS); }
        for (int s = 0; s < PR_MMA_WARPS; ++s) mbar_init(&ctl->turn[s], 1);
        mbar_init(&ctl->settled, PR_MMA_WARPS);
        ctl->abort = 0;
        ctl->tmem_base = 0xffffffffu;
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == F::MMA_WARP) tc::tmem_alloc(&ctl->tmem_base, 512);
    if constexpr (F::TABLE != 0) {
        for (int v = (int)threadIdx.x; v < 256 * 16; v += F::THREADS) {
            const uint32_t byte = (uint32_t)v >> 4;
            uint32_t digits = 0;
#pragma unroll
            for (int n = 0; n < 4; ++n) digits |= (uint32_t)(tq1_digit(byte, p.powers[n]) & 255) << (8 * n);
            *reinterpret_cast<uint2 *>(smem + F::TABLE_AT + v * 8) = make_uint2(digits, (uint32_t)(tq1_digit(byte, p.powers[4]) & 255));
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();                                            // the partner's barriers are there, and its tensor memory
    tc::fence_after_sync();
    constexpr uint32_t tmem = 0u, a_base = 512u - F::A_BUFFERS * F::A_COLUMNS;                       // all 512 columns are this CTA's: accumulators, then A
    const bool tmem_ok = *reinterpret_cast<volatile uint32_t *>(&ctl->tmem_base) == tmem;
    asm volatile("griddepcontrol.launch_dependents;");
    if (!tmem_ok && threadIdx.x == 0) {                                // the partner's roles leave through their waits
        ctl->abort = 1;
        tc::st_cluster_u32(tc::map_to_cta(smem_addr(&ctl->abort), (uint32_t)rank ^ 1u), 1u);
        report(p.status, ST_TMEM_ALLOC);
    }
    bool ok = tmem_ok;                                                 // of this warp's role

    if (warp < F::E_WARP0) {
        // ------------------------------------------------------------------ expanders: a thread per row, or per half of one
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F::X_REGS));
        const int half = warp >> 2, l = (warp & 3) * 32 + lane;
        const uint32_t lane_base = a_base + ((uint32_t)((warp & 3) * 32) << 16);
        const int row = pair_row_of<FMT>(l), record = pair_record_of<FMT>(l);
        const uint32_t skew0 = (uint32_t)((row & 7) * p.row_bytes);
        const bool tail = (p.n & 7) != 0;
        const uint32_t full_base = tc::map_to_cta(PR_BAR(a_full, 0), 0u);
        const uint32_t table = F::TABLE ? base + F::TABLE_AT + 8u * (lane & 15) : 0u;
        int tile = first_tile, b = first_b, slot = 0, buf = 0;
        uint32_t w_phase = 0, a_phase = 1;
        Window win{nullptr, 0u, 0u};
        PairRecord<FMT> rec;
        auto read = [&]() {
            if (!pr_wait(PR_BAR(w_full, slot), w_phase, bars)) return false;
            const uint8_t *raw = s_raw + slot * (128 * F::PITCH) + record * F::PITCH;
            const uint32_t skew = F::SHIFTED ? (skew0 + (uint32_t)(b * F::UNIT)) & 15u : 0u;
            if (F::SHIFTED && tail) {                           // rows after the last whole super-row lie apart
                const long long r = (long long)(tile / p.token_tiles) * PR_ROWS + 128 * rank + row;
                if (r >= (p.n & ~7LL) && r < p.n) {
                    raw = smem + F::TAIL_AT + slot * F::TAIL + (row & 7) * F::PITCH;
                    if (r == p.n - 1 && b == p.nb - 1) {        // what follows the matrix's last whole 16 bytes: both threads of the row fetch it
                        const uint8_t *src = p.w + r * p.row_bytes + (long long)b * F::UNIT - skew;
                        for (uint32_t i = (skew + F::UNIT) & ~15u; i < skew + F::UNIT; i += 2)
                            *reinterpret_cast<uint16_t *>(const_cast<uint8_t *>(raw) + i) = __ldg(reinterpret_cast<const uint16_t *>(src + i));
                        fence_proxy_async();                    // the next copy lands on these bytes
                    }
                }
            }
            win = Window{raw, skew >> 2, skew & 2u ? 0x5432u : 0x3210u};
            rec.read(half, win, skew);
            return true;
        };
        ok = ok && read();
        if constexpr (F::GROUPED) {                             // a block is two rounds through A
            for (int it = 0; ok && it < total; ++it) {
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const int ring = (2 * it + h) & (PR_RING - 1);      // free without asking, as below
                    float d[4];
                    PairGroups<FMT>::scales(h, win.p, d);
#pragma unroll
                    for (int g = 0; g < 4; ++g) s_dd[ring * DD + g * 128 + l] = d[g];
                    __syncwarp();
                    if (lane == 0) pr_arrive(PR_BAR(scales_full, ring));
                    ok = pr_wait(PR_BAR(a_empty, buf), a_phase, bars);
                    if (!ok) break;
                    tc::fence_after_sync();
                    rec.expand(h, win, 0u, lane_base + (uint32_t)(buf * F::A_COLUMNS), 0u);
                    tc::tmem_st_wait();
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive_cluster(full_base + 8u * (uint32_t)buf);
                    if (++buf == F::A_BUFFERS) { buf = 0; a_phase ^= 1u; }
                }
                if (!ok) break;
                if (lane == 0) pr_arrive(PR_BAR(w_empty, slot));
                if (++slot == F::W_SLOTS) { slot = 0; w_phase ^= 1u; }
                advance(it, tile, b);
                if (it + 1 < total) ok = read();
            }
        } else
        for (int it = 0; ok && it < total; ++it) {
            if (half == 0) {
                // The ring's slot is free without asking: the A buffer of the block before was free, so the block A_BUFFERS before that is
                // multiplied, and the epilogue had read its scales for the chunk SLOTS before then.
                static_assert(PR_RING >= F::A_BUFFERS + 1 + F::SLOTS, "the ring of the scales");
                const int ring = it & (PR_RING - 1);
                s_dd[ring * DD + l] = rec.d0;
                if (F::MINS) s_dd[ring * DD + 128 + l] = rec.d1;
                __syncwarp();
                if (lane == 0) pr_arrive(PR_BAR(scales_full, ring));
            }
            ok = pr_wait(PR_BAR(a_empty, buf), a_phase, bars);
            if (!ok) break;
            tc::fence_after_sync();
#pragma unroll 1
            for (int h = half; h < 2; h += F::X_WARPS / 4) {
                if (h != half) rec.read(h, win, (win.skip << 2) | (win.select == 0x5432u ? 2u : 0u));
                rec.expand(h, win, table, lane_base + (uint32_t)(buf * F::A_COLUMNS) + (uint32_t)h * (F::I8 ? 32u : 64u), base + F::AMIN_AT + (uint32_t)(buf * F::AMIN + h * 4096 + l * 16));
            }
            __syncwarp();                                       // every lane has read its record
            if (lane == 0) pr_arrive(PR_BAR(w_empty, slot));
            if (++slot == F::W_SLOTS) { slot = 0; w_phase ^= 1u; }
            advance(it, tile, b);
            if (F::X_WARPS == 4 && it + 1 < total) ok = read();
            tc::tmem_st_wait();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster(full_base + 8u * (uint32_t)buf);
            if (F::X_WARPS == 8 && it + 1 < total) ok = read();
            if (++buf == F::A_BUFFERS) { buf = 0; a_phase ^= 1u; }
        }
    } else if (warp < F::TOKEN_WARP) {
        // ------------------------------------------------------------------ epilogue: lane = weight row, columns = tokens
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F::E_REGS));
        asm volatile("griddepcontrol.wait;" ::: "memory");              // Y may still be read by the kernel before
        constexpr int OWN = F::OWN, MOST = F::TOKENS / F::CHUNK, SUMS = F::TOKENS / 8;      // chunks of a tile at most; packed sums of a thread
        const int e = warp - F::E_WARP0, part = e >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(part * OWN);
        const uint32_t empty_base = tc::map_to_cta(PR_BAR(d_empty, 0), 0u);
        const float *dd = s_dd + (warp & 3) * 32 + lane, *xd_base = s_xd + part * OWN;
        int tile = first_tile, b = first_b, slot = 0;
        uint32_t d_phase = 0;
        // The loops are nested, and the sums set to zero in front of the inner one only: set to zero inside of it, every pair is
        // moved on every block.
        for (int it = 0; ok && it < total;) {
            uint64_t acc[SUMS];                                         // pairs of neighbouring tokens
#pragma unroll
            for (int i = 0; i < SUMS; ++i) acc[i] = 0;
            const int from_b = b, tile_end = min(it + p.nb - b, total);
            if constexpr (F::GROUPED) {
#pragma unroll 1
                for (int at = 2 * it; at < 2 * tile_end; ++at) {        // half blocks
                    const int ring = at & (PR_RING - 1);
                    if (!pr_wait(PR_BAR(scales_full, ring), (uint32_t)(at / PR_RING) & 1u, bars)) { ok = false; break; }
#pragma unroll
                    for (int c = 0; c < MOST; ++c) {
                        if (c >= chunks) break;
                        const float *xd = xd_base + ring * XD + c * F::CHUNK;
#pragma unroll
                        for (int g = 0; g < F::GROUPS; ++g, xd += F::TOKENS) {
                            ok = pr_wait(PR_BAR(d_full, slot), d_phase, bars);
                            if (!ok) break;
                            tc::fence_after_sync();
                            const uint32_t from = lane_base + (uint32_t)(F::CHUNK * slot);
                            const float d = dd[ring * DD + g * 128];
                            const uint64_t scale = pack2(d, d);
#pragma unroll
                            for (int k = 0; k < OWN / 16; ++k) {
                                uint64_t v[8];
                                tmem_pairs(from + 16 * k, v);
                                if (k == OWN / 16 - 1) {                // all read: the slot is free
                                    tc::fence_before_sync();
                                    __syncwarp();
                                    if (lane == 0) tc::mbar_arrive_cluster(empty_base + 8u * (uint32_t)slot);
                                    if (++slot == F::SLOTS) { slot = 0; d_phase ^= 1u; }
                                }
#pragma unroll
                                for (int j = 0; j < 8; j += 2) {
                                    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(xd + 16 * k + 2 * j);
                                    uint64_t &to = acc[(c * OWN + 16 * k) / 2 + j], &next = acc[(c * OWN + 16 * k) / 2 + j + 1];
                                    to = fma2(x.x, mul2(scale, v[j]), to);
                                    next = fma2(x.y, mul2(scale, v[j + 1]), next);
                                }
                            }
                        }
                        if (!ok) break;
                    }
                    if (!ok) break;
                    __syncwarp();
                    if (lane == 0) pr_arrive(PR_BAR(scales_empty, ring));
                }
            } else
#pragma unroll 1
            for (int at = it; at < tile_end; ++at) {
                const int ring = at & (PR_RING - 1);
                if (!pr_wait(PR_BAR(scales_full, ring), (uint32_t)(at / PR_RING) & 1u, bars)) { ok = false; break; }
                const float d0 = dd[ring * DD], d1 = F::MINS ? dd[ring * DD + 128] : 0.0f;
                const uint64_t s0 = pack2(d0, d0), s1 = pack2(d1, d1);
                const float *xd = xd_base + ring * F::TOKENS;
#pragma unroll
                for (int c = 0; c < MOST; ++c) {
                    if (c >= chunks) break;
                    ok = pr_wait(PR_BAR(d_full, slot), d_phase, bars);
                    if (!ok) break;
                    tc::fence_after_sync();
                    const uint32_t from = lane_base + (uint32_t)(F::SUMS * F::CHUNK * slot);
                    constexpr int BATCH = F::SUMS == 1 ? 16 : 8, PAIRS = BATCH / 2;
#pragma unroll
                    for (int k = 0; k < OWN / BATCH; ++k) {
                        uint64_t v[PAIRS], u[4], m[4];
                        if constexpr (F::SUMS == 3) tmem_pairs(from + BATCH * k, from + F::CHUNK + BATCH * k, from + 2 * F::CHUNK + BATCH * k, v, u, m);
                        else if constexpr (F::SUMS == 2) tmem_pairs(from + BATCH * k, from + F::CHUNK + BATCH * k, v, u);
                        else tmem_pairs(from + BATCH * k, v);
                        if (k == OWN / BATCH - 1) {                     // all read: the slot is free
                            tc::fence_before_sync();
                            __syncwarp();
                            if (lane == 0) tc::mbar_arrive_cluster(empty_base + 8u * (uint32_t)slot);
                            if (++slot == F::SLOTS) { slot = 0; d_phase ^= 1u; }
                        }
#pragma unroll
                        for (int j = 0; j < PAIRS; j += 2) {
                            const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(xd + c * F::CHUNK + BATCH * k + 2 * j);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                uint64_t sum = v[j + h];
                                if constexpr (F::LIMBS == 2) {           // 256 * high is exact, and so is the whole up to the rounding of the sum
                                    sum = mul2(s0, add2(as_floats(sum), fma2(as_floats(u[j + h]), pack2(256.0f, 256.0f), pack2(-257.0f * PR_MAGIC, -257.0f * PR_MAGIC))));
                                    if constexpr (F::MINS) sum = fma2(s1, m[j + h], sum);
                                } else if constexpr (F::I8) {
                                    sum = mul2(s0, add2(as_floats(sum), pack2(-PR_MAGIC, -PR_MAGIC)));
                                } else {
                                    sum = fma2(s1, u[j + h], mul2(s0, sum));
                                }
                                uint64_t &to = acc[(c * OWN + BATCH * k) / 2 + j + h];
                                to = fma2(h ? x.y : x.x, sum, to);
                            }
                        }
                    }
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) pr_arrive(PR_BAR(scales_empty, ring));
            }
            if (!ok) break;
            b += tile_end - it;
            it = tile_end;
            if (from_b == 0 && b == p.nb) {                             // ---- the tile's sums into Y
                const long long n = (long long)(tile / p.token_tiles) * PR_ROWS + 128 * rank + pair_row_of<FMT>((warp & 3) * 32 + lane);
                const int token = (tile % p.token_tiles) * chunks * F::CHUNK + part * OWN, live = n < p.n ? p.m - token : 0;
                float *y = p.y + n + (long long)token * p.ldy;
#pragma unroll
                for (int c = 0; c < MOST; ++c) {
                    if (c >= chunks) break;
#pragma unroll
                    for (int j = 0; j < OWN; ++j) {
                        if (c * F::CHUNK + j < live) *y = half_of(acc[(c * OWN + j) / 2], j & 1);
                        y += p.ldy;
                    }
                    y += (F::CHUNK - OWN) * p.ldy;
                }
            } else {                                                    // ---- this pair's part of them: the first shared tile into slot 0, the second into slot 1
                ulonglong2 *own = p.parts + pair_part<FMT>(pair, shared0 > (tile - p.rounds * p.pairs) * p.nb, rank, e, lane);
#pragma unroll
                for (int i = 0; i < SUMS / 2; ++i) __stcg(own + 32 * i, make_ulonglong2(acc[2 * i], acc[2 * i + 1]));
            }
            if (it == shared_from) { tile = first_shared; b = shared0 % p.nb; }
            else { tile += it < shared_from ? p.pairs : 1; b = 0; }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F::IO_REGS));
        if (warp == F::TOKEN_WARP) {
            // -------------------------------------------------------------- tokens: a chunk a stage
            asm volatile("griddepcontrol.wait;" ::: "memory");          // the planes come from the kernel before
            const uint32_t full_base = tc::map_to_cta(PR_BAR(b_full, 0), 0u);                  // the even CTA's, for the halves of both
            int tile = first_tile, b = first_b, s = 0;
            uint32_t phase = 1;
            for (int it = 0; ok && it < total; ++it) {
                const int t0 = (tile % p.token_tiles) * chunks * F::CHUNK;
                for (int h = 0; ok && h < F::HALVES; ++h) {
                    const int at = F::HALVES * it + h, ring = at & (PR_RING - 1);
                    ok = pr_wait(PR_BAR(scales_empty, ring), ((uint32_t)(at / PR_RING) & 1u) ^ 1u, bars);
                    if (!ok) break;
                    if (elect_one()) {
                        const uint32_t bytes = (uint32_t)(chunks * F::CHUNK * 4);
                        pr_expect(PR_BAR(scales_full, ring), F::GROUPS * bytes);
                        for (int g = 0; g < F::GROUPS; ++g)
                            bulk_g2s(s_xd + ring * XD + g * F::TOKENS, p.xd + (long long)((F::HALVES * b + h) * F::GROUPS + g) * p.pitch + t0, bytes, &ctl->scales_full[ring]);
                    }
                    __syncwarp();
                    for (int c = 0; c < chunks; ++c) {
                        if (!pr_wait(PR_BAR(b_empty, s), phase, bars)) { ok = false; break; }
                        if (elect_one()) {
                            const int token = t0 + c * F::CHUNK + rank * (F::CHUNK / 2);
                            const uint32_t full = full_base + 8u * (uint32_t)s;
                            if (rank == 0) pr_expect(PR_BAR(b_full, s), 2u * (F::STAGE + (F::MINS ? F::CHUNK * 16 : 0)));
                            pair_load_3d(base + F::TOKENS_AT + (uint32_t)(s * F::STAGE), &x_codes, 0, token, F::I8 ? 2 * b : 4 * b + 2 * h, full);
                            if (F::MINS) pair_load_3d(base + F::XMIN_AT + (uint32_t)(s * (F::CHUNK * 16)), &x_mins, 0, token, 2 * b, full);
                        }
                        __syncwarp();
                        if (++s == F::STAGES) { s = 0; phase ^= 1u; }
                    }
                }
                advance(it, tile, b);
            }
        } else if (warp == F::W_WARP) {
            // -------------------------------------------------------------- weight records
            int tile = first_tile, b = first_b, slot = 0;
            uint32_t phase = 1;
            for (int it = 0; ok && it < total; ++it) {
                ok = it < p.most_blocks && pr_wait(PR_BAR(w_empty, slot), phase, bars);
                if (!ok) break;
                if (elect_one()) {
                    uint8_t *to = s_raw + slot * (128 * F::PITCH);
                    const int row0 = (tile / p.token_tiles) * PR_ROWS + 128 * rank;
                    if constexpr (F::SHIFTED) {
                        // The rows after the last whole super-row, where this CTA has them: copies of their windows up to the matrix's last whole 16 bytes
                        const long long whole = p.n & ~7LL;
                        const int rows = whole >= row0 && whole < row0 + 128 ? (int)(p.n - whole) : 0;
                        const int end = (int)p.row_bytes * rows & ~15;
                        int x = b * F::UNIT, bytes = 128 * F::PITCH;    // byte of the record in the super-row, row by row
                        for (int j = 0, at = x; j < rows; ++j, at += (int)p.row_bytes) bytes += min(F::PITCH, end - (at & ~15));
                        pr_expect(PR_BAR(w_full, slot), (uint32_t)bytes);
#pragma unroll 1
                        for (int j = 0; j < 8; ++j, x += (int)p.row_bytes) {
                            tma_load_2d(to + j * (16 * F::PITCH), &w_rows, x & ~15, row0 / 8, &ctl->w_full[slot]);
                            if (j < rows)
                                bulk_g2s(smem + F::TAIL_AT + slot * F::TAIL + j * F::PITCH, p.w + whole * p.row_bytes + (x & ~15), (uint32_t)min(F::PITCH, end - (x & ~15)), &ctl->w_full[slot]);
                        }
                    } else {
                        pr_expect(PR_BAR(w_full, slot), 128 * F::PITCH);
                        tma_load_2d(to, &w_rows, b * (F::UNIT / 4), row0, &ctl->w_full[slot]);
                    }
                }
                __syncwarp();
                if (++slot == F::W_SLOTS) { slot = 0; phase ^= 1u; }
                advance(it, tile, b);
            }
        } else if (warp >= F::MMA_WARP && rank == 0) {
            // -------------------------------------------------------------- MMA issue, for both CTAs: two warps take the chunks in turn
            const int issuer = warp - F::MMA_WARP;
            const uint32_t idesc = F::I8 ? tc::idesc_i8(PR_ROWS, F::CHUNK, true, true) : tc::idesc_f16_f32acc(PR_ROWS, F::CHUNK);
            const uint64_t b0 = tc::smem_desc_sw128(base + F::TOKENS_AT);
            const uint64_t am0 = tc::smem_desc(base + F::AMIN_AT, 2048, 128), xm0 = tc::smem_desc(base + F::XMIN_AT, F::CHUNK * 8, 128);
            int s = 0, buf = 0, slot = 0;
            uint32_t b_phase = 0, a_phase = 0, d_phase = 1, turn = issuer ^ 1;
            bool mine = issuer == 0;
            if constexpr (F::GROUPED) {
                const uint32_t floats = tc::idesc_f16_f32acc(PR_ROWS, F::CHUNK);
                for (int at = 0; ok && at < 2 * total; ++at) {          // half blocks; a group of 32 elements a turn
                    ok = pr_wait(PR_BAR(a_full, buf), a_phase, bars);
                    if (!ok) break;
                    const uint32_t a = a_base + (uint32_t)(buf * F::A_COLUMNS);
                    for (int c = 0; ok && c < chunks; ++c) {
                        const uint64_t bs = b0 + (uint64_t)((uint32_t)(s * F::STAGE) >> 4);
                        if (!pr_wait(PR_BAR(b_full, s), b_phase, bars)) { ok = false; break; }
#pragma unroll 1
                        for (int g = 0; g < F::GROUPS; ++g) {
                            if ((g & 1) == issuer) {
                                if (!pr_wait(PR_BAR(d_empty, slot), d_phase, bars)) { ok = false; break; }
                                if (!pr_wait(PR_BAR(turn, issuer), turn, bars)) { ok = false; break; }
                                turn ^= 1u;
                                tc::fence_after_sync();
                                if (elect_one()) {
                                    const uint32_t d = tmem + (uint32_t)(F::CHUNK * slot);
                                    const uint64_t bg = bs + (uint64_t)((g >> 1) * (F::CHUNK / 2 * 128 >> 4)) + (uint64_t)((g & 1) * 4);
                                    pair_mma<false>(d, a + 16u * (uint32_t)g, bg, floats, 0);
                                    pair_mma<false>(d, a + 16u * (uint32_t)g + 8u, bg + 2, floats, 1);
                                    pr_arrive(PR_BAR(turn, issuer ^ 1));
                                    commit_both(PR_BAR(d_full, slot));
                                    if (g >= F::GROUPS - 2) commit_both(PR_BAR(b_empty, s));
                                }
                                __syncwarp();
                            }
                            if (++slot == F::SLOTS) { slot = 0; d_phase ^= 1u; }
                        }
                        if (++s == F::STAGES) { s = 0; b_phase ^= 1u; }
                    }
                    if (ok && elect_one()) commit_both(PR_BAR(a_empty, buf));
                    __syncwarp();
                    if (++buf == F::A_BUFFERS) { buf = 0; a_phase ^= 1u; }
                }
            } else
            for (int it = 0; ok && it < total; ++it) {
                ok = pr_wait(PR_BAR(a_full, buf), a_phase, bars);
                if (!ok) break;
                const uint32_t a = a_base + (uint32_t)(buf * F::A_COLUMNS);
                for (int c = 0; c < chunks; ++c) {
                    if (mine) {
                        if (!pr_wait(PR_BAR(b_full, s), b_phase, bars)) { ok = false; break; }
                        if (!pr_wait(PR_BAR(d_empty, slot), d_phase, bars)) { ok = false; break; }
                        if (!pr_wait(PR_BAR(turn, issuer), turn, bars)) { ok = false; break; }
                        turn ^= 1u;
                        tc::fence_after_sync();
                        if (elect_one()) {
                            const uint32_t d = tmem + (uint32_t)(F::SUMS * F::CHUNK * slot);
                            const uint64_t bs = b0 + (uint64_t)((uint32_t)(s * F::STAGE) >> 4);
#pragma unroll
                            for (int limb = 0; limb < F::LIMBS; ++limb)
#pragma unroll
                                for (int k = 0; k < F::STEPS; ++k)
                                    pair_mma<F::I8>(d + (uint32_t)(limb * F::CHUNK), a + (uint32_t)(64 * limb + 8 * k), bs + (uint64_t)(((k >> 2) * (F::CHUNK / 2 * 128) + 32 * (k & 3)) >> 4), idesc, k);
                            if constexpr (F::MINS) {
                                const uint64_t xm = xm0 + (uint64_t)((uint32_t)(s * F::CHUNK * 16) >> 4), am = am0 + (uint64_t)((uint32_t)(buf * F::AMIN) >> 4);
                                const uint32_t floats = tc::idesc_f16_f32acc(PR_ROWS, F::CHUNK);
                                if (!F::I8) pair_mma_f16_ss(d, am + (4096 >> 4), xm, floats, 1);   // 8 * scales * sums of the codes: what the centred codes left out
                                pair_mma_f16_ss(d + F::LIMBS * F::CHUNK, am, xm, floats, 0);       // mins * sums of the codes
                            }
                            pr_arrive(PR_BAR(turn, issuer ^ 1));
                            commit_both(PR_BAR(d_full, slot));
                            commit_both(PR_BAR(b_empty, s));
                        }
                        __syncwarp();
                    }
                    mine = !mine;
                    if (++s == F::STAGES) { s = 0; b_phase ^= 1u; }
                    if (++slot == F::SLOTS) { slot = 0; d_phase ^= 1u; }
                }
                if (ok && elect_one()) commit_both(PR_BAR(a_empty, buf));
                __syncwarp();
                if (++buf == F::A_BUFFERS) { buf = 0; a_phase ^= 1u; }
            }
        }
    }

    // A CTA stays until everything addressed to it has landed: the last commits,
    __syncwarp();
    if (ok && warp == F::TOKEN_WARP) {
        const int loads = total * F::HALVES * chunks;
        for (int k = max(0, loads - F::STAGES); ok && k < loads; ++k) ok = pr_wait(PR_BAR(b_empty, k % F::STAGES), (uint32_t)(k / F::STAGES) & 1u, bars);
    } else if (ok && warp == F::MMA_WARP) {
        for (int k = max(0, total * F::HALVES - F::A_BUFFERS); ok && k < total * F::HALVES; ++k) ok = pr_wait(PR_BAR(a_empty, k % F::A_BUFFERS), (uint32_t)(k / F::A_BUFFERS) & 1u, bars);
    }
    if (tmem_ok && !ok && lane == 0) {                                 // gave up, or was told: both CTAs are to leave
        const uint32_t abort = bars + (uint32_t)offsetof(PairControl, abort);
        sts_u32(abort, 1u);
        tc::st_cluster_u32(tc::map_to_cta(abort, (uint32_t)rank ^ 1u), 1u);
        report(p.status, ST_WAIT_TIMEOUT);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();
    if (*reinterpret_cast<volatile int *>(&ctl->abort)) {              // the same in both CTAs now
        // or, when a role has given up, whatever has been issued: MMAs, behind which the tensor core arrives once more, and copies (a few us; a millisecond
        // is waited for those that no complete phase counts)
        if (warp >= F::MMA_WARP && rank == 0) {
            if (elect_one()) commit_both(PR_BAR(settled, 0));
            __syncwarp();
        }
        uint64_t until;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(until));
        until += 1000000u;
        if (warp == F::MMA_WARP) {
            for (uint32_t i = 0; i < (1u << 20) && !__all_sync(0xffffffffu, pr_try(PR_BAR(settled, 0), 0u)); ++i) {}
        } else if (warp == F::W_WARP) {
            for (int s = 0; s < F::W_SLOTS; ++s) pr_settle(PR_BAR(w_full, s), until);
        } else if (warp == F::TOKEN_WARP) {
            for (int s = 0; s < PR_RING; ++s) pr_settle(PR_BAR(scales_full, s), until);
            for (int s = 0; rank == 0 && s < F::STAGES; ++s) pr_settle(PR_BAR(b_full, s), until);      // they count the halves of both CTAs
        }
        __syncthreads();
        tc::cluster_sync_all();
    }
    if (warp == F::MMA_WARP && *reinterpret_cast<volatile uint32_t *>(&ctl->tmem_base) != 0xffffffffu) tc::tmem_free(*reinterpret_cast<volatile uint32_t *>(&ctl->tmem_base), 512);
}

// Adds the parts of the tiles that pairs share, in the order of their blocks: a CTA for what one epilogue warp of a CTA left.  L2-bound:
// each part is read once, Y written once.
template <int FMT>
__global__ void __launch_bounds__(512) pair_parts_kernel(const __grid_constant__ PairParams p) {
    using F = PairFormat<FMT>;
    asm volatile("griddepcontrol.launch_dependents;");
    const int tile_first = (int)blockIdx.x * p.nb, p0 = p.pair_of(tile_first), p1 = p.pair_of(tile_first + p.nb - 1);
    const int rank = (int)blockIdx.y >> 4, e = (int)blockIdx.y & 15, i = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    const int tile = p.rounds * p.pairs + (int)blockIdx.x, at = 4 * i / F::OWN * F::CHUNK + 4 * i % F::OWN, token = (tile % p.token_tiles) * p.chunks * F::CHUNK + (e >> 2) * F::OWN + at;
    const long long n = (long long)(tile / p.token_tiles) * PR_ROWS + 128 * rank + pair_row_of<FMT>((e & 3) * 32 + lane);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (p0 == p1 || at >= p.chunks * F::CHUNK || n >= p.n || token >= p.m) return;     // a pair alone has stored it; nothing there
    ulonglong2 sum = make_ulonglong2(0, 0);
    for (int q = p0; q <= p1; ++q) {
        const ulonglong2 v = __ldcg(p.parts + pair_part<FMT>(q, p.start_of(q) > tile_first, rank, e, lane) + 32 * i);
        sum = make_ulonglong2(add2(sum.x, v.x), add2(sum.y, v.y));
    }
    float *y = p.y + n + (long long)token * p.ldy;
    y[0] = half_of(sum.x, 0);
    if (token + 1 < p.m) y[p.ldy] = half_of(sum.x, 1);
    if (token + 2 < p.m) y[2 * p.ldy] = half_of(sum.y, 0);
    if (token + 3 < p.m) y[3 * p.ldy] = half_of(sum.y, 1);
}

template <int FMT> cudaError_t launch_pair_kernel(const PairParams &params, const CUtensorMap &codes, const CUtensorMap &mins, const CUtensorMap &rows, int pairs, cudaStream_t stream) {
    using F = PairFormat<FMT>;
    cudaError_t e = grant_dynamic_smem(reinterpret_cast<const void *>(pair_kernel<FMT>), F::BYTES);
    if (e == cudaSuccess) e = check_launch_registers(reinterpret_cast<const void *>(pair_kernel<FMT>), F::REGS);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(F::THREADS);
    cfg.dynamicSmemBytes = (size_t)F::BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, pair_kernel<FMT>, params, codes, mins, rows);
    if (e != cudaSuccess || !params.rest || !params.share) return e;
    cfg.gridDim = dim3((unsigned)params.rest, 2 * PR_E_WARPS);
    cfg.blockDim = dim3(F::TOKENS / 16 * 32);
    cfg.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&cfg, pair_parts_kernel<FMT>, params);
}

#define PR_EACH_FORMAT(DO) DO(F_Q4_K) DO(F_Q5_K) DO(F_Q6_K) DO(F_TQ1_0) DO(F_Q4_0) DO(F_Q8_0)

}  // namespace weft
