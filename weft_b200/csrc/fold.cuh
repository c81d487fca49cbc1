// mul_mat for smaller batches of Q4_K on tcgen05 with the weights as the operand in TENSOR MEMORY (larger ones: pairs.cuh).
//
// D[128 weight rows, Nt tokens] += A[128, 256] * B[256, Nt] per 256-element block, kind::f16 with fp32 accumulators.  The A
// operand is the block's integers with the sub-block scales multiplied in, B the activation codes as f16.  One scale pair per
// (row, block) and one per (token, block) is left for the epilogue: acc += x.d * (d * S - dmin * M).
//
// S is an integer, and the accumulator holds its part of it exactly, whatever the order of its terms: scale * (q - 8), at most
// 504 * 128 * 256 in all, stays below 2^24 (times the power of two that all terms share) with codes up to 128 and every bit of a
// record set.  8 * sum(scale * sum of the group's codes), what the centre left out, follows as one K = 16 step, the only one that may
// round (sums beyond 2^24, by at most 2^-23).  (Scales times whole codes reach 3.1e7: a block whose terms cancel lost its low bits on
// the way.)
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
// the rest: S twice (a block's is read while the next one is summed), M once, A for one block up to 128 tokens, for two up to 80.
// A passes from the expanders to the MMAs in half blocks (in quarters more was lost to the MMA warp's waits, about 150 clocks each,
// than was gained).
//
// Roles (28 warps): 16 expanders in four groups that take the blocks in turn (a warp alone issues every four to seven clocks:
// with two groups a block took 1900 clocks), 8 epilogue warps (lane quarter x every other eight
// tokens), a warp each for the token copies, the weight records and the MMAs.  The records come by TMA.  The warps that issue copies and
// MMAs run as a whole with warp-uniform operands and elect a lane for the instruction only: issued from a divergent lane, each operand
// of each MMA moves to the uniform registers on its own, about 100 clocks per instruction.  Few
// tiles: a cluster of CTAs shares a tile, each with a slice of K; the partial sums meet through distributed shared memory in
// rank order.
//
// What bounds it: the hand-overs of A (expanders, MMAs, expanders) and the instructions of the unpacking, 1750 clocks a
// block up to 64 tokens and 2500 with 128 against 1088 of tensor work.  Measured on B200 (us, device time with the kernel that makes
// the planes; before: register tiles): 128 x 4096 x 4096 27.5 -> 16.5, 64 x 4096 x 14336 46.0 -> 26.2, 512 x 1024 x 4096 29.0 -> 17.7
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
constexpr int FD_W_SLOTS = 4;                   // most blocks of weight records
constexpr int FD_SMEM = 227 * 1024;
constexpr int FD_B_MAX = 6, FD_SLOTS = 8;      // most half-block stages of tokens; slots of the x.d ring
constexpr int FD_DD_SLOTS = 4;
// Registers a thread: at launch, and after the roles have traded (setmaxnreg).  The trade stays inside what the CTA got.
constexpr int FD_REGS = 72, FD_X_REGS = 64, FD_E_REGS = 104, FD_IO_REGS = 40;
static_assert(FD_GROUPS * 128 * FD_X_REGS + 256 * FD_E_REGS + 128 * FD_IO_REGS <= FD_THREADS * FD_REGS, "setmaxnreg would wait for ever");

constexpr int FD_UNIT = unit_bytes(F_Q4_K), FD_CHUNKS = 2;         // A buffers (of 64 columns, half a block) of a block
constexpr int fold_columns(int nt) { return 3 * nt; }             // accumulators of nt columns: S twice (a block's is drained while the next one's is filled) and M
static_assert(FD_UNIT / 16 % 2 == 1, "rows in different banks");

struct FoldParams {
    const float *xd;             // (nb, pitch)
    float *y;
    long long n, ldy, pitch;
    int m, nb, nt;               // tokens, blocks per row, tokens per tile (a multiple of 16)
    int token_tiles, tiles, slices, b_stages, a_buffers;
    int most_blocks;             // that the record warp fetches before it gives up
    int *status;
};

struct FoldControl {
    uint64_t b_full[FD_B_MAX], b_empty[FD_B_MAX], a_full[4], a_empty[4][FD_GROUPS], d_full[2], d_empty[2], xd_full[FD_SLOTS], w_full[FD_GROUPS], w_empty[FD_W_SLOTS], settled;
    uint32_t tmem_base;
    int abort;
};

// Shared memory, in this order; the token stages must lie on 1024-byte boundaries.
struct FoldLayout {
    static constexpr int CONTROL = 1024;
    // wide tiles keep two blocks of records (one per expander group) so that more tokens can be on their way
    static __host__ __device__ constexpr int w_slots(int tt) { return tt > 64 ? 2 : FD_W_SLOTS; }
    // tt: tokens per tile
    static __host__ __device__ constexpr int stage(int tt) { return tt * 256; }
    static __host__ __device__ constexpr int tokens_at() { return CONTROL; }
    static __host__ __device__ constexpr int raw_at(int tt, int stages) { return tokens_at() + stages * stage(tt); }
    static __host__ __device__ constexpr int dd_at(int tt, int stages) { return raw_at(tt, stages) + w_slots(tt) * FD_ROWS * FD_UNIT; }
    static __host__ __device__ constexpr int xd_at(int tt, int stages) { return dd_at(tt, stages) + FD_DD_SLOTS * 2 * FD_ROWS * 4; }
    static __host__ __device__ constexpr int xmin_at(int tt, int stages) { return xd_at(tt, stages) + FD_SLOTS * tt * 4; }
    static __host__ __device__ constexpr int amin_at(int tt, int stages) { return xmin_at(tt, stages) + 4 * tt * 32; }
    // A operands over the sums of 32 codes: FD_AMIN slots for the mins, as many for the scales
    static __host__ __device__ constexpr int bytes(int tt, int stages) { return amin_at(tt, stages) + 2 * FD_AMIN * 4096; }
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

__device__ __forceinline__ void fd_give_up(FoldControl *ctl, int *status) {
    *reinterpret_cast<volatile int *>(&ctl->abort) = 1;
    report(status, ST_WAIT_TIMEOUT);
}
// Bounded wait of a whole warp.  Gives up when another role has, or after the limit; then every role leaves.  What follows a wait is for whole warps,
// so its lanes must not part: those that are about to give up look once more, and a phase that another lane has seen complete they see so too.
__device__ __forceinline__ bool fd_wait(uint64_t *bar, uint32_t parity, FoldControl *ctl, int *status) {
    for (uint32_t left = 1u << 20; left; --left) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((left & 7u) == 0u && *reinterpret_cast<volatile int *>(&ctl->abort)) left = 2u;
    }
    fd_give_up(ctl, status);
    return false;
}

// ------------------------------------------------------------------ unpacking: a quarter of a block (64 elements) of one row
// Word i of the result holds elements {0, 2} (even i) or {1, 3} (odd i) of the i / 2 -th group of four: the order of the
// activation plane.  A code's bits where they lie are an f16 below the normal range, q * 2^-24 (high nibbles
// q * 2^-20); one multiply-add applies the scale and the centre: q * 2^-24 * (scale * 2^10) - 8 * scale * 2^-14, exactly.

// the 6-bit scales of a record, four to a word: [0] scales 0..3, [1] 4..7; mins alike
struct FoldScales { uint32_t sc[2], mn[2]; };

// The scales of quarter q's two groups and what centres their codes, as f16 pairs
struct FoldQuarterScales {
    uint32_t slo, shi, clo, chi;
    __device__ __forceinline__ FoldQuarterScales(int q, const FoldScales &s) {
        const uint32_t scales = (q & 2 ? s.sc[1] : s.sc[0]) >> (16 * (q & 1));
        const uint32_t lo = small_half2(scales & 255u), hi = small_half2((scales >> 8) & 255u);
        slo = hmul2(lo, 0x64006400u);                  // * 2^10
        shi = hmul2(hi, 0x54005400u);                  // * 2^6: high nibbles stay where they are
        clo = hmul2(lo, 0x90009000u);                  // * -2^-11
        chi = hmul2(hi, 0x90009000u);
    }
};

// (q - 8) * scale * 2^-14
__device__ __forceinline__ void fold_quarter(int q, const uint8_t *record, const FoldQuarterScales &s, uint32_t (&out)[32]) {
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const uint4 q4 = *reinterpret_cast<const uint4 *>(record + 16 + 32 * q + 16 * v);
        const uint32_t w4[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const uint32_t w = o ? w4[i] >> 8 : w4[i];
                out[8 * v + 2 * i + o] = hfma2(w & 0x000f000fu, s.slo, s.clo);
                out[16 + 8 * v + 2 * i + o] = hfma2(w & 0x00f000f0u, s.shi, s.chi);
            }
    }
}

// ------------------------------------------------------------------ the kernel

// The CTA's work: tiles first, first + stride, ..., and of each the blocks [begin, end) of its slice of K.
struct FoldAt {
    int tile, b;
    __device__ __forceinline__ void advance(int begin, int end, int stride) { if (++b == end) { b = begin; tile += stride; } }
};

__global__ void __launch_bounds__(FD_THREADS, 1) fold_kernel(const __grid_constant__ FoldParams p, const __grid_constant__ CUtensorMap x_codes, const __grid_constant__ CUtensorMap x_mins,
                                                                const __grid_constant__ CUtensorMap w_rows) {
    using L = FoldLayout;
    extern __shared__ __align__(1024) uint8_t smem[];
    FoldControl *ctl = reinterpret_cast<FoldControl *>(smem);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int nt = p.nt, stages = p.b_stages, abufs = p.a_buffers, w_slots = L::w_slots(nt), w_shift = w_slots == 4 ? 2 : 1;
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
        mbar_init(&ctl->settled, 1);
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
    const int a_blocks = abufs / FD_CHUNKS;             // 0: two buffers, each filled twice in a block of four
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
        bool ok = true;
        for (int it = group; it < total && ok; it += FD_GROUPS) {
            const int slot = it & (w_slots - 1);
            if (!fd_wait(&ctl->w_full[group], (uint32_t)(it / FD_GROUPS) & 1u, ctl, p.status)) break;
            const uint8_t *record = s_raw + slot * (FD_ROWS * FD_UNIT) + (quarter * 32 + lane) * FD_UNIT;
            float *dd = s_dd + (it % FD_DD_SLOTS) * (2 * FD_ROWS) + quarter * 32 + lane;
            const uint4 head = *reinterpret_cast<const uint4 *>(record);
            const float d0 = half_bits_to_float(head.x) * 16384.0f, d1 = -half_bits_to_float(head.x >> 16);      // the operands carry 2^-14
            const Q4KScales u = q4k_unpack_scales(head.y, head.z, head.w);
            const FoldScales s{{u.sc_lo, u.sc_hi}, {u.mn_lo, u.mn_hi}};
            // One loop body for all quarters: the roles' code has to stay in the instruction caches.  Unrolled by quarters, every
            // instruction took 7 to 19 clocks (1.8 to 2.4 thousand clocks a block).
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                const int buf = (it * FD_CHUNKS + c / 2) & (abufs - 1);
                uint32_t v[32];
                fold_quarter(c, record, FoldQuarterScales(c, s), v);
                if (c % 2 == 0) {
                    if (!fd_wait(&ctl->a_empty[buf][group], a_parity(it, c / 2), ctl, p.status)) { ok = false; break; }
                    tc::fence_after_sync();
                }
                if (c == 0) { dd[0] = d0; dd[FD_ROWS] = d1; }
                tmem_st32(lane_base + (uint32_t)(64 * buf + 32 * (c % 2)), v);
                if (c == 3) {             // two 16-byte chunks of a K = 16 operand: {m_0 .. m_7 | 64 m_0 .. 64 m_7}, and 8 * 2^-14 times the scales
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
                if (c % 2 == 1) {
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
                const int slot = it % FD_SLOTS, buf = it & 1;
                const uint32_t d_phase = (uint32_t)(it >> 1) & 1u;
                const float *xd = s_xd + slot * nt + 8 * group, *dd = s_dd + (it % FD_DD_SLOTS) * (2 * FD_ROWS) + row;
                if (!fd_wait(&ctl->xd_full[slot], (uint32_t)(it / FD_SLOTS) & 1u, ctl, p.status) || !fd_wait(&ctl->d_full[buf], d_phase, ctl, p.status)) { ok = false; break; }
                tc::fence_after_sync();
                const float d0 = dd[0], d1 = dd[FD_ROWS];
                const uint64_t s0 = pack2(d0, d0), s1 = pack2(d1, d1);
                const uint32_t from = lane_base + (uint32_t)(buf * nt), from_min = lane_base + (uint32_t)(2 * nt);
                // eight columns at a time, the next ones on their way while these are added
                uint32_t v0[2][8], vm[2][8];
                auto load = [&](int k) {
                    tc::tmem_ld8(from + (uint32_t)(16 * k), v0[k % 2]);
                    tc::tmem_ld8(from_min + (uint32_t)(16 * k), vm[k % 2]);
                };
                auto pair = [&](const uint32_t (&v)[8], int e) { return pack2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])); };
                auto scaled = [&](int k, int e) { return fma2(s1, pair(vm[k % 2], e), mul2(s0, pair(v0[k % 2], e))); };     // d * S - dmin * M
                load(0);
                tc::tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < OWN / 8; ++k) {
                    if (k < pieces) {
                        if (k + 1 < pieces) load(k + 1);
#pragma unroll
                        for (int i = 0; i < 8; i += 4) {
                            const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(xd + 16 * k + i);
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int j = i + 2 * e;
                                uint64_t a = pack2(acc[8 * k + j], acc[8 * k + j + 1]);
                                a = fma2(e ? x.y : x.x, scaled(k, j / 2), a);
                                unpack2(a, acc[8 * k + j], acc[8 * k + j + 1]);
                            }
                        }
                        if (k + 1 < pieces) tc::tmem_ld_wait();
                    }
                    // all read: the buffers are free
                    if (k == 0 ? pieces <= 2 : k + 2 == pieces) {
                        tc::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&ctl->d_empty[buf]);
                    }
                }
            }
            if (!ok) break;
            if (p.slices == 1) {
                const long long n = (long long)(tile / p.token_tiles) * FD_ROWS + row;
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
                    mbar_expect_tx(full, (uint32_t)(nt * 256 + (h == 1 ? nt * 32 : 0)));
                    tma_load_2d(stage, &x_codes, 256 * at.b + 128 * h, t0, full);
                    tma_load_2d(stage + nt * 128, &x_codes, 256 * at.b + 128 * h + 64, t0, full);
                    if (h == 1) {
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
            for (int it = 0; it < total && ok; ++it) {
                const int set = it & 1;
                const uint32_t d = tmem + (uint32_t)(set * nt);
#pragma unroll 1
                for (int j = 0; j < FD_CHUNKS; ++j) {
                    if (!fd_wait(&ctl->b_full[s], b_phase, ctl, p.status) || !fd_wait(&ctl->a_full[buf], a_phase, ctl, p.status)) { ok = false; break; }
                    const uint64_t b = b0 + (uint64_t)((uint32_t)(s * L::stage(nt)) >> 4);
                    const uint32_t a = a_base + 64u * (uint32_t)buf;
                    tc::fence_after_sync();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 8; ++k)                     // K steps of the half-block in order
                            mma_f16_ts(d, a + (uint32_t)(8 * k), b + (uint64_t)(((uint32_t)(k >> 2) * slab + 32u * (k & 3)) >> 4), idesc, j | k);
                        tc::commit(&ctl->a_empty[buf][(it * FD_CHUNKS + j + abufs) / FD_CHUNKS % FD_GROUPS]);
                        tc::commit(&ctl->b_empty[s]);
                        // 8 * scales * sums of the codes, what the centred codes left out
                        if (j == FD_CHUNKS - 1)
                            tc::mma_f16(d, am0 + (uint64_t)((FD_AMIN + (it & (FD_AMIN - 1))) * (4096 >> 4)), xm0 + (uint64_t)((uint32_t)((it & 3) * nt * 32) >> 4), idesc, 1);
                    }
                    __syncwarp();
                    if (++buf == abufs) { buf = 0; a_phase ^= 1u; }
                    if (++s == stages) { s = 0; b_phase ^= 1u; }
                }
                if (ok) {
                    // M of the block before has been read, and so has its S
                    if (it > 0 && !fd_wait(&ctl->d_empty[(it - 1) & 1], (uint32_t)((it - 1) >> 1) & 1u, ctl, p.status)) { ok = false; break; }
                    tc::fence_after_sync();
                    if (elect_one()) {
                        tc::mma_f16(tmem + (uint32_t)(2 * nt), am0 + (uint64_t)((it & (FD_AMIN - 1)) * (4096 >> 4)), xm0 + (uint64_t)((uint32_t)((it & 3) * nt * 32) >> 4), idesc, 0);
                        tc::commit(&ctl->d_full[set]);
                    }
                    __syncwarp();
                }
            }
            // the last commits have to arrive before the CTA leaves
            if (ok && !*reinterpret_cast<volatile int *>(&ctl->abort)) {
                for (int k = max(0, FD_CHUNKS * total - abufs); k < FD_CHUNKS * total; ++k) {
                    const int next = k + abufs, block = next / FD_CHUNKS;
                    mbar_wait(&ctl->a_empty[k & (abufs - 1)][block % FD_GROUPS], a_parity(block, next % FD_CHUNKS), 1u << 20);
                }
                for (int k = max(0, 2 * total - stages); k < 2 * total; ++k) mbar_wait(&ctl->b_empty[k % stages], (uint32_t)(k / stages) & 1u, 1u << 20);
            } else {
                // a role has given up: the MMAs issued so far have to be done, and their commits here, before tensor memory is freed
                if (elect_one()) tc::commit(&ctl->settled);
                __syncwarp();
                mbar_wait(&ctl->settled, 0u, 1u << 20);
            }
        }
        } else if (warp == FD_W_WARP) {
        // ------------------------------------------------------------------ weight records
        FoldAt at{first_tile, begin};
        int issued = 0;
        for (int it = 0; it < total; ++it, at.advance(begin, end, stride)) {
            const int slot = it & (w_slots - 1), row0 = (at.tile / p.token_tiles) * FD_ROWS;
            if (it >= p.most_blocks) { fd_give_up(ctl, p.status); break; }
            if (!fd_wait(&ctl->w_empty[slot], ((uint32_t)(it >> w_shift) & 1u) ^ 1u, ctl, p.status)) break;
            if (elect_one()) {
                uint8_t *to = s_raw + slot * (FD_ROWS * FD_UNIT);
                mbar_expect_tx(&ctl->w_full[it % FD_GROUPS], FD_ROWS * FD_UNIT);
                tma_load_2d(to, &w_rows, at.b * (FD_UNIT / 4), row0, &ctl->w_full[it % FD_GROUPS]);
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
                const long long n = n0 + (i & (FD_ROWS - 1));
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

// ------------------------------------------------------------------ launch

struct FoldPlan { int nt, slices, stages, a_buffers; double cost; };

inline int fold_stages(int tt) {
    for (int s = FD_B_MAX; s >= 2; --s)
        if (FoldLayout::bytes(tt, s) <= FD_SMEM) return s;
    return 0;
}

constexpr int FD_SMEM_LEAST = 118 * 1024;

// How many clusters of `slices` CTAs, one CTA per SM, the device holds at once (0: unknown).  Clusters stay inside a GPC, whose
// SMs are not a multiple of eight, so it is fewer than SMs / slices, and those that do not fit run in a second round: 512 x 2048
// with 64 tokens took 18.0 us on 16 clusters of eight and 10.7 us where the plan asks for no more than fit.
inline int fold_clusters(int slices) {
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
    if (grant_dynamic_smem(reinterpret_cast<const void *>(fold_kernel), FD_SMEM_LEAST) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, fold_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    known[slices].store(n > 0 ? n : -1, std::memory_order_relaxed);
    return n;
}

inline cudaError_t launch_fold_kernel(const FoldParams &params, const CUtensorMap &codes, const CUtensorMap &mins, const CUtensorMap &rows, int sm_count, cudaStream_t stream) {
    // at least half of an SM's shared memory: a second CTA beside this one would wait for the tensor memory this one holds,
    // and two clusters waiting for each other that way would never end
    const int smem = std::max(FoldLayout::bytes(params.nt, params.b_stages), FD_SMEM_LEAST);
    cudaError_t e = grant_dynamic_smem(reinterpret_cast<const void *>(fold_kernel), smem);
    if (e == cudaSuccess) e = check_launch_registers(reinterpret_cast<const void *>(fold_kernel), FD_REGS);
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
    return cudaLaunchKernelEx(&cfg, fold_kernel, params, codes, mins, rows);
}

}  // namespace weft
