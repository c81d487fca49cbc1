// Host side of the tensor-memory contraction (fold.cuh) and the kernel that quantizes activations into its planes.
#include "fold.cuh"
#include "quantize.cuh"

#include <algorithm>

namespace weft {

// ------------------------------------------------------------------ activation planes
// One warp per (token, 256-element block): quantizes the fp32 values (same bodies as the standalone quantizers), stores the
// caller's records, the codes as f16 (each group of four as elements 0, 2, 1, 3: the order in which the weights unpack), the
// scales by (block, token) and the sums of 32 codes as 64 h + l in two exact f16 limbs.  Without X
// the caller's records are the source.  HBM/L2-bound: 4 bytes in, 1.14 out to the records and 2.1 to the planes.
template <bool FROM_X, bool A16>
__global__ void __launch_bounds__(256) fold_planes_kernel(const float *__restrict__ x, uint8_t *__restrict__ xq, uint4 *__restrict__ codes, float *__restrict__ xd,
                                                          __half *__restrict__ mins, int m, int nb, long long pitch) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= (long long)m * nb) return;
    const int token = (int)(unit / nb), block = (int)(unit - (long long)token * nb);
    uint32_t q0, q1;
    float d;
    {
        uint8_t *rec = xq + unit * 292;
        int sum;                                  // of the lane pair's 16 codes (the record's bsum)
        if constexpr (FROM_X) {
            float v[8];
            load8<A16>(x + unit * 256 + 8 * lane, v);
            q8_k_warp(v, q0, q1, sum, d);
            store_q8_k(rec, lane, q0, q1, sum, d);
        } else {
            q0 = *reinterpret_cast<const uint32_t *>(rec + 4 + 8 * lane);
            q1 = *reinterpret_cast<const uint32_t *>(rec + 8 + 8 * lane);
            sum = *reinterpret_cast<const int16_t *>(rec + 260 + (lane & ~1));
            d = *reinterpret_cast<const float *>(rec);
        }
        if (lane == 0) xd[(long long)block * pitch + token] = d;
        {
            const int pair = sum + __shfl_xor_sync(0xffffffffu, sum, 2);       // lanes 4 g .. 4 g + 3: sum of group g
            if ((lane & 3) == 0) {
                __half *to = mins + unit * 16 + (lane >> 2);
                to[0] = __int2half_rn(pair & 63);
                to[8] = __int2half_rn(pair >> 6);
            }
        }
    }
    // bytes as f16: set under the exponent of 1024, 128 added to make them unsigned, both taken out again
    const uint32_t u0 = q0 ^ 0x80808080u, u1 = q1 ^ 0x80808080u;
    codes[unit * 32 + lane] = make_uint4(hadd2(__byte_perm(u0, 0x64646464u, 0x4240), 0xe480e480u), hadd2(__byte_perm(u0, 0x64646464u, 0x4341), 0xe480e480u),
                                         hadd2(__byte_perm(u1, 0x64646464u, 0x4240), 0xe480e480u), hadd2(__byte_perm(u1, 0x64646464u, 0x4341), 0xe480e480u));
}

static cudaError_t launch_planes(const TileArgs &a, uint4 *codes, float *xd, __half *mins, long long pitch, cudaStream_t stream) {
    const int nb = (int)(a.k / 256), m = (int)a.m;
    const unsigned grid = (unsigned)((a.m * nb + 7) / 8);
    uint8_t *xq = static_cast<uint8_t *>(const_cast<void *>(a.xq));
    if (!a.x) fold_planes_kernel<false, false><<<grid, 256, 0, stream>>>(nullptr, xq, codes, xd, mins, m, nb, pitch);
    else if (reinterpret_cast<uintptr_t>(a.x) & 15u) fold_planes_kernel<true, false><<<grid, 256, 0, stream>>>(a.x, xq, codes, xd, mins, m, nb, pitch);
    else fold_planes_kernel<true, true><<<grid, 256, 0, stream>>>(a.x, xq, codes, xd, mins, m, nb, pitch);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ dispatch

struct FoldPlaneSizes { size_t codes, xd, mins; long long pitch; };
static FoldPlaneSizes plane_sizes(long long m, long long k) {
    const size_t nb = (size_t)(k / 256), rows = nb;
    FoldPlaneSizes s;
    s.pitch = (m + 127) / 128 * 128 + 128;       // the last tile of tokens reads whole
    s.codes = (size_t)m * (size_t)k * 2;
    s.xd = rows * (size_t)s.pitch * 4;
    s.mins = (size_t)m * nb * 32;
    return s;
}
size_t fold_plane_bytes(const TileArgs &a) {
    const FoldPlaneSizes s = plane_sizes(a.m, a.k);
    return s.codes + s.xd + s.mins;
}

// Tensor memory (512 columns): the accumulators, and A for two blocks where there is room, else for one.
static int fold_a_buffers(int nt) { return fold_columns(nt) + 256 <= 512 ? 4 : 2; }
// Picks tokens per tile and slices of K by estimated clocks: rounds of the grid times the blocks of a tile.  A block takes
// about 1800 clocks when A has buffers for two (up to 80 tokens) and 2350 with one, whatever the tokens (measured from 16 to
// 128).  A tile's start, its stores and the meeting of the slices are small beside it.
static double fold_tile_cost(int nt, int abufs, long long steps) { return steps * (abufs >= 2 * FD_CHUNKS ? 1800.0 : 2350.0) + 1200.0 + 4.0 * nt; }

static FoldPlan fold_plan(long long m, long long n, long long nb, int sm_count) {
    FoldPlan best{0, 0, 0, 0, 0.0};
    const long long row_tiles = (n + FD_ROWS - 1) / FD_ROWS;
    for (int nt = 16; nt <= FD_TOKENS; nt += 16) {
        const int stages = fold_stages(nt), abufs = fold_a_buffers(nt);
        if (stages < 2) continue;
        const long long tiles = row_tiles * ((m + nt - 1) / nt);
        for (int slices = 1; slices <= 8 && slices <= nb; ++slices) {
            if (slices > 1 && tiles > fold_clusters(slices)) break;
            const long long rounds = slices > 1 ? 1 : (tiles + sm_count - 1) / sm_count, steps = (nb + slices - 1) / slices;
            const double cost = rounds * fold_tile_cost(nt, abufs, steps) + (slices > 1 ? 1500.0 : 0.0);
            if (!best.nt || cost < best.cost) best = FoldPlan{nt, slices, stages, abufs, cost};
        }
    }
    return best;
}

// One launch, or two: where the last round of the grid would be nearly empty, the rows of the full rounds go first and the others
// follow as a launch of their own, which can share K among the SMs (512 x 14336 x 4096: 448 tiles of 128 tokens are three rounds
// of 148 and four tiles: 92.7 us as one launch, 86.0 as two; 200 x 28672 x 4096 106 and 82).
struct FoldSplit { FoldPlan first, second; long long rows; double cost; };     // rows of the first launch; all of them: no second
constexpr double FD_SECOND = 12000.0;     // clocks that a second launch costs beside its tiles
static FoldSplit fold_split(long long m, long long n, long long nb, int sm_count) {
    FoldSplit best{fold_plan(m, n, nb, sm_count), FoldPlan{0, 0, 0, 0, 0.0}, n, 0.0};
    best.cost = best.first.cost;
    const long long row_tiles = (n + FD_ROWS - 1) / FD_ROWS;
    for (int nt = 16; nt <= FD_TOKENS; nt += 16) {
        const int stages = fold_stages(nt), abufs = fold_a_buffers(nt);
        if (stages < 2) continue;
        const long long token_tiles = (m + nt - 1) / nt, rounds = row_tiles * token_tiles / sm_count, rows = rounds * sm_count / token_tiles * FD_ROWS;
        if (rows <= 0 || rows >= n) continue;
        const FoldPlan rest = fold_plan(m, n - rows, nb, sm_count);
        const double cost = rounds * fold_tile_cost(nt, abufs, nb);
        if (!rest.nt || cost + rest.cost + FD_SECOND >= best.cost) continue;
        best = FoldSplit{FoldPlan{nt, 1, stages, abufs, cost}, rest, rows, cost + rest.cost + FD_SECOND};
    }
    return best;
}

// The plan's clocks beside a start, the planes and the results: within 8 % (rms) of the times of 930 sizes, 33 to 8192 tokens.  Tiles of 80
// tokens take 28 % longer than the plan counts, as long as those of 96.
double fold_estimate(const TileArgs &a, int sm_count) {
    const FoldSplit s = fold_split(a.m, a.n, a.k / 256, sm_count);
    const double clocks = s.cost + (s.first.nt == 80 ? 0.28 * s.first.cost : 0.0) + (s.second.nt == 80 ? 0.28 * s.second.cost : 0.0);
    return 8.2 + 5.0e-4 * clocks + (1.17 * (double)a.k + 0.69 * (double)a.n) * (double)a.m * 1e-6;
}

bool fold_supported(const TileArgs &a) {
    if (a.fmt != F_Q4_K) return false;
    // Below these the register tiles are quicker: this kernel starts about 4 us later (cluster, tensor memory, planes) and takes
    // as long for 16 tokens as for 64; the tiles go by 8 tokens up to 32 and get slow steps at 17, 25 and 33.  Tiles / this, us on
    // the device: 4096 x 4096 with 48 tokens (0.81e9 products) 13.4 / 13.7, with 56 (0.94e9) 15.4 / 14.0; 1024 x 4096 with 160
    // (0.67e9) 13.0 / 13.9, with 256 (1.07e9) 15.6 / 15.0; 14336 x 4096 with 24 tokens 22.5 / 24.3, with 33 29.0 / 25.0.
    const double products = (double)a.m * (double)a.n * (double)a.k;
    if (a.m <= 24 || products < (a.m <= 32 ? 1.2e9 : 9e8)) return false;
    // 16-byte copies of records need a 16-byte aligned matrix; extents are 32-bit in the kernel
    return a.m < (1 << 20) && a.k % 256 == 0 && a.k < (1LL << 22) && a.n >= 8 && a.n < (1LL << 31) && (reinterpret_cast<uintptr_t>(a.w) & 15u) == 0;
}

// The contraction of `n` rows from `w` on into `y`; `planes` holds what does not depend on the cut.
static cudaError_t launch_rows(const TileArgs &a, const FoldPlan &plan, const FoldParams &planes, const uint4 *codes, const __half *mins,
                               const uint8_t *w, long long row_bytes, float *y, long long n, int sm_count, cudaStream_t stream) {
    FoldParams p = planes;
    p.y = y; p.n = n;
    p.nt = plan.nt; p.slices = plan.slices; p.b_stages = plan.stages; p.a_buffers = plan.a_buffers;
    p.token_tiles = (int)((a.m + p.nt - 1) / p.nt);
    p.tiles = p.token_tiles * (int)((n + FD_ROWS - 1) / FD_ROWS);
    CUtensorMap x_codes, x_mins, w_rows;
    cudaError_t e = encode_tile_map(&x_codes, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, codes, (unsigned long long)a.k, (unsigned long long)a.m, (unsigned long long)a.k * 2, 64, (unsigned)p.nt, true);
    if (e == cudaSuccess)
        e = encode_tile_map(&x_mins, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, mins, (unsigned long long)p.nb * 16, (unsigned long long)a.m, (unsigned long long)p.nb * 32, 8, (unsigned)p.nt, false);
    if (e == cudaSuccess)
        e = encode_tile_map(&w_rows, CU_TENSOR_MAP_DATA_TYPE_UINT32, w, (unsigned long long)row_bytes / 4, (unsigned long long)n, (unsigned long long)row_bytes, FD_UNIT / 4, FD_ROWS, false);
    return e == cudaSuccess ? launch_fold_kernel(p, x_codes, x_mins, w_rows, sm_count, stream) : e;
}

cudaError_t launch_fold(const TileArgs &a, uint8_t *planes, int *status, int sm_count, cudaStream_t stream, unsigned *launches) {
    const FoldPlaneSizes s = plane_sizes(a.m, a.k);
    uint4 *codes = reinterpret_cast<uint4 *>(planes);
    float *xd = reinterpret_cast<float *>(planes + s.codes);
    __half *mins = reinterpret_cast<__half *>(planes + s.codes + s.xd);
    FoldParams p{};
    p.xd = xd; p.ldy = a.ldy; p.pitch = s.pitch; p.most_blocks = a.most_blocks; p.status = status;
    p.m = (int)a.m;
    p.nb = (int)(a.k / 256);
    const long long row_bytes = (long long)p.nb * FD_UNIT;
    const FoldSplit split = fold_split(a.m, a.n, p.nb, sm_count);
    if (!split.first.nt) return cudaErrorNotSupported;
    *launches = split.second.nt ? 3 : 2;
    cudaError_t e = launch_planes(a, codes, xd, mins, s.pitch, stream);
    const uint8_t *w = static_cast<const uint8_t *>(a.w);
    if (e == cudaSuccess) e = launch_rows(a, split.first, p, codes, mins, w, row_bytes, a.y, split.rows, sm_count, stream);
    if (e == cudaSuccess && split.second.nt)
        e = launch_rows(a, split.second, p, codes, mins, w + split.rows * row_bytes, row_bytes, a.y + split.rows, a.n - split.rows, sm_count, stream);
    return e;
}

}  // namespace weft
