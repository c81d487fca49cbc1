// Host side of the kernel for a few tokens (few.cuh): which batches take it instead of the register tiles.
#include "few.cuh"

namespace weft {

static bool plan_of(const TileArgs &a, FewPlan &plan) {
    const int nt = (int)((a.m + 7) / 8);
    switch (a.fmt) {
#define FW_PLAN(FMT) case FMT: return few_plan<FMT>(plan, nt, a.k / 256);
    TL_EACH_FORMAT(FW_PLAN)
#undef FW_PLAN
    default: return false;
    }
}

// Where the streaming kernel is the quicker one.  Measured at 3400 sizes (3 to 32 tokens, 256 to 32768 rows, K 512 to 14336, all formats) against
// the register tiles: 2300 of them are taken, with 0.83 of their time in the median; 1.5 % of those are more than 2 % slower, none more than 7 %.
// What is not, with streaming / tiles in us:
// * Q4_0 and Q8_0, with an epilogue for every 32 elements, gain where the tiles' grid is more than one round and rows are long
//   (16 x 14336 x 4096 Q8_0 18.7 / 23.0, Q4_0 17.3 / 19.8; 16 x 8192 x 2048 Q4_0 9.6 / 8.2);
// * a ring with one slot for each team only (the planes take the rest) leaves nothing to hide the copies behind, which the formats with
//   little arithmetic feel (8 x 4096 x 14336 Q5_K 18.1 / 15.7; Q6_K 6144 rows 29.7 / 37.4);
// * tiles of few rows: more than eight tokens on fewer rows than SMs take K in slices there (16 x 512 x 4096 Q4_K 5.4 / 5.1, 24 x 512 Q6_K 7.0 / 6.4);
// * short rows: the collector's turn for a tile is as long as the tile (32 x 28672 x 1024 Q5_K 17.6 / 14.7).
bool few_supported(const TileArgs &a) {
    FewPlan plan;
    if (a.m < 3 || a.m > 32 || a.k % 256 || a.k < 256 || a.n > (1LL << 30) || (reinterpret_cast<uintptr_t>(a.w) & 15u) || !plan_of(a, plan)) return false;
    const bool tight = plan.slots < 2 * FW_WARPS / fw_members(a.fmt);
    switch (a.fmt) {
    case F_Q4_0: return !tight && (a.m <= 8 ? a.k >= 8192 : a.k >= 4096 && (a.m <= 16 ? a.n >= 6144 : a.m <= 24 && a.n >= 9472));
    case F_Q8_0: return a.m > 8 && a.m <= 24 && a.n >= 6144 && a.k >= (a.m <= 16 ? 2048 : 4096);
    case F_Q4_K: case F_Q5_K: if (tight) return a.n >= 24576; break;
    case F_Q2_K: if (a.m > 24 || a.k < 2048) return false; break;
    case F_IQ2_XXS: break;
    case F_Q3_K: return a.m <= 16 || a.n >= 512;
    case F_TQ1_0: if (a.m <= 8 && a.k <= 4096 && a.n >= 2048 && a.n <= 5120) return false; break;      // a tile and three quarters for a CTA
    default: break;
    }
    if (a.m <= 8) return true;
    if (a.fmt != F_IQ2_XXS && a.n < (a.m <= 16 && a.k >= 4096 ? 1024 : 1536)) return false;
    return a.k >= 2048 || a.n <= 16384;
}

cudaError_t launch_few(const TileArgs &a, uint8_t *planes, int *status, int sm_count, cudaStream_t stream) {
    const cudaError_t e = launch_tile_planes(a, planes, stream);
    if (e != cudaSuccess) return e;
    switch (a.fmt) {
#define FW_LAUNCH(FMT) case FMT: return launch_few_kernel<FMT>(a, planes, status, sm_count, stream);
    TL_EACH_FORMAT(FW_LAUNCH)
#undef FW_LAUNCH
    default: return cudaErrorNotSupported;
    }
}

}  // namespace weft
