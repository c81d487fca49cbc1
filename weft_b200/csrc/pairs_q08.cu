// Instantiations of the contraction on CTA pairs (pairs.cuh), a file per family so that they compile side by side.
#include "pairs.cuh"

namespace weft {
template cudaError_t launch_pair_kernel<F_Q4_0>(const PairParams &, const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, int, cudaStream_t);
template cudaError_t launch_pair_kernel<F_Q8_0>(const PairParams &, const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, int, cudaStream_t);
}  // namespace weft
