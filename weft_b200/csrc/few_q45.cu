// Instantiations of the kernel for a few tokens (few.cuh), one file per family so that they compile side by side.
#include "few.cuh"

namespace weft {
template cudaError_t launch_few_kernel<F_Q4_0>(const TileArgs &, const uint8_t *, int *, int, cudaStream_t);
template cudaError_t launch_few_kernel<F_Q4_K>(const TileArgs &, const uint8_t *, int *, int, cudaStream_t);
template cudaError_t launch_few_kernel<F_Q5_K>(const TileArgs &, const uint8_t *, int *, int, cudaStream_t);
}  // namespace weft
