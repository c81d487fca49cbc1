// Instantiations of the tensor-memory contraction (fold.cuh), a file per family so that they compile side by side.
#include "fold.cuh"

namespace weft {
template int fold_clusters<F_Q6_K>(int);
template cudaError_t launch_fold_kernel<F_Q6_K>(const FoldParams &, const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, int, cudaStream_t);
}  // namespace weft
