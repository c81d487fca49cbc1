// Instantiations of the tensor-memory contraction (fold.cuh), a file per family so that they compile side by side.
#include "fold.cuh"

namespace weft {
template int fold_clusters<F_Q4_K>(int);
template cudaError_t launch_fold_kernel<F_Q4_K>(const FoldParams &, const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, int, cudaStream_t);
template int fold_clusters<F_Q5_K>(int);
template cudaError_t launch_fold_kernel<F_Q5_K>(const FoldParams &, const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, int, cudaStream_t);
}  // namespace weft
