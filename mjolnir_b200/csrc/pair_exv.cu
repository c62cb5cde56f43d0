// The pair kernels of the ExcludedVolume family.
#include "pair_kernels.cuh"

namespace mjg {
template void pair_term<G_EXV>(const Arena&, TermArrays&, bool, bool, cudaStream_t);
}  // namespace mjg
