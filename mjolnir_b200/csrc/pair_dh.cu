// The pair kernels of the DebyeHuckel.
#include "pair_kernels.cuh"

namespace mjg {
template void pair_term<G_DH>(const Arena&, TermArrays&, bool, bool, cudaStream_t);
}  // namespace mjg
