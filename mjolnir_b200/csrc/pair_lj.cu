// The pair kernels of the Lennard-Jones family.
#include "pair_kernels.cuh"

namespace mjg {
template void pair_term<G_LJ>(const Arena&, TermArrays&, bool, bool, cudaStream_t);
}  // namespace mjg
