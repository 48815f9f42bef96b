// Contact-solve kernels of small mixed batches: each world runs the code of its size class; FP64 Hessian and factor.
#include "sapb_contact_solve.cuh"

namespace sapb {
template cudaError_t launch_solve_np<kMixed, false>(const SolveParams&, cudaStream_t, int*);
}  // namespace sapb
