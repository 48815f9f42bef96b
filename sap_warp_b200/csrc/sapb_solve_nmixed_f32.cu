// Contact-solve kernels of small mixed batches: each world runs the code of its size class; FP32 Hessian and factor.
#include "sapb_contact_solve.cuh"

namespace sapb {
template cudaError_t launch_solve_np<kMixed, true>(const SolveParams&, cudaStream_t, int*);
}  // namespace sapb
