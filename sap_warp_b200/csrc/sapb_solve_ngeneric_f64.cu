// Contact-solve kernels sized at run time (n <= 60); FP64 Hessian and factor.
#include "sapb_contact_solve.cuh"

namespace sapb {
template cudaError_t launch_solve_np<0, false>(const SolveParams&, cudaStream_t, int*);
}  // namespace sapb
