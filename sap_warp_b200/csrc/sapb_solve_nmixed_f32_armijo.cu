// The contact-solve kernel of small mixed batches (every size class), 128 threads per world, armijo_decay line search; FP32 Hessian and factor.
#include "sapb_contact_solve.cuh"

namespace sapb {
template cudaError_t launch_solve_ls<128, float, 4, kMixed, SAPB_LS_ARMIJO_DECAY, LdltBlocks<0>::kW[0]>(const SolveParams&, cudaStream_t,
                                                                                      int*);
}  // namespace sapb
