// The contact-solve kernel of small mixed batches (every size class), 128 threads per world, exact_root line search; FP64 Hessian and factor.
#include "sapb_contact_solve.cuh"

namespace sapb {
template cudaError_t launch_solve_ls<128, double, 3, kMixed, SAPB_LS_EXACT_ROOT, LdltBlocks<0>::kW[0]>(const SolveParams&, cudaStream_t,
                                                                                      int*);
}  // namespace sapb
