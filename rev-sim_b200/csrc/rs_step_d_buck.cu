// Instantiation of the fused step kernels for (double, F_BUCK).
#include "rs_step_impl.cuh"

namespace rs {
template cudaError_t launch_form<double, F_BUCK>(bool, int, int, int, int, const StepArgs &,
                                           const NbConsts<double> &, const BondConsts &, cudaStream_t);
}  // namespace rs
