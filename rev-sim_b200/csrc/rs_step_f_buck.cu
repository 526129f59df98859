// Instantiation of the fused step kernels for (float, F_BUCK).
#include "rs_step_impl.cuh"

namespace rs {
template cudaError_t launch_form<float, F_BUCK>(bool, int, int, int, int, const StepArgs &,
                                           const NbConsts<float> &, const BondConsts &, cudaStream_t);
}  // namespace rs
