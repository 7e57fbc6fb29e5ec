// k_general.cu -- the step kernels of lattices with nodes on the general boundary path
// (StepArgs::general 2).
#include "step_variants.cuh"

namespace tslb_launch {

template cudaError_t step_variants<2>(const tslb::StepArgs&, int, int, cudaStream_t, bool, bool);
template cudaError_t ensemble_variants<2>(const tslb::StepArgs*, const tslb::WorkItem*, int, int, int, int, unsigned int*,
                                          cudaStream_t, bool);

}  // namespace tslb_launch
