// k_inlet.cu -- the step kernels of lattices with inlet or outlet faces normal to y or z and
// no other boundary nodes without closed sums (StepArgs::general 1).
#include "step_variants.cuh"

namespace tslb_launch {

template cudaError_t step_variants<1>(const tslb::StepArgs&, int, int, cudaStream_t, bool, bool);
template cudaError_t ensemble_variants<1>(const tslb::StepArgs*, const tslb::WorkItem*, int, int, int, int, unsigned int*,
                                          cudaStream_t, bool);

}  // namespace tslb_launch
