// k_scalar.cu -- the step kernels of lattices whose boundary nodes all have closed
// sums, and the choice between them and the others (StepArgs::general).
#include "step_variants.cuh"

namespace tslb_launch {

extern template cudaError_t step_variants<1>(const tslb::StepArgs&, int, int, cudaStream_t, bool, bool);
extern template cudaError_t ensemble_variants<1>(const tslb::StepArgs*, const tslb::WorkItem*, int, int, int, int, unsigned int*,
                                          cudaStream_t, bool);
extern template cudaError_t step_variants<2>(const tslb::StepArgs&, int, int, cudaStream_t, bool, bool);
extern template cudaError_t ensemble_variants<2>(const tslb::StepArgs*, const tslb::WorkItem*, int, int, int, int, unsigned int*,
                                          cudaStream_t, bool);

cudaError_t scalar_step(const tslb::StepArgs& a, int mode, int prec, cudaStream_t st, bool launch, bool early) {
    return a.general == 0   ? step_variants<0>(a, mode, prec, st, launch, early)
           : a.general == 1 ? step_variants<1>(a, mode, prec, st, launch, early)
                            : step_variants<2>(a, mode, prec, st, launch, early);
}

cudaError_t scalar_ensemble(const tslb::StepArgs* args, const tslb::WorkItem* work, int nwork, int grid, int mode, int prec,
                            int general, unsigned int* step, cudaStream_t st, bool launch) {
    return general == 0   ? ensemble_variants<0>(args, work, nwork, grid, mode, prec, step, st, launch)
           : general == 1 ? ensemble_variants<1>(args, work, nwork, grid, mode, prec, step, st, launch)
                          : ensemble_variants<2>(args, work, nwork, grid, mode, prec, step, st, launch);
}

}  // namespace tslb_launch
